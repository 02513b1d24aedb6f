// How the CTAs that share an output tile (its K slices) agree on who adds the partial tiles.
#pragma once

#include <stdint.h>

namespace ribn {

// The sum of a tile is cut into shares, one per slice (the first 24 of them): added by one CTA alone, the partial tiles are read at what
// a single SM can have in flight (nine of 128 x 256: 24 us).  A CTA whose slice is done waits for the others, but not for long: they may
// not be running, because kernels of other streams hold their SMs -- and such a kernel may be waiting in the same way.  When its patience
// ends, a CTA leaves its share to the last slice to arrive and goes.  So every wait ends without an error, whatever else runs on the GPU.
//
// The word of a tile holds the arrivals (bits 0..7) and the shares left behind (bits 8..31): the last arrival's own increment returns
// every share left before it, and a CTA that leaves its share learns from the same atomic whether the last one had arrived already, in
// which case it adds the share after all.
constexpr int kExchangeShares = 24;

__device__ __forceinline__ int exchange_shares(int slices) { return slices < kExchangeShares ? slices : kExchangeShares; }

// One thread per CTA, after its slice's partial tile is visible to the GPU.  Returns a bit per share that the CTA is to add.
// patience_ns 0: nobody waits, the last arrival adds everything and leaves the word at zero.  Otherwise each CTA calls
// exchange_depart once it has the answer.
__device__ __forceinline__ uint32_t exchange_arrive(unsigned int* word, int slices, int slice, uint32_t patience_ns) {
    const unsigned int before = atomicAdd(word, 1u);
    if (patience_ns == 0u) {
        if (before != static_cast<unsigned int>(slices - 1)) return 0u;
        *word = 0u;   // ready for the next launch
        return (1u << exchange_shares(slices)) - 1u;
    }
    const uint32_t own = slice < kExchangeShares ? 1u << slice : 0u;
    // The first look is on its way together with the increment: waiting for the increment's answer first is a round trip more for all
    // that arrive just before the last (0.35 us per projection of a decode step of 32 sequences).
    const volatile unsigned int* arrivals = word;
    bool all = (*arrivals & 0xffu) == static_cast<unsigned int>(slices);
    if ((before & 0xffu) == static_cast<unsigned int>(slices - 1)) return own | before >> 8;
    if (all || own == 0u) return own;
    unsigned long long start, now;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(start));
    do {
        for (int poll = 0; poll < 64 && !all; ++poll) all = (*arrivals & 0xffu) == static_cast<unsigned int>(slices);
        if (all) return own;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
    } while (now - start < patience_ns);
    return (atomicOr(word, own << 8) & 0xffu) == static_cast<unsigned int>(slices) ? own : 0u;
}

// How many of a tile's CTAs have departed before; the one that answers slices - 1 is the last to have looked at the word and calls
// exchange_reset.
__device__ __forceinline__ unsigned int exchange_depart(unsigned int* departed) { return atomicAdd(departed, 1u); }
__device__ __forceinline__ void exchange_reset(unsigned int* word, unsigned int* departed) {
    *departed = 0u;
    *word = 0u;
}

// Takes the lowest run of neighbouring shares off `mine`: items [first, last) of `items` (32-bit divisions, items * 24 below 2^31: the
// 64-bit ones cost the batch kernel's Q6_K form, which has no register to spare, up to twenty bytes of spills).
__device__ __forceinline__ void exchange_next(uint32_t& mine, int shares, int items, int& first, int& last) {
    const int begin = __ffs(static_cast<int>(mine)) - 1;
    const uint32_t rest = ~(mine >> begin);
    const int run = __ffs(static_cast<int>(rest)) - 1;   // at most 24 bits are set
    mine &= ~(((1u << run) - 1u) << begin);
    first = static_cast<int>(static_cast<uint32_t>(items * begin) / static_cast<uint32_t>(shares));
    last = static_cast<int>(static_cast<uint32_t>(items * (begin + run)) / static_cast<uint32_t>(shares));
}

}  // namespace ribn
