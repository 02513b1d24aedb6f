// Quantized GEMM on the 5th-generation tensor cores (tcgen05 + TMEM) with the
// dequantisation fused into the operand producer.
//
//   Y[m][n] = sum_k dequant(W[n][k]) * X[m][k]      X bf16 (or f32) [M][K], f32 accumulate
//
// The reference has no such kernel: its prefill runs the batched GEMV eight
// tokens at a time (crates/nvidia/src/decode.rs:1953-1977, :2149-2267 over
// q4_k.cu:161-258 and twins), and batches above eight are not served at all
// (crates/nvidia/src/quantized.rs:464-469).  This kernel serves ribn_gemm.
//
// A pair of CTAs (a cluster of two, cta_group::2) works on units of 256 weight
// rows, 128 per CTA (one TMEM lane per row), x NT tokens (a multiple of 16 up to
// 256) x a range of K; the grid is one pair per two SMs, each walking its share
// of the units.  Per 64-wide K step:
//   A = 128 x 64 dequantised weights per CTA as f16, made by sixteen dequant warps
//       (two sets of eight, super-blocks in turn) from the raw GGUF bytes that a
//       producer thread streams in as tiled TMA boxes.  Units with one sum keep
//       A in tensor memory (tcgen05.st), two super-blocks of it behind 256
//       accumulator columns; units with two sums of up to 256 tokens fill TMEM
//       with accumulators and keep A as swizzled tiles in shared memory;
//   B = NT x 64 activations as f16, half of the tile in each CTA of the pair: a
//       pre-pass multiplies every token row by a power of two (largest magnitude
//       at most 2^14), which the epilogue undoes, and lays the rows out as the
//       tiles the MMA reads: a bulk copy per step brings the half tile;
//   D (TMEM, f32) += A * B  with four tcgen05.mma of 256 x NT x 16, issued by one
//       thread of the pair's first CTA; tcgen05.commit releases the stages of
//       both CTAs.
//
// What bounds it: a step of NT tokens takes the tensor pipe 2 NT clocks; the
// issuing warp needs about 510 for its four MMAs, wait and commit, the dequant
// warps 500 (Q4_K) to 650 (Q6_K) of half-rate logic.  One CTA per tile of 128
// rows (the form before this one) took 1800 clocks per step of 256 tokens: three
// stages at most for weights and activations together, and a dequant warp that
// waited for its stage before it began its step.  Now the pair halves what each
// SM reads of B and leaves room for rings of five to seven stages, a step is
// complete in registers before its stage is asked for, and K ranges are added by
// all CTAs of a tile.  Measured, pre-pass included: 173 tokens, Q5_K 5120 x 5120:
// 55.2 -> 25.1 us; 512 tokens, Q4_K 12288 x 4096: 128.6 -> 67.8 us; 2048 tokens,
// Q6_K 4096 x 12288: 288 -> 207 us (1 PFLOP/s).
//
// The epilogue reads D with tcgen05.ld (thread = weight row, registers = tokens)
// and stores Y, 4 to 8 thousand clocks per unit (all SMs store at once), half of
// it under the next unit's first MMAs.  With split-K the partial tiles go to a
// scratch buffer and are added in slice order, so results are deterministic.
//
// Precision: a single bf16 rounding of the weights (2^-9 relative) does not
// meet the 2e-3 bound of the path over millions of outputs; an f16 rounding
// (2^-12 relative, what the decode batch kernels apply) does, with one MMA per
// K step where a split of every weight into two bf16 parts needed two.  Both
// operands of kind::f16 must have the same format (an f16 A operand with a
// bf16 B operand is an illegal instruction), hence the f16 copy of the
// activations; bf16 activations convert exactly.  Weights beyond the f16 range
// (|w| > 65504: super-block scales no checkpoint has) come out as infinities.
//
// Every wait on an mbarrier is bounded; a wait that runs out sets the status
// word, and every warp still reaches the common teardown that frees TMEM.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "formats.cuh"
#include "internal.h"
#include "row_dequant.cuh"
#include "split_exchange.cuh"
#include "tc_host.h"
#include "tcgen05.cuh"
#include "unpack.cuh"

namespace ribn {
namespace {

constexpr int kBM = 128;            // weight rows per CTA
constexpr int kBK = 64;             // K elements per step (one 128-byte swizzled row)
constexpr int kSub = kSuperBlock / kBK;  // steps per super-block
constexpr int kSlots = kSub;         // step s of every super-block goes through stage s of the A ring, and of one half of the B ring or the other
constexpr int kProducerWarp = 0;     // raw weight bytes
constexpr int kActivationWarp = 1;   // activation tiles
constexpr int kIssuerWarp = 2;       // first CTA of the pair: the MMAs; second: tells the first that its half of a B tile is in place
constexpr int kFirstDequantWarp = 4; // a multiple of four: a warp reaches the TMEM lanes of quadrant warp % 4
constexpr int kDequantWarps = 16;    // two sets, a thread per (weight row, half super-block)
constexpr int kTcThreads = (kFirstDequantWarp + kDequantWarps) * 32;
constexpr int kMaxTokens = 256;      // per unit: the UMMA N dimension
constexpr int kARingColumns = 32 * kSlots;   // of TMEM, for the A operand of one super-block: 64 halves per row and step
constexpr int kATileBytes = kBM * kBK * 2;   // of shared memory, for the A operand of one step
constexpr int kGroupBytes = 8 * kBK * 2;   // eight token rows of one K step, one swizzle atom

// Tiled TMA wants 16-byte aligned bases and row pitches.  The rows of a Q6_K matrix (210-byte super-blocks) have them only
// when K/256 is a multiple of eight; otherwise rows c, c + P, c + 2 P, ... (P = 16 / gcd(row bytes, 16)) are a multiple of 16
// bytes apart and the matrix is P interleaved ones, a tensor map each (base rounded down to 16 bytes): a tile is P boxes of
// 128 / P rows.
struct RawMaps {
    CUtensorMap map[8];
};

// Which of a unit's K steps are added together in TMEM.  Two sums are added to each other at the end.  The choice goes with the
// call's token count, not with the tile NT, so that results do not change with how the work is cut.
enum SumOrder { kOneSum = 0, kEvenOdd = 1, kEveryThird = 2 };   // every third: steps 1, 4, 7, ... and the rest

struct GemmParams {
    const uint8_t* image;    // the activations as MMA tiles (see gemm_image_kernel)
    int row_groups;          // groups of eight token rows the image is laid out for
    void* y;                 // [m][n] f32 or bf16
    float* partial;          // split-K scratch: [ksplit][m][n] f32
    const float* x_scale;    // power-of-two factor per token row (activations were divided by it)
    unsigned int* tickets;   // one counter per (tile of 128 rows, token tile), zero between launches
    int n, m, nsb, ksplit, y_bf16;
    int nt, m_tiles, row_pairs, units;   // tokens per unit; units = row_pairs * m_tiles * ksplit, token tile fastest, K range slowest
    int order;               // SumOrder
    unsigned int patience_ns;   // how long the CTAs of a tile wait for one another to share the sum of its partial tiles; 0: the last one adds
    int ticket_stride;       // departures are counted this far behind the arrivals
    int row_classes;         // P above
    unsigned int row_bytes;
    int* status;
};

// SMEM_A: where the A operand lives.  One sum per unit takes half of TMEM and leaves the other half to an A ring of two
// super-blocks; two sums of 256 tokens take all of it, and the A ring, of one super-block, lies in shared memory.
template <uint32_t FMT, bool SMEM_A>
struct TcGeometry {
    using F = Format<FMT>;
    // A box starts on the 16-byte boundary at or below its super-block: Q6_K super-blocks start anywhere on 2-byte boundaries.
    static constexpr int kSlot = FMT == kQ6_K ? 240 : F::kBytes;
    static constexpr int kRawStageBytes = kBM * kSlot;
    static constexpr int kBTileBytes = kMaxTokens / 2 * kBK * 2;   // this CTA's half of the largest token tile
    static constexpr int kADepth = SMEM_A ? 1 : 2;                 // super-blocks in the A ring
    // Even: a stage always belongs to the same set of dequant warps.
    static constexpr int kRawStages = !SMEM_A && (FMT == kQ4_K || FMT == kQ5_K) ? 4 : 2;
    static constexpr int kFixedBytes = 1024 + 512 + kRawStages * kRawStageBytes + (SMEM_A ? kSlots * kATileBytes : 0);   // and alignment slack, barriers
    // Up to 7: the load of a step waits for the MMAs of the step that many before it on a barrier they share with the step eight
    // before.
    static constexpr int kBFit = (227 * 1024 - kFixedBytes) / kBTileBytes;
    static constexpr int kBStages = kBFit > 7 ? 7 : kBFit;
    static constexpr int kSmemBytes = kFixedBytes + kBStages * kBTileBytes;
    static_assert(kBStages >= 5, "tile plan exceeds shared memory");
};

// One unit of work.
struct Unit {
    int row_tile;      // of 128 rows, this CTA's
    int token0, sb_begin, sb_count, k_slice, token_tile;
};
__device__ __forceinline__ Unit unit_at(const GemmParams& p, int u, int rank) {
    Unit w;
    w.token_tile = u % p.m_tiles;
    const int rest = u / p.m_tiles;
    w.row_tile = 2 * (rest % p.row_pairs) + rank;
    w.k_slice = rest / p.row_pairs;
    w.token0 = w.token_tile * p.nt;
    w.sb_begin = static_cast<int>(static_cast<long long>(p.nsb) * w.k_slice / p.ksplit);
    w.sb_count = static_cast<int>(static_cast<long long>(p.nsb) * (w.k_slice + 1) / p.ksplit) - w.sb_begin;
    return w;
}
// A ring position: stage and the parity of its current round.
struct Ring {
    int stage = 0;
    uint32_t round = 0;
    __device__ void advance(int stages) {
        if (++stage == stages) {
            stage = 0;
            ++round;
        }
    }
};
// TMEM: accumulators, then (A ring in TMEM) the A ring.  Two buffers of accumulators where tokens leave room, one otherwise.
__device__ __forceinline__ int acc_buffers(int nt) { return nt <= kMaxTokens / 2 ? 2 : 1; }
template <bool SMEM_A>
__device__ __forceinline__ uint32_t acc_column(int nt, int buffer, int sum) {
    return static_cast<uint32_t>(buffer * (SMEM_A ? kMaxTokens : kMaxTokens / 2) + sum * (nt <= kMaxTokens / 2 ? kMaxTokens / 2 : kMaxTokens));
}
constexpr uint32_t kARing = kMaxTokens;   // first TMEM column of the A ring

// ---------------------------------------------------------------- pair primitives
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Arrive on the barrier at the same offset in the pair's first CTA.  What it publishes has been handed to the async proxy (by a
// bulk copy's own completion, or fence.proxy.async in the writer), so the arrival keeps the CTA scope: with .release.cluster it
// waits for every store of the SM and costs its thread about 1100 clocks, a K step and a half.
__device__ __forceinline__ uint32_t address_in_first(const void* p) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(smem_addr(p)));
    return a;
}
__device__ __forceinline__ void mbar_arrive_first(uint32_t bar_in_first) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar_in_first) : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* holder, uint32_t columns) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(holder)), "r"(columns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t base, uint32_t columns) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(columns) : "memory");
}
// The four K slices of a step, A slices 8 TMEM columns apart, B slices 32 bytes along the swizzled rows, and the commit that arrives
// on `bar` in both CTAs once they have completed; by the elected lane of a converged warp.
__device__ __forceinline__ void umma_pair_step_elected(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate_first, uint32_t bar) {
    asm volatile(
        "{\n\t"
        ".reg .pred pf, pt, pe;\n\t"
        ".reg .b64 b1, b2, b3;\n\t"
        ".reg .b32 a1, a2, a3, leader;\n\t"
        ".reg .b16 both;\n\t"
        "elect.sync leader|pe, 0xffffffff;\n\t"
        "setp.ne.b32 pf, %4, 0;\n\t"
        "setp.eq.b32 pt, 0, 0;\n\t"
        "mov.b16 both, 3;\n\t"
        "add.u32 a1, %1, 8;\n\t"
        "add.u32 a2, %1, 16;\n\t"
        "add.u32 a3, %1, 24;\n\t"
        "add.s64 b1, %2, 2;\n\t"
        "add.s64 b2, %2, 4;\n\t"
        "add.s64 b3, %2, 6;\n\t"
        "@pe tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, pf;\n\t"
        "@pe tcgen05.mma.cta_group::2.kind::f16 [%0], [a1], b1, %3, pt;\n\t"
        "@pe tcgen05.mma.cta_group::2.kind::f16 [%0], [a2], b2, %3, pt;\n\t"
        "@pe tcgen05.mma.cta_group::2.kind::f16 [%0], [a3], b3, %3, pt;\n\t"
        "@pe tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%5], both;\n\t"
        "}"
        :
        : "r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate_first), "r"(bar)
        : "memory");
}
// The same with the A operand in shared memory (a swizzled K-major tile like B's).
__device__ __forceinline__ void umma_pair_step_elected(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate_first, uint32_t bar) {
    asm volatile(
        "{\n\t"
        ".reg .pred pf, pt, pe;\n\t"
        ".reg .b64 a1, a2, a3, b1, b2, b3;\n\t"
        ".reg .b32 leader;\n\t"
        ".reg .b16 both;\n\t"
        "elect.sync leader|pe, 0xffffffff;\n\t"
        "setp.ne.b32 pf, %4, 0;\n\t"
        "setp.eq.b32 pt, 0, 0;\n\t"
        "mov.b16 both, 3;\n\t"
        "add.s64 a1, %1, 2;\n\t"
        "add.s64 a2, %1, 4;\n\t"
        "add.s64 a3, %1, 6;\n\t"
        "add.s64 b1, %2, 2;\n\t"
        "add.s64 b2, %2, 4;\n\t"
        "add.s64 b3, %2, 6;\n\t"
        "@pe tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, pf;\n\t"
        "@pe tcgen05.mma.cta_group::2.kind::f16 [%0], a1, b1, %3, pt;\n\t"
        "@pe tcgen05.mma.cta_group::2.kind::f16 [%0], a2, b2, %3, pt;\n\t"
        "@pe tcgen05.mma.cta_group::2.kind::f16 [%0], a3, b3, %3, pt;\n\t"
        "@pe tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%5], both;\n\t"
        "}"
        :
        : "r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate_first), "r"(bar)
        : "memory");
}
// 32 lanes x 32 columns: thread i of the warp writes TMEM lane (base lane + i).
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint4 (&r)[8]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,"
        "%26,%27,%28,%29,%30,%31,%32};\n\t"
        "tcgen05.wait::st.sync.aligned;" ::"r"(taddr),
        "r"(r[0].x), "r"(r[0].y), "r"(r[0].z), "r"(r[0].w), "r"(r[1].x), "r"(r[1].y), "r"(r[1].z), "r"(r[1].w), "r"(r[2].x), "r"(r[2].y),
        "r"(r[2].z), "r"(r[2].w), "r"(r[3].x), "r"(r[3].y), "r"(r[3].z), "r"(r[3].w), "r"(r[4].x), "r"(r[4].y), "r"(r[4].z), "r"(r[4].w),
        "r"(r[5].x), "r"(r[5].y), "r"(r[5].z), "r"(r[5].w), "r"(r[6].x), "r"(r[6].y), "r"(r[6].z), "r"(r[6].w), "r"(r[7].x), "r"(r[7].y),
        "r"(r[7].z), "r"(r[7].w)
        : "memory");
}
__device__ __forceinline__ void mbar_arrive_local(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void sts128(uint32_t a, uint4 v) {
    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
// Keeps a value's computation ahead of what follows (the compiler would sink it below the wait that precedes its use).
__device__ __forceinline__ void settle(uint4 (&r)[8]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) asm volatile("" : "+r"(r[i].x), "+r"(r[i].y), "+r"(r[i].z), "+r"(r[i].w));
}
// Arrive on `bar` in both CTAs once the MMAs issued so far have completed (elected lane of a converged warp).
__device__ __forceinline__ void umma_commit_pair_elected(uint32_t bar) {
    asm volatile(
        "{\n\t"
        ".reg .pred pe;\n\t"
        ".reg .b32 leader;\n\t"
        ".reg .b16 both;\n\t"
        "mov.b16 both, 3;\n\t"
        "elect.sync leader|pe, 0xffffffff;\n\t"
        "@pe tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], both;\n\t"
        "}" ::"r"(bar)
        : "memory");
}

// ---------------------------------------------------------------- dequantisation: one row, one 64-wide K step
// Eight 16-byte chunks (K offsets 8 c .. 8 c + 7) of f16 weights, each rounded once from the f32 value that the rest of the
// library dequantises to: w = scale * (128 + q) - (scale * (128 + bias) + minimum), one prmt and one FMA per weight, one
// conversion per two (the folded constant is rounded at 2^-17 of a quant step, far below the f16 rounding).
struct Fold {
    float scale, offset;
    __device__ Fold(float s, float bias, float minimum) : scale(s), offset(-fmaf(s, 128.0f + bias, minimum)) {}
};
__device__ __forceinline__ uint32_t fold_pair(float x0, float x1, float scale, float offset) {
    return half2_bits(fmaf(x0, scale, offset), fmaf(x1, scale, offset));
}
__device__ __forceinline__ uint4 fold_chunk(uint32_t q0, uint32_t q1, const Fold& f) {
    return make_uint4(fold_pair(byte_plus_128<0>(q0), byte_plus_128<1>(q0), f.scale, f.offset),
                      fold_pair(byte_plus_128<2>(q0), byte_plus_128<3>(q0), f.scale, f.offset),
                      fold_pair(byte_plus_128<0>(q1), byte_plus_128<1>(q1), f.scale, f.offset),
                      fold_pair(byte_plus_128<2>(q1), byte_plus_128<3>(q1), f.scale, f.offset));
}

// 32 bytes from an address on a 2-byte boundary, as eight words
__device__ __forceinline__ void lds256_unaligned(uint32_t a, uint32_t (&out)[8]) {
    const uint32_t base = a & ~15u, shift = (a & 2u) * 8u;
    const uint4 v0 = lds128(base), v1 = lds128(base + 16), v2 = lds128(base + 32);
    const uint32_t w[12] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w, v2.x, v2.y, v2.z, v2.w};
    switch ((a >> 2) & 3u) {   // the same for all rows of a class
        case 0:
#pragma unroll
            for (int i = 0; i < 8; ++i) out[i] = __funnelshift_r(w[i], w[i + 1], shift);
            break;
        case 1:
#pragma unroll
            for (int i = 0; i < 8; ++i) out[i] = __funnelshift_r(w[i + 1], w[i + 2], shift);
            break;
        case 2:
#pragma unroll
            for (int i = 0; i < 8; ++i) out[i] = __funnelshift_r(w[i + 2], w[i + 3], shift);
            break;
        default:
#pragma unroll
            for (int i = 0; i < 8; ++i) out[i] = __funnelshift_r(w[i + 3], w[i + 4 < 12 ? i + 4 : 11], shift);
            break;
    }
}

// Half a super-block of one row: `load` fetches what its two steps share, `step<J>` makes step 2 half + J.  One copy of the code
// serves all warps: with a copy per step, the shifts constants, the copies pushed each other out of the instruction cache.
template <uint32_t FMT>
struct HalfBlock;

// 32 low nibbles and 32 high nibbles of eight words, with their own scale and offset: one step
__device__ __forceinline__ void fold_nibbles(const uint32_t (&lo)[8], const uint32_t (&hi)[8], const Fold& f0, const Fold& f1, uint4 (&out)[8]) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        out[c] = fold_chunk(lo[2 * c], lo[2 * c + 1], f0);
        out[4 + c] = fold_chunk(hi[2 * c], hi[2 * c + 1], f1);
    }
}

// Scales and minima of the four sub-blocks of half a Q4_K / Q5_K super-block.
struct KScales {
    uint32_t sc, mn;
    float d, dmin;
    __device__ void load(uint32_t blk, int half) {
        const uint4 h = lds128(blk);
        d = f16_bits_to_f32(h.x & 0xffffu);
        dmin = f16_bits_to_f32(h.x >> 16);
        uint32_t sc_lo, sc_hi, m_lo, m_hi;
        unpack_k_scales(h.y, h.z, h.w, sc_lo, sc_hi, m_lo, m_hi);
        sc = half ? sc_hi : sc_lo;
        mn = half ? m_hi : m_lo;
    }
    __device__ Fold fold(int i) const { return Fold(d * byte_of(sc, i), 0.0f, dmin * byte_of(mn, i)); }
};

template <>
struct HalfBlock<kQ4_K> {
    static constexpr bool kHeld = false;   // after `load` the raw bytes are no longer needed
    KScales scales;
    uint32_t quants;
    __device__ void load(uint32_t blk, int half) {
        scales.load(blk, half);
        quants = blk + 16 + 64 * half;
    }
    template <int J>
    __device__ void step(uint4 (&out)[8]) const {
        const uint4 a = lds128(quants + 32 * J), b = lds128(quants + 32 * J + 16);
        const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        uint32_t lo[8], hi[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            lo[i] = w[i] & 0x0f0f0f0fu;
            hi[i] = (w[i] >> 4) & 0x0f0f0f0fu;
        }
        fold_nibbles(lo, hi, scales.fold(2 * J), scales.fold(2 * J + 1), out);
    }
};

template <>
struct HalfBlock<kQ5_K> {
    static constexpr bool kHeld = false;
    KScales scales;
    uint32_t quants;
    uint32_t bits[8];   // byte p holds, in bits 0..3, the fifth bits of position p of the half's four sub-blocks
    __device__ void load(uint32_t blk, int half) {
        scales.load(blk, half);
        quants = blk + 48 + 64 * half;
        const uint4 a = lds128(blk + 16), b = lds128(blk + 32);
        const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) bits[i] = w[i] >> (4 * half);
    }
    template <int J>
    __device__ void step(uint4 (&out)[8]) const {
        const uint4 a = lds128(quants + 32 * J), b = lds128(quants + 32 * J + 16);
        const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        uint32_t lo[8], hi[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            lo[i] = and_or(bits[i] << (4 - 2 * J), 0x10101010u, w[i] & 0x0f0f0f0fu);
            hi[i] = and_or(bits[i] << (3 - 2 * J), 0x10101010u, (w[i] >> 4) & 0x0f0f0f0fu);
        }
        fold_nibbles(lo, hi, scales.fold(2 * J), scales.fold(2 * J + 1), out);
    }
};

template <>
struct HalfBlock<kQ6_K> {
    static constexpr bool kHeld = true;
    // a chunk of 128: two runs of 32 bytes with the low four bits (step 0 in their low nibbles, step 1 in the high ones) and one
    // run with two bits for each of the four sub-blocks
    uint32_t l0[8], l1[8], hb[8];
    uint32_t scales[4];   // pairs of signed bytes
    float d;
    __device__ void load(uint32_t blk, int half) {
        lds256_unaligned(blk + 64 * half, l0);
        lds256_unaligned(blk + 64 * half + 32, l1);
        lds256_unaligned(blk + 128 + 32 * half, hb);
        d = f16_bits_to_f32(lds_u16(blk + 208));
#pragma unroll
        for (int i = 0; i < 4; ++i) scales[i] = lds_u16(blk + 192 + 8 * half + 2 * i);
    }
    template <int J>
    __device__ void step(uint4 (&out)[8]) const {
        const uint32_t pair0 = scales[2 * J], pair1 = scales[2 * J + 1];
        const Fold f[4] = {Fold(d * static_cast<float>(static_cast<int8_t>(pair0 & 0xffu)), 32.0f, 0.0f),
                           Fold(d * static_cast<float>(static_cast<int8_t>(pair0 >> 8)), 32.0f, 0.0f),
                           Fold(d * static_cast<float>(static_cast<int8_t>(pair1 & 0xffu)), 32.0f, 0.0f),
                           Fold(d * static_cast<float>(static_cast<int8_t>(pair1 >> 8)), 32.0f, 0.0f)};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            uint32_t a[2], b[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int i = 2 * c + h;
                a[h] = and_or(J == 0 ? l0[i] : l0[i] >> 4, 0x0f0f0f0fu, (J == 0 ? hb[i] << 4 : hb[i]) & 0x30303030u);
                b[h] = and_or(J == 0 ? l1[i] : l1[i] >> 4, 0x0f0f0f0fu, (J == 0 ? hb[i] << 2 : hb[i] >> 2) & 0x30303030u);
            }
            out[c] = fold_chunk(a[0], a[1], f[c >> 1]);
            out[4 + c] = fold_chunk(b[0], b[1], f[2 + (c >> 1)]);
        }
    }
};

template <>
struct HalfBlock<kQ8_0> {
    static constexpr bool kHeld = false;
    // four blocks of 34 bytes.  (q ^ 0x80) in bits 8..15 of the mantissa of 32768.0 is 32896 + q, and d * q is exact in f32: one FMA.
    uint32_t blocks;
    __device__ void load(uint32_t blk, int half) { blocks = blk + 136 * half; }
    template <int J>
    __device__ void step(uint4 (&out)[8]) const {
        auto value = [](uint32_t q, int i) { return __uint_as_float(__byte_perm(q, 0x47000000u, 0x7404u + (static_cast<uint32_t>(i) << 4))); };
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            const uint32_t block = blocks + 68 * J + 34 * b;
            uint32_t q[8];
            lds256_unaligned(block + 2, q);
            const float d = f16_bits_to_f32(lds_u16(block));
            const float offset = -32896.0f * d;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                uint32_t r[4];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint32_t w = q[2 * c + h] ^ 0x80808080u;
                    r[2 * h] = fold_pair(value(w, 0), value(w, 1), d, offset);
                    r[2 * h + 1] = fold_pair(value(w, 2), value(w, 3), d, offset);
                }
                out[4 * b + c] = make_uint4(r[0], r[1], r[2], r[3]);
            }
        }
    }
};

// ---------------------------------------------------------------- pre-pass: bf16 rows -> f16 MMA tiles
// One CTA per token row, which it reads once (up to 16384 values stay in registers): the power of two that brings the row's
// largest magnitude to [2^13, 2^14), the row times that power as f16, and the power's inverse for the epilogue.
// Image: [K step][group of eight rows][1024 bytes], a group being rows of 128 bytes with the 128-byte swizzle: the half tile of a
// CTA is one contiguous bulk copy.  Tiles fetched row by row from an [m][k] copy lie K * 2 bytes apart: every SM reads the same
// 128-byte columns of that copy at the same time, and they came at 14 bytes per clock and SM.
constexpr int kImageThreads = 256;
constexpr int kImageChunks = 8;   // of eight values per thread
__global__ void __launch_bounds__(kImageThreads) gemm_image_kernel(const __nv_bfloat16* __restrict__ x, uint8_t* __restrict__ image,
                                                                   float* __restrict__ factor, int k, int row_groups) {
    pdl_launch_dependents();
    pdl_wait_prior();   // x may be the previous kernel's output; the image may still be read by it
    __shared__ float red[kImageThreads / 32];
    const int row = blockIdx.x;
    const uint4* source = reinterpret_cast<const uint4*>(x + static_cast<size_t>(row) * k);
    const int chunks = k / 8;
    uint4 kept[kImageChunks];
    float biggest = 0.0f;
    auto largest = [&](uint4 v) {
        const uint32_t words[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
            biggest = fmaxf(biggest, fmaxf(fabsf(__uint_as_float(words[i] << 16)), fabsf(__uint_as_float(words[i] & 0xffff0000u))));
    };
#pragma unroll
    for (int u = 0; u < kImageChunks; ++u) {
        const int c = threadIdx.x + u * kImageThreads;
        kept[u] = c < chunks ? source[c] : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int u = 0; u < kImageChunks; ++u) largest(kept[u]);
    for (int c = threadIdx.x + kImageChunks * kImageThreads; c < chunks; c += kImageThreads) largest(source[c]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) biggest = fmaxf(biggest, __shfl_xor_sync(0xffffffffu, biggest, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = biggest;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < kImageThreads / 32; ++w) biggest = fmaxf(biggest, red[w]);
    float down = 1.0f, up = 1.0f;   // 2^-e, 2^e
    if (biggest > 0.0f && biggest < 3.0e38f) {
        int e = static_cast<int>(__float_as_uint(biggest) >> 23) - 127 + 1 - 14;   // biggest * 2^-e in [2^13, 2^14)
        e = max(-100, min(100, e));
        down = __uint_as_float(static_cast<uint32_t>(127 - e) << 23);
        up = __uint_as_float(static_cast<uint32_t>(127 + e) << 23);
    }
    if (threadIdx.x == 0) factor[row] = up;
    uint8_t* target = image + static_cast<size_t>(row >> 3) * kGroupBytes + (row & 7) * 128;
    auto store = [&](int c, uint4 v) {
        auto pair = [&](uint32_t w) { return half2_bits(__uint_as_float(w << 16) * down, __uint_as_float(w & 0xffff0000u) * down); };
        *reinterpret_cast<uint4*>(target + static_cast<size_t>(c >> 3) * row_groups * kGroupBytes + (((c & 7) ^ (row & 7)) << 4)) =
            make_uint4(pair(v.x), pair(v.y), pair(v.z), pair(v.w));
    };
#pragma unroll
    for (int u = 0; u < kImageChunks; ++u) {
        const int c = threadIdx.x + u * kImageThreads;
        if (c < chunks) store(c, kept[u]);
    }
    for (int c = threadIdx.x + kImageChunks * kImageThreads; c < chunks; c += kImageThreads) store(c, source[c]);
}

struct Barriers {
    uint64_t raw_full[4];    // bytes
    uint64_t raw_empty[4];   // the eight dequant warps of a set
    uint64_t full[2][kSlots];            // first CTA: four dequant warps of each CTA, its half of B, the second CTA's word for the other
    // One commit, on the barrier of the set that fills the A stage next (that of super-block b + 1 or b + 2): a set sees the phases of
    // its own barriers one after the other, which the one-bit parity needs.
    uint64_t empty[2][kSlots];
    uint64_t half[2][kSlots];            // second CTA: bytes of its half of B
    uint64_t acc_full[2];                // one commit
    uint64_t acc_empty[2];               // first CTA: the dequant warps of both CTAs
    unsigned int* word;   // of the tile, in split_exchange.cuh
    uint32_t tmem;
    uint32_t range;   // tokens whose partial sums this CTA adds: the first, and behind the last << 16
};
static_assert(sizeof(Barriers) <= 512, "the plan sets 512 bytes aside");

// ---------------------------------------------------------------- epilogue: TMEM -> registers -> Y (or split-K partials)
// By the sixteen dequant warps: four per TMEM lane quadrant, sixteen tokens at a time each.  After a wait that ran out (`ok` false)
// nothing is stored, but every warp still meets the others at the barriers.
template <bool SMEM_A>
__device__ __forceinline__ bool store_unit(const GemmParams& p, int u, uint32_t tmem_base, Barriers* bars, int buffer, uint32_t parity, bool ok) {
    const int rank = blockIdx.x & 1;
    const Unit w = unit_at(p, u, rank);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int worker = threadIdx.x - kFirstDequantWarp * 32;
    const int q = warp & 3;                 // a warp may only read TMEM lanes 32 * (warp % 4) .. + 31
    const int share = worker >> 7;
    const long long row = static_cast<long long>(w.row_tile) * kBM + q * 32 + lane;
    pdl_wait_prior();   // the factors are the pre-pass's output; earlier kernels may read y and the partial tiles
    // The factors of this warp's (at most four) groups of sixteen tokens, two per lane, on their way while the last MMAs run.
    const float* x_scale = p.x_scale + w.token0;
    const int last_token = p.m - 1 - w.token0;
    const int own_token = 16 * share + 64 * (lane >> 4) + (lane & 15);
    const float factors01 = x_scale[min(own_token, last_token)], factors23 = x_scale[min(own_token + 128, last_token)];
    ok = ok && __all_sync(0xffffffffu, mbar_spin(&bars->acc_full[buffer], parity));
    tcgen05_fence_after_sync();
    // what the loops need, in registers: a store might alias the parameters
    const bool split = p.ksplit > 1, y_bf16 = p.y_bf16 != 0;
    const int n = p.n;
    void* y = p.y;
    const size_t plane = static_cast<size_t>(p.m) * n;
    float* part = split ? p.partial + static_cast<size_t>(w.k_slice) * plane : nullptr;
    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
    const uint32_t sum0 = lane_base + acc_column<SMEM_A>(p.nt, buffer, 0), sum1 = lane_base + acc_column<SMEM_A>(p.nt, buffer, 1);
    const int tokens = min(p.nt, p.m - w.token0);
    if (ok) {
#pragma unroll
        for (int g = 0; g < kMaxTokens / 64; ++g) {
            const int c0 = 16 * share + 64 * g;
            if (c0 >= tokens) break;
            uint32_t v[16];
            tmem_ld16(sum0 + c0, v);
            if (SMEM_A) {   // two sums
                uint32_t second[16];
                tmem_ld16(sum1 + c0, second);
                tmem_ld_wait();
#pragma unroll
                for (int jj = 0; jj < 16; ++jj) v[jj] = __float_as_uint(__uint_as_float(v[jj]) + __uint_as_float(second[jj]));
            } else {
                tmem_ld_wait();
            }
            size_t o = static_cast<size_t>(w.token0 + c0) * n + row;
#pragma unroll
            for (int jj = 0; jj < 16; ++jj, o += n) {
                // the token row's factor, undone
                const float value = __uint_as_float(v[jj]) * __shfl_sync(0xffffffffu, g < 2 ? factors01 : factors23, 16 * (g & 1) + jj);
                if (c0 + jj < tokens && row < n) {
                    if (split) part[o] = value;
                    else if (y_bf16) static_cast<__nv_bfloat16*>(y)[o] = __float2bfloat16_rn(value);
                    else static_cast<float*>(y)[o] = value;
                }
            }
        }
    }
    tcgen05_fence_before_sync();
    __syncwarp();
    if (lane == 0) mbar_arrive_first(address_in_first(&bars->acc_empty[buffer]));
    // Split-K: the partial tiles of a tile are added in slice order, by all CTAs of the tile where the launch expects them to run
    // at the same time (split_exchange.cuh), else by the last to arrive.
    if (split) {
        const int ksplit = p.ksplit;
        __threadfence();
        named_barrier_sync(2, kDequantWarps * 32);
        if (worker == 0) {
            unsigned int* word = p.tickets + w.token_tile * 2 * p.row_pairs + w.row_tile;
            bars->word = word;
            // From the first to the last of the CTA's shares: one between them that another CTA adds gets the same bits from both, and
            // one range costs the loops below (and the dequantisation beside them) no registers.  Cut before the wait: nearly always
            // the CTA's own share.
            const uint32_t shares = static_cast<uint32_t>(exchange_shares(ksplit)), items = static_cast<uint32_t>(tokens);
            const uint32_t slice = static_cast<uint32_t>(w.k_slice);
            bars->range = items * slice / shares | items * (slice + 1) / shares << 16;
            const uint32_t mine = exchange_arrive(word, ksplit, w.k_slice, p.patience_ns);
            if (mine == 0) bars->range = 0;
            else if (mine != (slice < kExchangeShares ? 1u << slice : 0u))
                bars->range = items * (__ffs(static_cast<int>(mine)) - 1) / shares | items * (32 - __clz(static_cast<int>(mine))) / shares << 16;
        }
        named_barrier_sync(2, kDequantWarps * 32);
        const int t_begin = static_cast<int>(bars->range & 0xffffu), t_end = static_cast<int>(bars->range >> 16);
        if (t_begin < t_end) {
            __threadfence();
            const long long first_row = static_cast<long long>(w.row_tile) * kBM + 4 * lane;
            const float* partial = p.partial + static_cast<size_t>(w.token0) * n + first_row;
            if (first_row < n) {
                if ((n & 3) == 0) {
                    // a warp per token, four rows per lane, four tokens in flight
                    constexpr int kInFlight = 4;
                    for (int t = t_begin + (worker >> 5); t < t_end; t += kInFlight * kDequantWarps) {
                        const float* from[kInFlight];
                        float4 sum[kInFlight];
#pragma unroll
                        for (int i = 0; i < kInFlight; ++i) {
                            from[i] = partial + static_cast<size_t>(min(t + i * kDequantWarps, t_end - 1)) * n;
                            sum[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                        }
                        for (int z = 0; z < ksplit; ++z) {
                            float4 v[kInFlight];
#pragma unroll
                            for (int i = 0; i < kInFlight; ++i) v[i] = __ldcg(reinterpret_cast<const float4*>(from[i] + z * plane));
#pragma unroll
                            for (int i = 0; i < kInFlight; ++i) {
                                sum[i].x += v[i].x;
                                sum[i].y += v[i].y;
                                sum[i].z += v[i].z;
                                sum[i].w += v[i].w;
                            }
                        }
#pragma unroll
                        for (int i = 0; i < kInFlight; ++i) {
                            if (t + i * kDequantWarps >= t_end) break;
                            const size_t o = static_cast<size_t>(w.token0 + t + i * kDequantWarps) * n + first_row;
                            if (y_bf16) {
                                const __nv_bfloat162 low = __floats2bfloat162_rn(sum[i].x, sum[i].y), high = __floats2bfloat162_rn(sum[i].z, sum[i].w);
                                *reinterpret_cast<uint2*>(static_cast<__nv_bfloat16*>(y) + o) =
                                    make_uint2(*reinterpret_cast<const uint32_t*>(&low), *reinterpret_cast<const uint32_t*>(&high));
                            } else {
                                *reinterpret_cast<float4*>(static_cast<float*>(y) + o) = sum[i];
                            }
                        }
                    }
                } else {   // rows that do not keep 16-byte boundaries
                    for (int t = t_begin + (worker >> 5); t < t_end; t += kDequantWarps) {
                        for (int r = 0; r < 4 && first_row + r < n; ++r) {
                            float sum = 0.0f;
                            for (int z = 0; z < ksplit; ++z) sum += __ldcg(partial + static_cast<size_t>(t) * n + r + z * plane);
                            const size_t o = static_cast<size_t>(w.token0 + t) * n + first_row + r;
                            if (y_bf16) static_cast<__nv_bfloat16*>(y)[o] = __float2bfloat16_rn(sum);
                            else static_cast<float*>(y)[o] = sum;
                        }
                    }
                }
            }
        }
        named_barrier_sync(2, kDequantWarps * 32);   // `range` is free for the next unit
        if (p.patience_ns != 0 && worker == 0) {
            unsigned int* word = bars->word;
            if (exchange_depart(word + p.ticket_stride) == static_cast<unsigned int>(ksplit - 1)) exchange_reset(word, word + p.ticket_stride);
        }
    }
    return ok;
}

// ---------------------------------------------------------------- dequant warps
// Two sets of eight warps take the super-blocks in turn, four warps (128 rows) each half of one: the sets work half a period
// apart, so that the waits and hand-overs of one run under the arithmetic of the other.  A step is complete in registers before
// the thread asks for its stage of the A ring.  A unit's results are stored after the first super-block of the next one: its MMAs
// run meanwhile.
template <uint32_t FMT, bool SMEM_A>
__device__ __forceinline__ bool dequant_warps(const GemmParams& p, uint32_t raw, uint32_t a_tiles, Barriers* bars, uint32_t tmem_base, int rank) {
    using G = TcGeometry<FMT, SMEM_A>;
    const int lane = threadIdx.x & 31;
    const int worker = threadIdx.x - kFirstDequantWarp * 32;
    const int row_in_tile = worker & (kBM - 1), half = (worker >> 7) & 1, set = worker >> 8;
    // Where the row lies in the raw stage, and its super-block's distance from the 16-byte boundary the box starts on.
    uint32_t raw_row = static_cast<uint32_t>(row_in_tile), delta = 0;
    if (FMT == kQ6_K) {
        const int row_class = row_in_tile % p.row_classes;
        raw_row = static_cast<uint32_t>(row_class * (kBM / p.row_classes) + row_in_tile / p.row_classes);
        delta = (static_cast<uint32_t>(row_class) * p.row_bytes) & 15u;
    }
    raw += raw_row * G::kSlot;
    // where the row's 64 halves of step 2 half go: TMEM columns, or, chunk c of row r of a tile, (r / 8) * 1024 + (r % 8) * 128 +
    // ((c ^ (r % 8)) * 16)
    const uint32_t a_slot = SMEM_A ? a_tiles + 2 * half * kATileBytes + (row_in_tile >> 3) * 1024 + (row_in_tile & 7) * 128
                                   : tmem_base + (static_cast<uint32_t>(row_in_tile & ~31) << 16) + kARing + kARingColumns * set + 64 * half;
    const uint32_t raw_full = smem_addr(bars->raw_full), raw_empty = smem_addr(bars->raw_empty), empty = smem_addr(&bars->empty[set][2 * half]);
    const uint32_t full = address_in_first(&bars->full[set][2 * half]);
    const int buffers = acc_buffers(p.nt);
    const int stride = gridDim.x >> 1;
    Ring acc;
    // Super-block b of this CTA's sequence of units lies in raw stage b % kRawStages and belongs to set b % 2.  After a wait that ran out
    // nothing is waited for any more; what is computed then is reported as invalid.
    int base = 0;
    uint32_t polls = kPolls;
    for (int u = blockIdx.x >> 1;; u += stride) {
        const bool end = u >= p.units, first_unit = u < stride;
        const Unit w = unit_at(p, u, rank);
        const int last = base + (end ? 0 : w.sb_count);
        const int mine = base + ((base & 1) != set ? 1 : 0);
        // The set that has the unit's first super-block hands it over before it stores the previous unit's results; the other must
        // not wait for stages that only come free once this unit has an accumulator.
        const int store_at = mine == base ? mine + 2 : mine;
        bool stored = first_unit;
#pragma unroll 1
        for (int b = mine;; b += 2) {
            if (!stored && (b >= last || b == store_at)) {
                if (!store_unit<SMEM_A>(p, u - stride, tmem_base, bars, acc.stage, acc.round & 1, __all_sync(0xffffffffu, polls != 0))) polls = 0;
                acc.advance(buffers);
                stored = true;
            }
            if (b >= last) break;
            if (!mbar_spin(raw_full + 8 * (static_cast<uint32_t>(b) % G::kRawStages), (static_cast<uint32_t>(b) / G::kRawStages) & 1, polls)) polls = 0;
            uint32_t blk = raw + static_cast<uint32_t>(static_cast<uint32_t>(b) % G::kRawStages) * G::kRawStageBytes;
            if (FMT == kQ6_K) blk += (delta + static_cast<uint32_t>(w.sb_begin + b - base) * 210u) & 15u;
            HalfBlock<FMT> data;
            data.load(blk, half);
            if (HalfBlock<FMT>::kHeld) {
                __syncwarp();
                if (lane == 0) mbar_arrive_local(raw_empty + 8 * (static_cast<uint32_t>(b) % G::kRawStages));
            }
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                uint4 out[8];
                if (j == 0) data.template step<0>(out);
                else data.template step<1>(out);
                settle(out);
                if (!HalfBlock<FMT>::kHeld && j == 1) {
                    __syncwarp();
                    if (lane == 0) mbar_arrive_local(raw_empty + 8 * (static_cast<uint32_t>(b) % G::kRawStages));
                }
                // the first super-blocks: the parity of a phase before the first, which passes
                if (!mbar_spin(empty + 8 * j, ((b - G::kADepth) >> 1) & 1, polls)) polls = 0;
                __syncwarp();
                if (SMEM_A) {
#pragma unroll
                    for (uint32_t c = 0; c < 8; ++c) sts128(a_slot + j * kATileBytes + ((c ^ (row_in_tile & 7u)) << 4), out[c]);
                    fence_proxy_async_smem();
                } else {
                    tcgen05_fence_after_sync();
                    tmem_st32(a_slot + 32 * j, out);
                    tcgen05_fence_before_sync();
                }
                __syncwarp();
                if (lane == 0) mbar_arrive_first(full + 8 * j);
            }
        }
        base = last;
        if (end) break;
    }
    return polls != 0;
}

template <uint32_t FMT, bool SMEM_A>
__global__ void __launch_bounds__(kTcThreads, 1) __cluster_dims__(2, 1, 1)
qgemm_tc_kernel(const __grid_constant__ RawMaps wmaps, const __grid_constant__ GemmParams p) {
    using G = TcGeometry<FMT, SMEM_A>;
    extern __shared__ uint8_t smem_raw[];
    // The swizzled tiles need a 1024-byte aligned base, at the same offset in both CTAs.
    uint8_t* smem = smem_raw + ((1024u - (smem_addr(smem_raw) & 1023u)) & 1023u);
    uint8_t* b_tiles = smem;
    uint8_t* a_tiles = b_tiles + G::kBStages * G::kBTileBytes;
    uint8_t* raw = a_tiles + (SMEM_A ? kSlots * kATileBytes : 0);
    Barriers* bars = reinterpret_cast<Barriers*>(raw + G::kRawStages * G::kRawStageBytes);

    // (the shuffle tells the compiler that the warp index is uniform, and with it the branches on it)
    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;
    const int rank = blockIdx.x & 1;
    const int b_bytes = (p.nt / 2) * kBK * 2;
    pdl_launch_dependents();

    if (threadIdx.x == 0) {
        for (int s = 0; s < G::kRawStages; ++s) {
            mbar_init(&bars->raw_full[s], 1);
            mbar_init(&bars->raw_empty[s], kDequantWarps / 2);
        }
        for (int s = 0; s < kSlots; ++s) {
            for (int i = 0; i < 2; ++i) {
                mbar_init(&bars->full[i][s], 8 + 2);
                mbar_init(&bars->empty[i][s], 1);
                mbar_init(&bars->half[i][s], 1);
            }
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&bars->acc_full[s], 1);
            mbar_init(&bars->acc_empty[s], 2 * kDequantWarps);
        }
        mbar_fence_init();
        tma_prefetch_descriptor(&wmaps.map[0]);
    }
    if (warp == kIssuerWarp) tmem_alloc_pair(&bars->tmem, 512);
    tcgen05_fence_before_sync();
    cluster_sync();   // both CTAs' barriers and TMEM are ready
    tcgen05_fence_after_sync();
    constexpr uint32_t tmem_base = 0;   // of an allocation of all 512 columns; a constant keeps the MMAs' operands in uniform registers
    const int first_unit = blockIdx.x >> 1, unit_stride = gridDim.x >> 1;
    bool ok = true;

    if (warp == kProducerWarp) {
        // ---------------- raw weight bytes: they do not depend on the kernel before this one ----------------
        if (lane == 0) {
            const int class_rows = kBM / p.row_classes;
            Ring ring;
            for (int u = first_unit; u < p.units && ok; u += unit_stride) {
                const Unit w = unit_at(p, u, rank);
                for (int i = 0; i < w.sb_count && ok; ++i, ring.advance(G::kRawStages)) {
                    if (ring.round > 0) ok = mbar_spin(&bars->raw_empty[ring.stage], (ring.round - 1) & 1);
                    if (!ok) break;
                    mbar_arrive_expect_tx(&bars->raw_full[ring.stage], G::kRawStageBytes);
                    uint8_t* stage = raw + ring.stage * G::kRawStageBytes;
                    for (int c = 0; c < p.row_classes; ++c) {
                        const unsigned int delta = (static_cast<unsigned int>(c) * p.row_bytes) & 15u;
                        const unsigned int byte_x = (delta + static_cast<unsigned int>(w.sb_begin + i) * Format<FMT>::kBytes) & ~15u;
                        tma_load_2d(stage + c * class_rows * G::kSlot, &wmaps.map[c], static_cast<int>(byte_x / 2), w.row_tile * class_rows,
                                    &bars->raw_full[ring.stage]);
                    }
                }
            }
        }
        __syncwarp();
    } else if (warp == kActivationWarp) {
        // ---------------- this CTA's half of the activation tiles, one stage per K step ----------------
        if (lane == 0) {
            pdl_wait_prior();   // the image is the pre-pass's output
            const size_t step_bytes = static_cast<size_t>(p.row_groups) * kGroupBytes;
            uint32_t blocks = 0;
            int stage = 0;
            for (int u = first_unit; u < p.units && ok; u += unit_stride) {
                const Unit w = unit_at(p, u, rank);
                const uint8_t* source = p.image + static_cast<size_t>(w.sb_begin * kSub) * step_bytes +
                                        static_cast<size_t>((w.token0 + rank * (p.nt / 2)) / 8) * kGroupBytes;
                for (int i = 0; i < w.sb_count && ok; ++i, ++blocks) {
#pragma unroll
                    for (int s = 0; s < kSlots; ++s, source += step_bytes) {
                        // the step kBStages before this one has been multiplied
                        const int before = static_cast<int>(blocks) * kSlots + s - G::kBStages;
                        if (before >= 0) {
                            const int b = before / kSlots;
                            ok = ok && mbar_spin(&bars->empty[(b + G::kADepth) & 1][before % kSlots], (b >> 1) & 1);
                        }
                        if (!ok) break;
                        uint64_t* landed = rank == 0 ? &bars->full[blocks & 1][s] : &bars->half[blocks & 1][s];
                        mbar_arrive_expect_tx(landed, b_bytes);
                        bulk_copy_g2s(b_tiles + stage * G::kBTileBytes, source, b_bytes, landed);
                        stage = stage == G::kBStages - 1 ? 0 : stage + 1;
                    }
                }
            }
        }
        __syncwarp();
    } else if (warp == kIssuerWarp) {
        if (rank == 0) {
            // ---------------- the pair's MMAs ----------------
            // One wait and one commit per step, and no branch on a wait's outcome: the descriptors then stay in uniform registers.
            // (With a barrier per operand and such branches the warp spent 860 clocks per step, 33 moves to uniform registers among
            // them.)
            const uint32_t idesc = umma_instr_desc(2 * kBM, p.nt, /*A f16*/ 0, /*B f16*/ 0);
            const uint64_t desc_b = umma_smem_desc_sw128(smem_addr(b_tiles));
            const uint64_t desc_a = umma_smem_desc_sw128(smem_addr(a_tiles));
            const uint32_t full = smem_addr(&bars->full[0][0]), empty = smem_addr(&bars->empty[0][0]);
            const int buffers = acc_buffers(p.nt);
            uint32_t polls = kPolls;
            Ring acc;
            uint32_t blocks = 0, stage = 0;
            for (int u = first_unit; u < p.units; u += unit_stride) {
                const int sb_count = unit_at(p, u, rank).sb_count;
                // the unit before the last (or the last) has left this accumulator; the first round passes
                polls = mbar_spin(smem_addr(&bars->acc_empty[acc.stage]), (acc.round - 1) & 1, polls) ? polls : 0u;
                tcgen05_fence_after_sync();
                const uint32_t sum0 = acc_column<SMEM_A>(p.nt, acc.stage, 0), sum1 = acc_column<SMEM_A>(p.nt, acc.stage, 1);
                int third = 0;   // step % 3
                for (int i = 0; i < sb_count; ++i, ++blocks) {
                    const uint32_t half_ring = blocks & 1;
                    const uint32_t freed = empty + 8 * kSlots * ((blocks + G::kADepth) & 1);
#pragma unroll
                    for (int s = 0; s < kSlots; ++s) {
                        polls = mbar_spin(full + 8 * (kSlots * half_ring + s), (blocks >> 1) & 1, polls) ? polls : 0u;
                        tcgen05_fence_after_sync();
                        const bool second = p.order == kEvenOdd ? (s & 1) != 0 : p.order == kEveryThird && third == 1;
                        // steps 0 and 1 open the two sums
                        const uint64_t desc = desc_b + stage * (G::kBTileBytes >> 4);
                        if constexpr (SMEM_A)
                            umma_pair_step_elected(second ? sum1 : sum0, desc_a + s * (kATileBytes >> 4), desc, idesc, i > 0 || s > 1, freed + 8 * s);
                        else
                            umma_pair_step_elected(sum0, kARing + kARingColumns * half_ring + 32 * s, desc, idesc, i > 0 || s > 0, freed + 8 * s);
                        stage = stage == G::kBStages - 1 ? 0 : stage + 1;
                        third = third == 2 ? 0 : third + 1;
                    }
                }
                umma_commit_pair_elected(smem_addr(&bars->acc_full[acc.stage]));
                acc.advance(buffers);
            }
            ok = polls != 0;
        } else if (lane == 0) {
            // ---------------- second CTA: its half of the B tile has landed ----------------
            uint32_t blocks = 0;
            for (int u = first_unit; u < p.units && ok; u += unit_stride) {
                const int sb_count = unit_at(p, u, rank).sb_count;
                for (int i = 0; i < sb_count && ok; ++i, ++blocks) {
#pragma unroll
                    for (int s = 0; s < kSlots; ++s) {
                        ok = ok && mbar_spin(&bars->half[blocks & 1][s], (blocks >> 1) & 1);
                        if (ok) mbar_arrive_first(address_in_first(&bars->full[blocks & 1][s]));
                    }
                }
            }
        }
        __syncwarp();
    } else if (warp >= kFirstDequantWarp) {
        ok = dequant_warps<FMT, SMEM_A>(p, smem_addr(raw), smem_addr(a_tiles), bars, tmem_base, rank);
    }
    if (!ok) atomicExch(p.status, kDeviceWaitTimeout);

    // ---------------- teardown: every warp of the pair arrives here, then TMEM is released ----------------
    tcgen05_fence_before_sync();
    __syncwarp();
    cluster_sync();
    if (warp == kIssuerWarp) tmem_dealloc_pair(tmem_base, 512);
}

// Tokens per unit: the tile whose waves of units cost least.  A step of NT tokens takes the tensor pipe 2 NT clocks, and not less
// than kStep: that is what the issuing warp needs for four MMAs, a wait and a commit, and what a stage of an A ring of one
// super-block needs to come back from the other CTA of the pair.  A unit adds the fill of the pipeline, and, where its accumulators
// leave no room for a second unit, its drain and its stores.
int choose_tokens(int m, int row_pairs, int ksplit, int steps, int pairs) {
    constexpr int kStep = 570, kFill = 1500, kDrain = 3000;
    int best = 16;
    double best_cost = 1e30;
    for (int nt = 16; nt <= kMaxTokens; nt += 16) {
        const long long units = static_cast<long long>(row_pairs) * ((m + nt - 1) / nt) * ksplit;
        const double waves = static_cast<double>((units + pairs - 1) / pairs);
        const double unit = static_cast<double>(2 * nt > kStep ? 2 * nt : kStep) * steps + kFill + (nt <= kMaxTokens / 2 ? 0 : kDrain);
        if (waves * unit < best_cost) {
            best_cost = waves * unit;
            best = nt;
        }
    }
    return best;
}

template <uint32_t FMT, bool SMEM_A>
cudaError_t launch_kernel_for(const RawMaps& wmaps, const GemmParams& p, int pairs, cudaStream_t stream) {
    using G = TcGeometry<FMT, SMEM_A>;
    auto kernel = qgemm_tc_kernel<FMT, SMEM_A>;
    static int configured_device = -1;
    int device = 0;
    cudaGetDevice(&device);
    if (configured_device != device) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, G::kSmemBytes);
        if (e != cudaSuccess) return e;
        configured_device = device;
    }
    return launch_kernel(kernel, dim3(2 * (p.units < pairs ? p.units : pairs)), dim3(kTcThreads), G::kSmemBytes, stream, wmaps, p);
}

template <uint32_t FMT>
cudaError_t launch_format(const TcArgs& a) {
    using G = TcGeometry<FMT, false>;
    EncodeTiledFn encode = encode_tiled_fn();
    if (encode == nullptr) return cudaErrorNotSupported;
    if (!a.x_bf16) return cudaErrorInvalidValue;
    GemmParams p{};
    p.nsb = a.k / kSuperBlock;
    const int n_tiles = (a.n + kBM - 1) / kBM;
    p.row_pairs = (n_tiles + 1) / 2;
    // Sums and K ranges follow from the sizes of the call alone.  Up to 128 tokens: even and odd steps; up to 256, and where wide
    // tiles of 512 would leave more than a fifth of the SMs idle: every third; else one sum.  Nothing in this kernel asks for two
    // sums; they are the order of additions of the form it replaced, kept so that results keep their bits, and they cost it the plan
    // with A in tensor memory.
    const long long wide_tiles = static_cast<long long>(n_tiles) * ((a.m + 511) / 512);
    const bool wide = FMT != kQ8_0 && a.m > 256 && wide_tiles * 5 >= static_cast<long long>(a.sm_count) * 4;
    p.order = a.m <= 128 ? kEvenOdd : wide ? kOneSum : kEveryThird;
    int reach = 16;                       // tokens a K range is chosen for
    while (reach < a.m && reach < 256) reach *= 2;
    if (wide) reach = 512;
    const int tiles = n_tiles * ((a.m + reach - 1) / reach);
    const size_t plane_bytes = static_cast<size_t>(a.m) * a.n * sizeof(float);
    const size_t x_bytes = (static_cast<size_t>(a.m) * a.k * 2 + 1023) & ~static_cast<size_t>(1023);
    const size_t factor_bytes = (static_cast<size_t>(a.m) * sizeof(float) + 255) & ~static_cast<size_t>(255);
    const size_t partial_space = a.scratch_bytes > x_bytes + factor_bytes ? a.scratch_bytes - x_bytes - factor_bytes : 0;
    p.ksplit = choose_ksplit(tiles, p.nsb, a.sm_count, plane_bytes, partial_space, a.ticket_count);
    // Hundreds of tokens: a partial tile is megabytes, written and read once more per split.  K is split then only where the tiles
    // leave more than half of the SMs idle.  Measured, unsplit and in two: Q4_K 12288 x 4096, 512 tokens 58.0 and 70.7 us; 5120 x 5120,
    // 512 tokens 38.5 and 50.3; 8192 x 4096, 300 tokens 32.4 and 44.7; Q6_K 4096 x 12288, 900 tokens 87.8 and 102; on the other side of
    // the line Q4_K 4096 x 4096, 300 tokens 30.5 and 25.8; Q6_K 4096 x 12288, 512 tokens 75.7 and 55.3.  Long K is where the line is
    // wrong: Q6_K 5120 x 25600, 512 tokens, 162 unsplit, 140 in three.
    if (a.m > 256 && 2 * tiles > a.sm_count) p.ksplit = 1;
    if (a.force_ksplit > 0 && a.force_ksplit <= p.nsb && plane_bytes * a.force_ksplit <= partial_space) p.ksplit = a.force_ksplit;
    const int pairs = a.sm_count / 2;
    p.nt = choose_tokens(a.m, p.row_pairs, p.ksplit, (p.nsb + p.ksplit - 1) / p.ksplit * kSub, pairs);
    p.m_tiles = (a.m + p.nt - 1) / p.nt;
    // Scratch: [activation tiles, whole token tiles][one factor per token row][split-K partial tiles].
    p.row_groups = p.m_tiles * p.nt / 8;
    const size_t image_bytes = static_cast<size_t>(p.row_groups) * kGroupBytes * (a.k / kBK);
    if (image_bytes + factor_bytes > a.scratch_bytes) return cudaErrorMemoryAllocation;
    if (p.ksplit > 1 && (image_bytes + factor_bytes + plane_bytes * p.ksplit > a.scratch_bytes || 2 * p.row_pairs * p.m_tiles > a.ticket_count)) p.ksplit = 1;
    p.units = p.row_pairs * p.m_tiles * p.ksplit;
    // one round of units: the CTAs of a tile are likely to run at the same time
    p.patience_ns = p.ksplit > 1 && p.units <= pairs && 4 * p.row_pairs * p.m_tiles <= a.ticket_count ? a.patience_ns : 0;
    p.ticket_stride = a.ticket_count / 2;
    uint8_t* image = static_cast<uint8_t*>(a.scratch);
    float* factor = reinterpret_cast<float*>(image + image_bytes);
    p.partial = reinterpret_cast<float*>(image + image_bytes + factor_bytes);
    const cudaError_t converted = launch_kernel(gemm_image_kernel, dim3(a.m), dim3(kImageThreads), 0, a.stream, static_cast<const __nv_bfloat16*>(a.x), image,
                                                factor, a.k, p.row_groups);
    if (converted != cudaSuccess) return converted;
    const unsigned long long row_bytes = static_cast<unsigned long long>(p.nsb) * Format<FMT>::kBytes;
    int classes = 1;
    while ((row_bytes * classes) % 16 != 0) classes *= 2;   // only Q6_K rows can need more than one
    RawMaps wmaps{};
    for (int c = 0; c < classes; ++c) {
        if (c >= a.n) {
            wmaps.map[c] = wmaps.map[0];   // fewer rows than classes: what it brings is never stored
            continue;
        }
        const unsigned long long first = static_cast<unsigned long long>(c) * row_bytes, delta = first & 15ull;
        const cuuint64_t wdims[2] = {static_cast<cuuint64_t>((delta + row_bytes) / 2), (static_cast<cuuint64_t>(a.n) - c + classes - 1) / classes};
        const cuuint64_t wstrides[1] = {static_cast<cuuint64_t>(row_bytes * classes)};
        const cuuint32_t wbox[2] = {G::kSlot / 2, static_cast<cuuint32_t>(kBM / classes)};
        const cuuint32_t elem[2] = {1, 1};
        if (encode(&wmaps.map[c], CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<uint8_t*>(a.weights) + (first - delta), wdims, wstrides, wbox, elem,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return cudaErrorInvalidValue;
    }
    p.row_classes = classes;
    p.row_bytes = static_cast<unsigned int>(row_bytes);
    p.image = image;
    p.x_scale = factor;
    p.y = a.y;
    p.tickets = a.tickets;
    p.n = a.n;
    p.m = a.m;
    p.y_bf16 = a.y_bf16 ? 1 : 0;
    p.status = a.device_status;
    return p.order == kOneSum ? launch_kernel_for<FMT, false>(wmaps, p, pairs, a.stream) : launch_kernel_for<FMT, true>(wmaps, p, pairs, a.stream);
}

}  // namespace

bool qgemm_tc_supports(uint32_t value_type, int k) {
    // Whole 256-element super-blocks only (a Q8_0 row may end inside one; those go to the GEMV kernels).
    return k % kSuperBlock == 0 && (value_type == kQ4_K || value_type == kQ5_K || value_type == kQ6_K || value_type == kQ8_0);
}

cudaError_t launch_qgemm_tc(const TcArgs& a) {
    switch (a.value_type) {
        case kQ4_K: return launch_format<kQ4_K>(a);
        case kQ5_K: return launch_format<kQ5_K>(a);
        case kQ6_K: return launch_format<kQ6_K>(a);
        case kQ8_0: return launch_format<kQ8_0>(a);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace ribn
