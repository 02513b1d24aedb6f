// Dequant-fused GEMV for 1..8 activation rows per launch on the integer tensor-core instruction
// (mma.sync m16n8k32 u8 x s8 for Q4_K and Q5_K, s8 x s8 for Q8_0, m16n8k16 s8 x s8 for Q6_K; s32 accumulate).
//
//   y[m][n] = sum_k dequant(W[n][k]) * x[m][k]
//
// Why a second narrow kernel.  The f16 kernel of gemv_mma.cu turns every pair of quants into a half2 with one
// logic op and one HFMA2 and is bound by instruction issue (about 3.8 thread instructions per weight, the logic
// pipe half busy) at half of the HBM rate.  Here the packed nibbles ARE the operand: (word & 0x0f0f0f0f) is four
// unsigned 8-bit quants, so a weight costs 3/8 of a logic instruction, and nothing is multiplied before the
// tensor core.  What makes that possible:
//   * the activations are 22-bit integers X = rint(x * 2^e) per (member, super-block), 2^e the power of two
//     that brings the largest of the 256 magnitudes into [2^20, 2^21), stored as three 8-bit planes
//     X = 2^14 p2 + 2^7 p1 + p0 (p2 signed, p1 and p0 in 0..127).  The planes of a member are COLUMNS of the
//     same instruction (a column group is two members x [p0 p1 p2 0]), so two members cost one mma per
//     sub-block of 32 weights and eight members four;
//   * one m16n8k32 covers exactly one sub-block (the K order inside it is free, the activations are stored in
//     the order the bytes come in), so its s32 result is multiplied by the 6-bit sub-block scale as an
//     INTEGER (one IMAD per accumulator, on the pipe the unpacking does not use) and the sums over the eight
//     sub-blocks stay exact; d * 2^-e is applied in f32 once per super-block and row;
//   * the minima term (dmin * m_j * sum of the sub-block's activations) is one f16 mma per super-block, as in
//     the f16 kernel: A = the eight minima, B = the block sums as f16 hi + lo.
// Q6_K: scales cover 16 weights, so the instruction is the k16 one; a quant is six bits from two places
// (a nibble and two bits, merged with three logic ops per four weights), and q - 32 is made a signed byte in two
// more (set the top bit, subtract 32 without a borrow between bytes, clear the top bit again), which needs no
// block sums.  Super-blocks are 210 bytes: every second one starts two bytes off a word boundary, and its words
// are funnel-shifted out of two aligned loads.
// Q8_0: the signed instruction; see block_q8.
// What bounds a call: one row of a few megabytes is start-up (1.6 us from the end of the kernel before to the first multiply:
// loads, one conversion per warp, instructions fetched for the first time), then issue slots (about 67 weights per clock and
// SM, HBM delivers 42), then HBM.  So the work is laid out for few barriers and one conversion per SM: one CTA per SM, two groups of
// eight consumer warps that share the image and take row tiles in turn.  Measured, two CTAs of eight warps per SM before:
// Q4_K one row 12288 x 4096 9.6 -> 7.8 us; Q8_0 one row 4096 x 4096 10.9 -> 4.5 us and 12288 x 4096 25.8 -> 10.0 us, Q6_K three
// unaligned rows 1024 x 5120 10.6 -> 6.6 us (both on the integer-dot kernel before).
// Rounding: the weights are exact; an activation carries 2^-22 of its super-block's largest magnitude, all
// integer sums are exact, and a row's result does not depend on the rows launched with it.
//
// Reference counterparts: q*_gemv_warp / _warp_batch (crates/nvidia/src/kernels/quantized/q4_k.cu:103-258,
// q5_k.cu) for the contract; rms_norm (crates/nvidia/src/model_ops.rs:106-147) and silu_mul
// (model_ops.rs:316-328) for the fused prologues.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>

#include "formats.cuh"
#include "internal.h"
#include "pack_activations.cuh"
#include "pipeline.cuh"
#include "row_copy.h"
#include "tc_host.h"
#include "tcgen05.cuh"
#include "unpack.cuh"

namespace ribn {
namespace {

constexpr int kGroupWarps = 8;                 // warps of a consumer group = super-blocks per stage
constexpr int kGroups = 2;                     // consumer groups of a CTA
constexpr int kConsumerWarps = kGroups * kGroupWarps;
constexpr int kConsumers = kConsumerWarps * 32;
constexpr int kThreads = kConsumers + 32;      // + the producer warp
constexpr int kTileRows = 16;                  // weight rows per tile (the M of m16n8k32)
constexpr int kMaxStages = 8;                // of a CTA: in one ring, or in two (one per group) of half as many
constexpr int kMaxSlots = 5;                   // tiles of a group whose partial sums may be waiting for their finisher
constexpr int kMaxMembers = 8;                 // four column groups of two members
constexpr int kSliceBytes = 768;               // image bytes per (member, super-block): 8 sub-blocks x 3 planes x 32
constexpr int kZeroBytes = 1024;               // zeros the fourth column of every member (and absent members) read

// How the weight rows reach shared memory.
//   kBoxes: tiled TMA, every row on a 16-byte boundary;
//   kRowsEven: one bulk copy per row and box from the boundary below (Q6_K rows of an even number of super-blocks start on a
//          word, so whether a super-block starts on a word is the same for all rows);
//   kRowsOdd: the same for rows that start two bytes off a word in some lanes and on it in others.
enum Fetch { kBoxes = 0, kRowsEven = 1, kRowsOdd = 2 };

template <uint32_t FMT, int FETCH>
struct ImmaPlan {
    // bytes of 256 weights: one super-block, or eight blocks of Q8_0
    static constexpr int kSbBytes = Format<FMT>::kBytes;
    // Super-blocks per box, and bytes from one row of a box to the next (in 4-byte words, mod 32, below): long rows, because the
    // copy engine works in rows, and a pitch that spreads a warp's loads over the banks.  Q4_K / Q5_K: eight, 1184 / 1440
    // bytes = 8 words, so that the 64-bit loads of four rows x four lanes fall on 32 different banks.  Q6_K: eight, 1680
    // bytes = 4, or 1712 = 12 with room for a row that starts up to 14 bytes behind the boundary its copy starts at; Q8_0:
    // four, 1104 = 20: the 32-bit loads of eight rows x four lanes on 32 banks.
    static constexpr int kBoxSb = FMT == kQ8_0 ? 4 : 8;
    static constexpr int kBoxesPerStage = kGroupWarps / kBoxSb;
    static constexpr int kBoxSpan = kBoxSb * kSbBytes;   // bytes of a row from one box to the next
    static constexpr int kRowPitch = FMT == kQ8_0 ? kBoxSpan + 16 : FMT == kQ6_K && FETCH == kBoxes ? kBoxSpan : kBoxSpan + 32;
    static constexpr int kBoxBytes = kTileRows * kRowPitch;
    static constexpr int kStageBytes = kBoxesPerStage * kBoxBytes;
    static_assert(kRowPitch % 16 == 0 && kBoxBytes % 128 == 0, "box: 16-byte rows, 128-byte aligned destination");
    static_assert(kBoxSpan % 16 == 0, "every box of a row starts as far from a 16-byte boundary as the row does");
    static_assert(FETCH == kBoxes || FMT == kQ6_K || FMT == kQ8_0, "rows of the other formats are multiples of 16 bytes");
};

struct ImmaParams {
    const void* x;              // [members][k] (swiglu: [members][2k]) f32 or bf16; unused when `image` is set
    int x_bf16;
    int mode;                   // 0 plain, 1 RMSNorm first, 2 silu(gate) * up
    const float* norm_weight;
    float eps;
    const uint8_t* image;       // activation image made by the pre-pass (layout below), or null: convert here
    int rotated;                // Q8_0 in boxes: even blocks of the image start at their third element
    const uint8_t* weights;
    unsigned long long row_bytes, weight_bytes;
    void* y;
    int y_bf16;
    int accumulate;
    int k, n, nsb, members;
    int stages, rings;          // stages per ring, and rings: the consumer groups that take tiles
    int slots;                  // partial-sum slots per consumer group
    int tile_quotient, tile_remainder;   // tiles per CTA, and how many CTAs have one more
    int* status;
};

// ---------------------------------------------------------------- activation image
// Per call, in shared memory (and in global memory when a pre-pass makes it):
//   planes [members][nsb][8 sub-blocks][p0 32 B | p1 32 B | p2 32 B] int8, bytes in element order.  The 64-bit
//          fragment loads of a half-warp (one member: three planes and the zero column, four lanes each) then
//          cover 96 contiguous bytes plus 32 bytes of the zero area placed 96 bytes further on: 32 banks.
//          Rotated (Q8_0 blocks fetched in boxes): blocks 0, 2, 4, 6 hold elements 2 .. 31, 0, 1 -- see superblock_q8;
//   sums   [members][nsb][16] f16: (sum of the sub-block's 32 integers) / 2^11 as f16 hi (8 values) then f16 lo (8);
//   scale  [nsb][8] f32: 2^-e per (super-block, member), 0 for an all-zero slice, NaN when it holds a non-finite value.
__host__ __device__ inline size_t image_plane_bytes(int members, int nsb) { return static_cast<size_t>(members) * nsb * kSliceBytes; }
__host__ __device__ inline size_t image_sums_bytes(int members, int nsb) { return static_cast<size_t>(members) * nsb * 32; }
__host__ __device__ inline size_t image_scale_bytes(int nsb) { return static_cast<size_t>(nsb) * 32; }
__host__ __device__ inline size_t image_bytes(int members, int nsb) {
    return image_plane_bytes(members, nsb) + image_sums_bytes(members, nsb) + image_scale_bytes(nsb);
}

__device__ __forceinline__ AnyRow member_row(const ImmaParams& p, int m) {
    const size_t row_elements = static_cast<size_t>(p.k) * (p.mode == 2 ? 2 : 1);
    return AnyRow{static_cast<const uint8_t*>(p.x) + static_cast<size_t>(m) * row_elements * (p.x_bf16 ? 2 : 4), p.x_bf16};
}

// Lane `lane` of a warp loads elements 8 lane .. 8 lane + 7 of super-block sb (zeros behind the end of a row), and what the
// prologue multiplies them by: the norm weights (mode 1) or the row's second half (mode 2).
__device__ __forceinline__ void load_slice(const ImmaParams& p, int m, int sb, int lane, float (&v)[8], float (&by)[8]) {
    const int k0 = sb * kSuperBlock + lane * 8;
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = 0.0f;
    if (k0 >= p.k) return;
    const AnyRow row = member_row(p, m);
    load_row8(row + k0, v);
    if (p.mode != 0) load_row8(p.mode == 1 ? AnyRow{reinterpret_cast<const uint8_t*>(p.norm_weight), 0} + k0 : row + (p.k + k0), by);
}
// The prologue: x * inv_rms * norm weight, or silu(gate) * up.
__device__ __forceinline__ void apply_prologue(const ImmaParams& p, float inv_rms, float (&v)[8], const float (&by)[8]) {
    if (p.mode == 1) {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = v[j] * inv_rms * by[j];
    } else if (p.mode == 2) {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = (v[j] / (1.0f + expf(-v[j]))) * by[j];
    }
}

// The warp's 256 values -> three int8 planes, block sums and the slice's factor (generic pointers: shared or global).
__device__ __forceinline__ void store_slice(bool rotated, int m, int sb, int lane, float (&v)[8], uint8_t* planes_row, __half* sums_row, float* scale) {
    // Largest magnitude in one warp reduction: non-negative floats order like their bit patterns, and infinities
    // and NaNs (0x7f800000 and above) come out on top, which is how they are detected.
    uint32_t biggest = 0u;
#pragma unroll
    for (int j = 0; j < 8; ++j) biggest = max(biggest, __float_as_uint(fabsf(v[j])));
    biggest = __reduce_max_sync(0xffffffffu, biggest);
    const bool bad = biggest >= 0x7f800000u;
    // amax * 2^e in [2^20, 2^21); e clamped so that both 2^e and 2^-e are normal numbers
    int e = 20 - (static_cast<int>(biggest >> 23) - 127);
    e = max(-100, min(100, e));
    float down = __uint_as_float(static_cast<uint32_t>(127 + e) << 23);
    float up = __uint_as_float(static_cast<uint32_t>(127 - e) << 23);
    if (biggest == 0u) up = 0.0f;
    if (bad) {
        down = 0.0f;
        up = __int_as_float(0x7fc00000);
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = 0.0f;
    }
    int xi[8], sum = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        xi[j] = max(-2097151, min(2097151, __float2int_rn(v[j] * down)));
        sum += xi[j];
    }
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    const int j = lane >> 2, t = lane & 3;
    if (rotated) {
        // even blocks move by two elements: the lane's last two come from the next lane of the block
        const int next = (lane & ~3) | ((lane + 1) & 3);
        const int n0 = __shfl_sync(0xffffffffu, xi[0], next), n1 = __shfl_sync(0xffffffffu, xi[1], next);
        if ((j & 1) == 0) {
#pragma unroll
            for (int i = 0; i < 6; ++i) xi[i] = xi[i + 2];
            xi[6] = n0;
            xi[7] = n1;
        }
    }
    uint8_t* slot = planes_row + static_cast<size_t>(sb) * kSliceBytes + j * 96 + 8 * t;
    *reinterpret_cast<uint2*>(slot) = make_uint2(pack4(xi[0] & 127, xi[1] & 127, xi[2] & 127, xi[3] & 127),
                                                 pack4(xi[4] & 127, xi[5] & 127, xi[6] & 127, xi[7] & 127));
    *reinterpret_cast<uint2*>(slot + 32) = make_uint2(pack4((xi[0] >> 7) & 127, (xi[1] >> 7) & 127, (xi[2] >> 7) & 127, (xi[3] >> 7) & 127),
                                                      pack4((xi[4] >> 7) & 127, (xi[5] >> 7) & 127, (xi[6] >> 7) & 127, (xi[7] >> 7) & 127));
    *reinterpret_cast<uint2*>(slot + 64) = make_uint2(pack4(xi[0] >> 14, xi[1] >> 14, xi[2] >> 14, xi[3] >> 14),
                                                      pack4(xi[4] >> 14, xi[5] >> 14, xi[6] >> 14, xi[7] >> 14));
    if (t == 0) {
        const float s = static_cast<float>(sum) * 0.00048828125f;   // 2^-11: below the f16 range's top
        const __half hi = __float2half_rn(s);
        sums_row[sb * 16 + j] = hi;
        sums_row[sb * 16 + 8 + j] = __float2half_rn(s - __half2float(hi));
    }
    if (lane == 0) scale[sb * 8 + m] = up;
}

// sum of squares of member row m over the whole K range, by `threads` threads with index tid; the caller reduces.
__device__ __forceinline__ float partial_square_sum(const ImmaParams& p, int m, int tid, int threads) {
    const AnyRow row = member_row(p, m);
    float acc = 0.0f;
#pragma unroll 2
    for (int c = tid; c < p.k / 8; c += threads) {
        float v[8];
        load_row8(row + c * 8, v);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc = fmaf(v[j], v[j], acc);
    }
    return acc;
}

// D = A(16x32, s8, row) * B(32x8, s8, col), s32: the instruction of imma_zero with signed weights.
__device__ __forceinline__ void imma_signed_zero(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}

// D = A(16x32, u8, row) * B(32x8, s8, col), s32.  Lane (g = lane / 4, t = lane % 4) holds
//   a0: row g, K slots 4t..4t+3     a1: row g+8, same slots     a2: row g, K slots 16+4t..     a3: row g+8
//   b0: column g, K slots 4t..4t+3  b1: column g, K slots 16+4t..
//   c0,c1: row g, columns 2t,2t+1   c2,c3: row g+8, columns 2t,2t+1
__device__ __forceinline__ void imma_zero(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}
__device__ __forceinline__ void hmma_zero(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f));
}

// D = A(16x16, s8, row) * B(16x8, s8, col), s32.  Lane (g, t): a0 row g, a1 row g+8, K slots 4t..4t+3; b0 column g, the same slots.
__device__ __forceinline__ void imma16_zero(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
                 : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
                 : "r"(a0), "r"(a1), "r"(b0), "r"(0));
}

// A 32-bit word of shared memory at `address`: on a word boundary, two bytes past one, or one of the two by lane.
enum Parity { kEven = 0, kOdd = 1, kMixed = 2 };
template <int PARITY>
__device__ __forceinline__ uint32_t lds32_shifted(uint32_t address) {
    if (PARITY == kEven) return lds32(address);
    if (PARITY == kOdd) return __funnelshift_r(lds32(address - 2), lds32(address + 2), 16);
    const uint32_t word = address & ~3u;
    return __funnelshift_r(lds32(word), lds32(word + 4), (address & 3u) * 8u);
}

// Per-lane shared addresses at the super-block the warp works on.  Column g of column group q is plane g & 3 of
// member 2q + (g >> 2); the fourth plane and members the launch does not have are read from the zero area.
template <int GROUPS>
struct LaneX {
    uint32_t x[GROUPS];      // the lane's 8 bytes of sub-block j in group q: x[q] + 96 j
    uint32_t step[GROUPS];   // bytes from one super-block to the next (0 for lanes that read zeros)
    uint32_t sums;           // block sums of member g (the minima instruction has one column per member)
    uint32_t scale;          // the eight factors of the super-block

    __device__ __forceinline__ void advance(int superblocks) {
#pragma unroll
        for (int q = 0; q < GROUPS; ++q) x[q] += static_cast<uint32_t>(superblocks) * step[q];
        sums += static_cast<uint32_t>(superblocks * 32);
        scale += static_cast<uint32_t>(superblocks * 32);
    }
};

template <int J>
__device__ __forceinline__ uint32_t scale_byte(uint32_t lo, uint32_t hi) {
    return __byte_perm(J < 4 ? lo : hi, 0u, 0x4440u + (J & 3));
}

// Fifth bit of sub-block J from the lane's fifth-bit word (bit J of every byte) into bit 4 of every byte of `nibbles`.
template <int J>
__device__ __forceinline__ uint32_t with_fifth(uint32_t nibbles, uint32_t h) {
    const uint32_t moved = J < 4 ? (h << (4 - J)) : (h >> (J - 4));
    return and_or(moved, 0x10101010u, nibbles);
}

// One sub-block: the four A words are ready; multiply by every column group, then fold the 6-bit scales in as integers.
template <int J, int GROUPS>
__device__ __forceinline__ void subblock(uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, const LaneX<GROUPS>& lx, uint32_t sc_lo0,
                                         uint32_t sc_hi0, uint32_t sc_lo1, uint32_t sc_hi1, int (&total)[GROUPS][4]) {
    const int s0 = static_cast<int>(scale_byte<J>(sc_lo0, sc_hi0)), s1 = static_cast<int>(scale_byte<J>(sc_lo1, sc_hi1));
#pragma unroll
    for (int q = 0; q < GROUPS; ++q) {
        const uint2 b = lds64_at<96 * J>(lx.x[q]);
        int c[4];
        imma_zero(c, a0, a1, a2, a3, b.x, b.y);
        total[q][0] += s0 * c[0];
        total[q][1] += s0 * c[1];
        total[q][2] += s1 * c[2];
        total[q][3] += s1 * c[3];
    }
}

// One super-block of rows g (at p0) and g + 8 (at p1).
//   acc[q][0], acc[q][1]: rows g, g + 8 of member 2q + (t >> 1), the share of planes p0, p1 (t even) or of plane p2 (t odd);
//   mins[0..3]: the minima term of members 2t, 2t + 1 for row g, then for row g + 8.
template <uint32_t FMT, int GROUPS>
__device__ __forceinline__ void superblock(uint32_t p0, uint32_t p1, const LaneX<GROUPS>& lx, int t, float (&acc)[GROUPS][2], float (&mins)[4]) {
    constexpr uint32_t kQuantOffset = FMT == kQ4_K ? 16 : 48;   // Q5_K: 32 fifth-bit bytes between the header and the nibbles
    const uint4 h0 = lds128(p0), h1 = lds128(p1);   // d | dmin, 12 scale bytes
    uint32_t sc_lo0, sc_hi0, m_lo0, m_hi0, sc_lo1, sc_hi1, m_lo1, m_hi1;
    unpack_k_scales(h0.y, h0.z, h0.w, sc_lo0, sc_hi0, m_lo0, m_hi0);
    unpack_k_scales(h1.y, h1.z, h1.w, sc_lo1, sc_hi1, m_lo1, m_hi1);
    float cm[4];
    {
        // minimum term: A = the eight 6-bit minima, twice (K slots 0..7 and 8..15); B = column g: member g's block
        // sums, f16 hi in slots 0..7 and f16 lo in slots 8..15
        const uint32_t a0 = byte_pair_half2((t & 2) ? m_hi0 : m_lo0, (t & 1) != 0);
        const uint32_t a1 = byte_pair_half2((t & 2) ? m_hi1 : m_lo1, (t & 1) != 0);
        const uint32_t b0 = lds32(lx.sums + t * 4);
        const uint32_t b1 = lds32(lx.sums + 16 + t * 4);
        hmma_zero(cm, a0, a1, a0, a1, b0, b1);
    }
    uint2 f0 = make_uint2(0u, 0u), f1 = f0;
    if (FMT == kQ5_K) {
        f0 = lds64(p0 + 16 + 8 * t);
        f1 = lds64(p1 + 16 + 8 * t);
    }
    // Q4_K, up to two column groups: the high nibbles go to the instruction where they stand, as sixteen times the quants, and their
    // sums are kept apart (integers: 16 * low + high is sixteen times the sum, to the bit).  The logic pipe is what the loop is
    // bound by, and the four shifts per pair were a sixth of its work.
    constexpr bool kInPlace = FMT == kQ4_K && GROUPS <= 2;
    int total[GROUPS][4], high[GROUPS][4];
#pragma unroll
    for (int q = 0; q < GROUPS; ++q)
#pragma unroll
        for (int i = 0; i < 4; ++i) total[q][i] = high[q][i] = 0;
#define RIBN_IMMA_PAIR(G)                                                                                                      \
    {                                                                                                                          \
        const uint2 q0 = lds64(p0 + kQuantOffset + 32 * (G) + 8 * t), q1 = lds64(p1 + kQuantOffset + 32 * (G) + 8 * t);  \
        uint32_t a0 = q0.x & 0x0f0f0f0fu, a1 = q1.x & 0x0f0f0f0fu, a2 = q0.y & 0x0f0f0f0fu, a3 = q1.y & 0x0f0f0f0fu;           \
        if (FMT == kQ5_K) {                                                                                                    \
            a0 = with_fifth<2 * (G)>(a0, f0.x);                                                                                \
            a1 = with_fifth<2 * (G)>(a1, f1.x);                                                                                \
            a2 = with_fifth<2 * (G)>(a2, f0.y);                                                                                \
            a3 = with_fifth<2 * (G)>(a3, f1.y);                                                                                \
        }                                                                                                                      \
        subblock<2 * (G), GROUPS>(a0, a1, a2, a3, lx, sc_lo0, sc_hi0, sc_lo1, sc_hi1, total);                                  \
        if (kInPlace) {                                                                                                        \
            a0 = q0.x & 0xf0f0f0f0u;                                                                                           \
            a1 = q1.x & 0xf0f0f0f0u;                                                                                           \
            a2 = q0.y & 0xf0f0f0f0u;                                                                                           \
            a3 = q1.y & 0xf0f0f0f0u;                                                                                           \
        } else {                                                                                                               \
            a0 = (q0.x >> 4) & 0x0f0f0f0fu;                                                                                    \
            a1 = (q1.x >> 4) & 0x0f0f0f0fu;                                                                                    \
            a2 = (q0.y >> 4) & 0x0f0f0f0fu;                                                                                    \
            a3 = (q1.y >> 4) & 0x0f0f0f0fu;                                                                                    \
        }                                                                                                                      \
        if (FMT == kQ5_K) {                                                                                                    \
            a0 = with_fifth<2 * (G) + 1>(a0, f0.x);                                                                            \
            a1 = with_fifth<2 * (G) + 1>(a1, f1.x);                                                                            \
            a2 = with_fifth<2 * (G) + 1>(a2, f0.y);                                                                            \
            a3 = with_fifth<2 * (G) + 1>(a3, f1.y);                                                                            \
        }                                                                                                                      \
        subblock<2 * (G) + 1, GROUPS>(a0, a1, a2, a3, lx, sc_lo0, sc_hi0, sc_lo1, sc_hi1, kInPlace ? high : total);                              \
    }
    RIBN_IMMA_PAIR(0)
    RIBN_IMMA_PAIR(1)
    RIBN_IMMA_PAIR(2)
    RIBN_IMMA_PAIR(3)
#undef RIBN_IMMA_PAIR
    if (kInPlace) {
#pragma unroll
        for (int q = 0; q < GROUPS; ++q)
#pragma unroll
            for (int i = 0; i < 4; ++i) total[q][i] = 16 * total[q][i] + high[q][i];
    }
    const float d0 = f16_bits_to_f32(h0.x & 0xffffu), dm0 = f16_bits_to_f32(h0.x >> 16);
    const float d1 = f16_bits_to_f32(h1.x & 0xffffu), dm1 = f16_bits_to_f32(h1.x >> 16);
    // Columns 2t, 2t+1 of a group: planes (p0, p1) of its first or second member for t = 0, 2; (p2, zeros) for t = 1, 3.
    const float weight = ((t & 1) ? 16384.0f : 1.0f) * (kInPlace ? 0.0625f : 1.0f);
#pragma unroll
    for (int q = 0; q < GROUPS; ++q) {
        const float xs = __uint_as_float(lds32(lx.scale + 8 * q + 4 * (t >> 1))) * weight;
        const float v0 = fmaf(128.0f, static_cast<float>(total[q][1]), static_cast<float>(total[q][0]));
        const float v1 = fmaf(128.0f, static_cast<float>(total[q][3]), static_cast<float>(total[q][2]));
        acc[q][0] = fmaf(d0 * xs, v0, acc[q][0]);
        acc[q][1] = fmaf(d1 * xs, v1, acc[q][1]);
    }
    // the minima instruction: columns 2t, 2t+1 = members 2t, 2t+1; its sums were divided by 2^11
    const uint2 xm = lds64(lx.scale + 8 * t);
    const float xa = __uint_as_float(xm.x) * -2048.0f, xb = __uint_as_float(xm.y) * -2048.0f;
    mins[0] = fmaf(dm0 * xa, cm[0], mins[0]);
    mins[1] = fmaf(dm0 * xb, cm[1], mins[1]);
    mins[2] = fmaf(dm1 * xa, cm[2], mins[2]);
    mins[3] = fmaf(dm1 * xb, cm[3], mins[3]);
}

// ---- Q6_K.  Block b = 8 n2 + 2 v + h of the sixteen 16-weight blocks: positions 128 n2 + 32 v + 16 h .. + 15, low nibbles
// in ql byte 64 n2 + 32 (v & 1) + 16 h + l (the low half of the byte for v < 2, the high half above), two more bits in
// qh byte 32 n2 + 16 h + l at bit 2 v; lane t takes l = 4t .. 4t + 3 of every block, one word of each.
template <int V>
__device__ __forceinline__ uint32_t q6_signed_bytes(uint32_t ql_word, uint32_t qh_word) {
    // 128 + nibble in every byte, then bits 4..5 from qh: 128 + q; minus 32 without a borrow between bytes; top bit off again
    const uint32_t nibbles = and_or(V < 2 ? ql_word : (ql_word >> 4), 0x0f0f0f0fu, 0x80808080u);
    const uint32_t moved = V == 0 ? (qh_word << 4) : V == 1 ? (qh_word << 2) : V == 2 ? qh_word : (qh_word >> 2);
    return (and_or(moved, 0x30303030u, nibbles) - 0x20202020u) ^ 0x80808080u;
}

// Byte I of `word` as a sign-extended integer: prmt with the replicate-sign bit of the selector set for the three upper
// bytes (the __byte_perm intrinsic keeps only the byte index of a selector nibble).
template <int I>
__device__ __forceinline__ int signed_byte(uint32_t word) {
    int value;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(value) : "r"(word), "r"(0u), "n"(I | ((I | 8) << 4) | ((I | 8) << 8) | ((I | 8) << 12)));
    return value;
}

template <int B, int GROUPS>
__device__ __forceinline__ void block_q6(uint32_t a0, uint32_t a1, const LaneX<GROUPS>& lx, uint32_t scales0, uint32_t scales1,
                                         int (&total)[GROUPS][4]) {
    const int s0 = signed_byte<B & 3>(scales0), s1 = signed_byte<B & 3>(scales1);
#pragma unroll
    for (int q = 0; q < GROUPS; ++q) {
        uint32_t b0;
        asm volatile("ld.shared.u32 %0, [%1+%2];" : "=r"(b0) : "r"(lx.x[q]), "n"(96 * (B >> 1) + 16 * (B & 1)));
        int c[4];
        imma16_zero(c, a0, a1, b0);
        total[q][0] += s0 * c[0];
        total[q][1] += s0 * c[1];
        total[q][2] += s1 * c[2];
        total[q][3] += s1 * c[3];
    }
}

// The two blocks that share the ql word (N2, VLOW, H): block B = 8 N2 + 2 VLOW + H from its low nibbles, block B + 4 from
// its high nibbles.
template <int N2, int H, int VLOW, int GROUPS, int PARITY>
__device__ __forceinline__ void blocks_q6(uint32_t p0, uint32_t p1, uint32_t qh0, uint32_t qh1, uint32_t lane_bytes, const LaneX<GROUPS>& lx,
                                          const uint32_t (&sc0)[4], const uint32_t (&sc1)[4], int (&total)[GROUPS][4]) {
    constexpr int B = 8 * N2 + 2 * VLOW + H;
    const uint32_t ql0 = lds32_shifted<PARITY>(p0 + 64 * N2 + 32 * VLOW + 16 * H + lane_bytes);
    const uint32_t ql1 = lds32_shifted<PARITY>(p1 + 64 * N2 + 32 * VLOW + 16 * H + lane_bytes);
    block_q6<B, GROUPS>(q6_signed_bytes<VLOW>(ql0, qh0), q6_signed_bytes<VLOW>(ql1, qh1), lx, sc0[B >> 2], sc1[B >> 2], total);
    block_q6<B + 4, GROUPS>(q6_signed_bytes<VLOW + 2>(ql0, qh0), q6_signed_bytes<VLOW + 2>(ql1, qh1), lx, sc0[(B + 4) >> 2], sc1[(B + 4) >> 2],
                            total);
}

// The four blocks that share the qh word (N2, H).
template <int N2, int H, int GROUPS, int PARITY>
__device__ __forceinline__ void quarter_q6(uint32_t p0, uint32_t p1, uint32_t lane_bytes, const LaneX<GROUPS>& lx, const uint32_t (&sc0)[4],
                                           const uint32_t (&sc1)[4], int (&total)[GROUPS][4]) {
    const uint32_t qh0 = lds32_shifted<PARITY>(p0 + 128 + 32 * N2 + 16 * H + lane_bytes);
    const uint32_t qh1 = lds32_shifted<PARITY>(p1 + 128 + 32 * N2 + 16 * H + lane_bytes);
    blocks_q6<N2, H, 0, GROUPS, PARITY>(p0, p1, qh0, qh1, lane_bytes, lx, sc0, sc1, total);
    blocks_q6<N2, H, 1, GROUPS, PARITY>(p0, p1, qh0, qh1, lane_bytes, lx, sc0, sc1, total);
}

// One Q6_K super-block of rows g (at p0) and g + 8 (at p1); PARITY: where they start with respect to a word.
template <int GROUPS, int PARITY>
__device__ __forceinline__ void superblock_q6(uint32_t p0, uint32_t p1, const LaneX<GROUPS>& lx, int t, float (&acc)[GROUPS][2]) {
    int total[GROUPS][4];
#pragma unroll
    for (int q = 0; q < GROUPS; ++q)
#pragma unroll
        for (int i = 0; i < 4; ++i) total[q][i] = 0;
    const uint32_t lane_bytes = 4u * static_cast<uint32_t>(t);
    // the sixteen scale bytes of each row: word i holds blocks 4i .. 4i + 3
    uint32_t sc0[4], sc1[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        sc0[i] = lds32_shifted<PARITY>(p0 + 192 + 4 * i);
        sc1[i] = lds32_shifted<PARITY>(p1 + 192 + 4 * i);
    }
    quarter_q6<0, 0, GROUPS, PARITY>(p0, p1, lane_bytes, lx, sc0, sc1, total);
    quarter_q6<0, 1, GROUPS, PARITY>(p0, p1, lane_bytes, lx, sc0, sc1, total);
    quarter_q6<1, 0, GROUPS, PARITY>(p0, p1, lane_bytes, lx, sc0, sc1, total);
    quarter_q6<1, 1, GROUPS, PARITY>(p0, p1, lane_bytes, lx, sc0, sc1, total);
    const float d0 = f16_bits_to_f32(lds_u16(p0 + 208)), d1 = f16_bits_to_f32(lds_u16(p1 + 208));
    const float weight = (t & 1) ? 16384.0f : 1.0f;
#pragma unroll
    for (int q = 0; q < GROUPS; ++q) {
        const float xs = __uint_as_float(lds32(lx.scale + 8 * q + 4 * (t >> 1))) * weight;
        const float v0 = fmaf(128.0f, static_cast<float>(total[q][1]), static_cast<float>(total[q][0]));
        const float v1 = fmaf(128.0f, static_cast<float>(total[q][3]), static_cast<float>(total[q][2]));
        acc[q][0] = fmaf(d0 * xs, v0, acc[q][0]);
        acc[q][1] = fmaf(d1 * xs, v1, acc[q][1]);
    }
}

// ---- Q8_0: eight blocks of a 2-byte factor and 32 signed bytes stand for a super-block.  Blocks are 34 bytes, so in rows
// that start on a word the quants of even blocks sit two bytes off a word and those of odd blocks on one.
// An even block is taken as the words it does have: lane t takes words 1 + t and 5 + t behind the block's start; the last of
// them, which lane 3 would share with the next block, is merged with the two quants behind the factor -- the K order
// 2 .. 31, 0, 1 that the rotated image has for these blocks.
// kRowsOdd: rows start anywhere; two words and a shift per operand word, image in plain order.
template <int J, int GROUPS, bool ODD_ROWS>
__device__ __forceinline__ void block_q8(uint32_t p0, uint32_t p1, const LaneX<GROUPS>& lx, int t, bool real, float (&sum)[GROUPS][2]) {
    uint32_t a[2][2];
    float d[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const uint32_t block = (r == 0 ? p0 : p1) + 34 * J;
        if constexpr (ODD_ROWS) {
            const uint32_t start = block + 2 + 4 * static_cast<uint32_t>(t), word = start & ~3u, shift = (start & 3u) * 8u;
            a[r][0] = __funnelshift_r(lds32(word), lds32(word + 4), shift);
            a[r][1] = __funnelshift_r(lds32(word + 16), lds32(word + 20), shift);
            d[r] = real ? f16_bits_to_f32(lds_u16(block)) : 0.0f;
        } else if constexpr ((J & 1) == 0) {
            const uint32_t first = lds32(block);   // factor, quants 0 and 1
            a[r][0] = lds32(block + 4 + 4 * static_cast<uint32_t>(t));
            const uint32_t last = lds32(block + 20 + 4 * static_cast<uint32_t>(t));
            a[r][1] = t == 3 ? __byte_perm(last, first, 0x7610) : last;
            d[r] = f16_bits_to_f32(first & 0xffffu);
        } else {
            a[r][0] = lds32(block + 2 + 4 * static_cast<uint32_t>(t));
            a[r][1] = lds32(block + 18 + 4 * static_cast<uint32_t>(t));
            d[r] = f16_bits_to_f32(lds_u16(block));
        }
    }
#pragma unroll
    for (int q = 0; q < GROUPS; ++q) {
        uint32_t b0, b1;
        asm volatile("ld.shared.u32 %0, [%1+%2];" : "=r"(b0) : "r"(lx.x[q]), "n"(96 * J));
        asm volatile("ld.shared.u32 %0, [%1+%2];" : "=r"(b1) : "r"(lx.x[q]), "n"(96 * J + 16));
        int c[4];
        imma_signed_zero(c, a[0][0], a[1][0], a[0][1], a[1][1], b0, b1);
        // columns 2t, 2t + 1: planes p0 and p1 (t even, below 2^27 together), or p2 and zeros
        sum[q][0] = fmaf(d[0], static_cast<float>(c[0] + 128 * c[1]), sum[q][0]);
        sum[q][1] = fmaf(d[1], static_cast<float>(c[2] + 128 * c[3]), sum[q][1]);
    }
}

// One group of eight Q8_0 blocks of rows g (at p0) and g + 8 (at p1); `blocks`: how many of them the row has.
template <int GROUPS, bool ODD_ROWS>
__device__ __forceinline__ void superblock_q8(uint32_t p0, uint32_t p1, const LaneX<GROUPS>& lx, int t, int blocks, float (&acc)[GROUPS][2]) {
    float sum[GROUPS][2];
#pragma unroll
    for (int q = 0; q < GROUPS; ++q) sum[q][0] = sum[q][1] = 0.0f;
    block_q8<0, GROUPS, ODD_ROWS>(p0, p1, lx, t, 0 < blocks, sum);
    block_q8<1, GROUPS, ODD_ROWS>(p0, p1, lx, t, 1 < blocks, sum);
    block_q8<2, GROUPS, ODD_ROWS>(p0, p1, lx, t, 2 < blocks, sum);
    block_q8<3, GROUPS, ODD_ROWS>(p0, p1, lx, t, 3 < blocks, sum);
    block_q8<4, GROUPS, ODD_ROWS>(p0, p1, lx, t, 4 < blocks, sum);
    block_q8<5, GROUPS, ODD_ROWS>(p0, p1, lx, t, 5 < blocks, sum);
    block_q8<6, GROUPS, ODD_ROWS>(p0, p1, lx, t, 6 < blocks, sum);
    block_q8<7, GROUPS, ODD_ROWS>(p0, p1, lx, t, 7 < blocks, sum);
    const float weight = (t & 1) ? 16384.0f : 1.0f;
#pragma unroll
    for (int q = 0; q < GROUPS; ++q) {
        const float xs = __uint_as_float(lds32(lx.scale + 8 * q + 4 * (t >> 1))) * weight;
        acc[q][0] = fmaf(xs, sum[q][0], acc[q][0]);
        acc[q][1] = fmaf(xs, sum[q][1], acc[q][1]);
    }
}

// ---------------------------------------------------------------- the kernel
// Shared-memory plan: [ring: stages x stage][zeros 1 KiB][image: planes | sums | scale][red: groups x slots x 8 warps x 16 rows x
//                     members of the column groups][norm: 2 x 9 x 8 f32][barriers]
__host__ __device__ inline size_t imma_fixed_bytes(int members, int nsb, int slots) {
    const size_t columns = static_cast<size_t>((members + 1) / 2 * 2);
    return 128 /*alignment*/ + kZeroBytes + image_bytes(members, nsb) + kGroups * static_cast<size_t>(slots) * kGroupWarps * kTileRows * columns * 4 +
           kGroups * kGroupWarps * kMaxMembers * 4 + (2 * kMaxStages + kGroups * kMaxSlots + 1) * 8;
}

// Where a CTA's stream of stages goes: chunk c (eight super-blocks) of its tiles, pairs of tiles interleaved chunk by chunk,
// group g taking tile 2 i + g; an odd last tile is group 0's alone.  Each group has a ring of its own: a wait on one parity bit
// is only safe for a warp that sees every phase of the barrier.  With one ring group 0 takes every tile.
struct Walk {
    int first, stage, phase;
    __device__ __forceinline__ int slot() const { return first + stage; }
    __device__ __forceinline__ void step(int stages) {
        if (++stage == stages) {
            stage = 0;
            phase ^= 1;
        }
    }
};

template <uint32_t FMT, int FETCH, int GROUPS>
__device__ __forceinline__ void gemv_imma_body(const CUtensorMap& wmap, const ImmaParams& p, int cta) {
    using P = ImmaPlan<FMT, FETCH>;
    constexpr int kColumns = 2 * GROUPS;   // members of the column groups
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((128u - (smem_addr(smem_raw) & 127u)) & 127u);
    uint8_t* ring = smem;
    uint8_t* zeros = ring + static_cast<size_t>(p.stages * p.rings) * P::kStageBytes;
    uint8_t* image = zeros + kZeroBytes;
    uint8_t* planes = image;
    __half* sums = reinterpret_cast<__half*>(planes + image_plane_bytes(p.members, p.nsb));
    float* scale = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(sums) + image_sums_bytes(p.members, p.nsb));
    float* red = scale + static_cast<size_t>(p.nsb) * 8;
    float* norm = red + kGroups * p.slots * (kGroupWarps * kTileRows * kColumns);
    uint64_t* full = reinterpret_cast<uint64_t*>(norm + kGroups * kGroupWarps * kMaxMembers);
    uint64_t* empty = full + kMaxStages;
    uint64_t* summed = empty + kMaxStages;      // [group][slot]
    uint64_t* image_bar = summed + kGroups * kMaxSlots;

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int stages = p.stages;
    pdl_launch_dependents();
    // The producer warp initialises the barriers and goes straight on to request weights; the consumers only
    // need to know that the barriers exist before their first wait (named barrier 2: they sync, the producer arrives).
    if (warp == kConsumerWarps) {
        if (lane == 0 && FETCH == kBoxes) tma_prefetch_descriptor(&wmap);
        for (int b = lane; b < 2 * kMaxStages + kGroups * kMaxSlots + 1; b += 32) {
            const bool is_empty = b >= kMaxStages && b < 2 * kMaxStages, is_summed = b >= 2 * kMaxStages && b < 2 * kMaxStages + kGroups * kMaxSlots;
            mbar_init(&full[b], is_empty || is_summed ? kGroupWarps : 1);
        }
        mbar_fence_init();
        __syncwarp();
        asm volatile("bar.arrive 2, %0;" ::"n"(kThreads) : "memory");
    }

    const int tile_begin = cta * p.tile_quotient + min(cta, p.tile_remainder);
    const int tiles = p.tile_quotient + (cta < p.tile_remainder ? 1 : 0);
    const int chunks = (p.nsb + kGroupWarps - 1) / kGroupWarps;
    bool ok = true;

    if (warp == kConsumerWarps) {
        // ---------------- producer warp: the weight stream does not depend on the activations ----------------
        // the first round of every stage waits for nothing: parity 1 of a fresh barrier has passed
        Walk walk{0, 0, 1}, other{stages, 0, 1};
        auto request = [&](int tile, int chunk) {
            if (lane == 0 || FETCH != kBoxes) ok = ok && mbar_spin(&empty[walk.slot()], walk.phase);
            if (FETCH != kBoxes) ok = __all_sync(0xffffffffu, ok);
            if (ok) {
                const int row0 = (tile_begin + tile) * kTileRows;
                const int sbs = min(kGroupWarps, p.nsb - chunk * kGroupWarps);
                const int boxes = (sbs + P::kBoxSb - 1) / P::kBoxSb;
                uint8_t* stage = ring + static_cast<size_t>(walk.slot()) * P::kStageBytes;
                uint64_t* bar = &full[walk.slot()];
                if constexpr (FETCH == kBoxes) {
                    if (lane == 0) {
                        mbar_arrive_expect_tx(bar, static_cast<uint32_t>(boxes * P::kBoxBytes));
                        const int x = chunk * (P::kBoxesPerStage * P::kBoxSpan / 8);
                        for (int b = 0; b < boxes; ++b) tma_load_2d(stage + b * P::kBoxBytes, &wmap, x + b * (P::kBoxSpan / 8), row0, bar);
                    }
                } else {
                    // lane = (box, row): the row's share of the box from the 16-byte boundary below, up to the one above, and no
                    // further than the tensor reaches
                    static_assert(P::kBoxesPerStage * kTileRows <= 32, "one copy per lane");
                    const int row = lane & (kTileRows - 1), b = lane >> 4;
                    const unsigned long long row_start = static_cast<unsigned long long>(row0 + row) * p.row_bytes;
                    const unsigned long long from = row_start + static_cast<unsigned long long>(chunk * P::kBoxesPerStage + b) * P::kBoxSpan;
                    const unsigned long long to = min(from + P::kBoxSpan, row_start + p.row_bytes);
                    const unsigned long long first = from & ~15ull;
                    const bool mine = b < boxes && row0 + row < p.n;
                    uint32_t bytes = mine ? static_cast<uint32_t>(((to + 15ull) & ~15ull) - first) : 0u;
                    uint8_t* target = stage + b * P::kBoxBytes + row * P::kRowPitch;
                    if (row0 + kTileRows >= p.n) {
                        // The last tile: its last row may end inside the tensor's last 16 bytes.  (Clamping in every tile cost this
                        // thread 130 clocks per stage: Q6_K 4096 x 11520, one row, 16.8 -> 17.6 us.)
                        RowCopy copy{0ull, 0u, 0u};
                        if (mine) copy = row_copy(from, to, p.weight_bytes);
                        bytes = copy.bytes;
                        const uint16_t* from_tail = reinterpret_cast<const uint16_t*>(p.weights + first + bytes);   // rows are whole pairs of bytes
                        uint16_t pairs[7];
#pragma unroll
                        for (uint32_t i = 0; i < 7; ++i) pairs[i] = 2 * i < copy.tail ? from_tail[i] : uint16_t{0};
#pragma unroll
                        for (uint32_t i = 0; i < 7; ++i)
                            if (2 * i < copy.tail) reinterpret_cast<uint16_t*>(target + bytes)[i] = pairs[i];
                        __syncwarp();   // the tail is in place before the stage is said to be
                    }
                    const uint32_t total = __reduce_add_sync(0xffffffffu, bytes);
                    if (lane == 0) mbar_arrive_expect_tx(bar, total);
                    __syncwarp();
                    if (bytes > 0) bulk_copy_g2s(target, p.weights + first, bytes, bar);
                }
            }
            walk.step(stages);
        };
#pragma unroll 1
        for (int tile = 0; tile < tiles; tile += p.rings) {
            const int both = p.rings == 2 && tile + 1 < tiles ? 2 : 1;
#pragma unroll 1
            for (int step = 0; step < both * chunks; ++step) {
                if (both == 1) {
                    request(tile, step);
                } else {
                    request(tile + (step & 1), step >> 1);
                    const Walk next = other;
                    other = walk;
                    walk = next;
                }
            }
        }
        ok = __all_sync(0xffffffffu, ok);
    } else {
        // ---------------- consumers ----------------
        const int group = warp / kGroupWarps, w8 = warp % kGroupWarps;
        const int g = lane >> 2, t = lane & 3;
        if (threadIdx.x < kZeroBytes / 4) reinterpret_cast<uint32_t*>(zeros)[threadIdx.x] = 0u;
        named_barrier_sync(2, kThreads);
        pdl_wait_prior();   // the activations may be the previous kernel's output, and y may still be read by it
        if (p.image != nullptr) {
            // a consumer asks for the image: the producer may be far behind the previous kernel's end, filling the ring
            if (threadIdx.x == 0) {
                const uint32_t bytes = static_cast<uint32_t>(image_bytes(p.members, p.nsb));
                mbar_arrive_expect_tx(image_bar, bytes);
                for (uint32_t done = 0; done < bytes; done += 32768u) bulk_copy_g2s(image + done, p.image + done, min(bytes - done, 32768u), image_bar);
            }
        } else {
            // The warp's slices (every sixteenth of [member][super-block]); the next one is on its way while one is converted.  One
            // copy of the code: it runs once or twice, and most of its time is fetching the instructions.
            float* my_norm = norm + group * kGroupWarps * kMaxMembers;   // both groups make the same sums
            float v[8], by[8];
            int m = 0, sb = warp, held_m = 0, held_sb = -1;
#pragma unroll 1
            for (;;) {
                while (sb >= p.nsb && m < p.members) {
                    sb -= p.nsb;
                    ++m;
                }
                float next[8], next_by[8];
                if (m < p.members) load_slice(p, m, sb, lane, next, next_by);
                if (held_sb >= 0) {
                    float inv_rms = 1.0f;
                    if (p.mode == 1) {
                        float totalsq = 0.0f;
#pragma unroll
                        for (int w = 0; w < kGroupWarps; ++w) totalsq += my_norm[w * kMaxMembers + held_m];
                        inv_rms = 1.0f / sqrtf(totalsq / static_cast<float>(p.k) + p.eps);
                    }
                    apply_prologue(p, inv_rms, v, by);
                    store_slice(p.rotated != 0, held_m, held_sb, lane, v, planes + static_cast<size_t>(held_m) * p.nsb * kSliceBytes,
                                sums + static_cast<size_t>(held_m) * p.nsb * 16, scale);
                } else if (p.mode == 1) {
                    for (int row = 0; row < p.members; ++row) {
                        float part = partial_square_sum(p, row, w8 * 32 + lane, kGroupWarps * 32);
#pragma unroll
                        for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
                        if (lane == 0) my_norm[w8 * kMaxMembers + row] = part;
                    }
                    named_barrier_sync(3 + group, kGroupWarps * 32);
                }
                if (m >= p.members) break;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    v[j] = next[j];
                    by[j] = next_by[j];
                }
                held_m = m;
                held_sb = sb;
                sb += kConsumerWarps;
            }
        }
        named_barrier_sync(1, kConsumers);   // the zero area, and the slices the other warps converted
        if (p.image != nullptr) ok = mbar_spin(image_bar, 0);

        LaneX<GROUPS> lx;
        {
#pragma unroll
            for (int q = 0; q < GROUPS; ++q) {
                const int member = 2 * q + (g >> 2), plane = g & 3;
                const bool real = member < p.members && plane < 3;
                // the lane's share of a block: 8 bytes of a 32-weight sub-block (Q4_K / Q5_K), 4 bytes of 16 weights (Q6_K, Q8_0)
                const uint32_t lane_bytes = (FMT == kQ6_K || FMT == kQ8_0 ? 4u : 8u) * t;
                lx.x[q] = real ? smem_addr(planes) + static_cast<uint32_t>(member) * static_cast<uint32_t>(p.nsb) * kSliceBytes + plane * 32u + lane_bytes
                               : smem_addr(zeros) + 96u + lane_bytes;
                lx.step[q] = real ? static_cast<uint32_t>(kSliceBytes) : 0u;
            }
            const uint32_t sums_member = g < p.members ? static_cast<uint32_t>(g) : 0u;
            lx.sums = smem_addr(sums) + sums_member * static_cast<uint32_t>(p.nsb) * 32u;
            lx.scale = smem_addr(scale);
        }
        // This warp's super-block inside a stage: box w8 / kBoxSb, position w8 % kBoxSb, rows g and g + 8.
        const uint32_t ring_addr = smem_addr(ring) + static_cast<uint32_t>((w8 / P::kBoxSb) * P::kBoxBytes + (w8 % P::kBoxSb) * P::kSbBytes + g * P::kRowPitch);
        lx.advance(w8);   // the warp's super-block of the first chunk
        Walk walk{group * stages, 0, 0};
        int slot = 0, slot_phase = 0, turn = 0;   // of the group's next tile: where its sums meet, and which warp finishes it

#pragma unroll 1
        for (int tile = group < p.rings ? group : tiles; tile < tiles; tile += p.rings) {
            const int row0 = (tile_begin + tile) * kTileRows;
            float acc[GROUPS][2], mins[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int q = 0; q < GROUPS; ++q) acc[q][0] = acc[q][1] = 0.0f;
            uint32_t delta0 = 0u, delta1 = 0u;   // how far behind the copied boundary the rows start
            if (FETCH != kBoxes) {
                delta0 = static_cast<uint32_t>(static_cast<unsigned long long>(row0 + g) * p.row_bytes) & 15u;
                delta1 = (delta0 + 8u * static_cast<uint32_t>(p.row_bytes)) & 15u;
            }
#pragma unroll 1
            for (int chunk = 0; chunk < chunks; ++chunk) {
                ok = ok && mbar_spin(&full[walk.slot()], walk.phase);
                const int sb = chunk * kGroupWarps + w8;
                if (sb < p.nsb) {
                    const uint32_t base = ring_addr + static_cast<uint32_t>(walk.slot()) * P::kStageBytes;
                    const uint32_t p0 = base + delta0, p1 = base + 8 * P::kRowPitch + delta1;
                    if constexpr (FMT == kQ6_K) {
                        // 210-byte super-blocks: in rows that start on a word the warp's one does when its position in the box is even
                        if constexpr (FETCH == kRowsOdd) superblock_q6<GROUPS, kMixed>(p0, p1, lx, t, acc);
                        else if (w8 & 1) superblock_q6<GROUPS, kOdd>(p0, p1, lx, t, acc);
                        else superblock_q6<GROUPS, kEven>(p0, p1, lx, t, acc);
                    } else if constexpr (FMT == kQ8_0) {
                        superblock_q8<GROUPS, FETCH != kBoxes>(p0, p1, lx, t, p.k / 32 - sb * 8, acc);
                    } else {
                        superblock<FMT, GROUPS>(p0, p1, lx, t, acc, mins);
                    }
                }
                lx.advance(kGroupWarps);
                __syncwarp();
                if (lane == 0) mbar_arrive(&empty[walk.slot()]);
                walk.step(stages);
            }
            lx.advance(-chunks * kGroupWarps);
            // Tile end: a member's two plane shares sit in neighbouring lanes and its minima in lane q of the four; the eight warps'
            // partial sums meet in a slot of shared memory, and one warp -- each in turn -- adds them and stores the rows.  The
            // others go on: a slot is written again only by a warp that has seen a stage which the finisher gave back later.
            float* part = red + (group * p.slots + slot) * (kGroupWarps * kTileRows * kColumns);
            float* buf = part + w8 * (kTileRows * kColumns);
#pragma unroll
            for (int q = 0; q < GROUPS; ++q) {
                float v0 = acc[q][0] + __shfl_xor_sync(0xffffffffu, acc[q][0], 1);
                float v1 = acc[q][1] + __shfl_xor_sync(0xffffffffu, acc[q][1], 1);
                if (FMT == kQ4_K || FMT == kQ5_K) {
                    const int holder = (lane & ~3) | q;
                    const float m0 = __shfl_sync(0xffffffffu, mins[0], holder), m1 = __shfl_sync(0xffffffffu, mins[1], holder);
                    const float m2 = __shfl_sync(0xffffffffu, mins[2], holder), m3 = __shfl_sync(0xffffffffu, mins[3], holder);
                    v0 += t < 2 ? m0 : m1;
                    v1 += t < 2 ? m2 : m3;
                }
                if ((t & 1) == 0) {
                    buf[g * kColumns + 2 * q + (t >> 1)] = v0;
                    buf[(g + 8) * kColumns + 2 * q + (t >> 1)] = v1;
                }
            }
            __syncwarp();
            uint64_t* bar = &summed[group * kMaxSlots + slot];
            if (lane == 0) mbar_arrive(bar);
            if (w8 == turn) {
                constexpr int kOutputs = kTileRows * kColumns / 32;   // per lane
                float old[kOutputs];
#pragma unroll
                for (int i = 0; i < kOutputs; ++i) {
                    const int item = i * 32 + lane, m = item % kColumns, row = row0 + item / kColumns;
                    old[i] = 0.0f;
                    if (p.accumulate && m < p.members && row < p.n) {
                        const size_t o = static_cast<size_t>(m) * p.n + static_cast<size_t>(row);
                        old[i] = p.y_bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(p.y)[o]) : static_cast<const float*>(p.y)[o];
                    }
                }
                ok = ok && mbar_spin(bar, slot_phase);
#pragma unroll
                for (int i = 0; i < kOutputs; ++i) {
                    const int item = i * 32 + lane, m = item % kColumns, row = row0 + item / kColumns;
                    float v = part[item];
#pragma unroll
                    for (int w = 1; w < kGroupWarps; ++w) v += part[w * (kTileRows * kColumns) + item];
                    if (m < p.members && row < p.n) {
                        const size_t o = static_cast<size_t>(m) * p.n + static_cast<size_t>(row);
                        if (p.accumulate) v += old[i];
                        if (p.y_bf16) static_cast<__nv_bfloat16*>(p.y)[o] = __float2bfloat16_rn(v);
                        else static_cast<float*>(p.y)[o] = v;
                    }
                }
            }
            turn = (turn + 1) % kGroupWarps;
            if (++slot == p.slots) {
                slot = 0;
                slot_phase ^= 1;
            }
        }
    }
    // A wait that ran out: copies may still be in flight into this CTA's shared memory; give them time to land before the
    // memory is handed to another CTA.  (Otherwise every copy has been waited for by the consumers.)
    if (!ok) {
        atomicExch(p.status, kDeviceWaitTimeout);
        for (int spin = 0; spin < 64; ++spin) __nanosleep(1000);
    }
}

template <uint32_t FMT, int FETCH, int GROUPS>
__global__ void __launch_bounds__(kThreads, 1) gemv_imma_kernel(const __grid_constant__ CUtensorMap wmap, const ImmaParams p) {
    gemv_imma_body<FMT, FETCH, GROUPS>(wmap, p, static_cast<int>(blockIdx.x));
}

// Two projections of one input (a decode step's [q | k] and v) in one launch: the first `first_ctas` CTAs work on the first.
// A small projection costs its start-up -- the end of the kernel before it, the conversion of the activations, the first
// weights -- whatever its size: Q6_K 1024 x 4096 behind Q4_K 5120 x 4096 took 5.1 us, together they take no longer than
// the first alone.
template <uint32_t FMT1, uint32_t FMT2, int GROUPS>
__global__ void __launch_bounds__(kThreads, 1) gemv_imma_pair_kernel(const __grid_constant__ CUtensorMap wmap1, const __grid_constant__ CUtensorMap wmap2,
                                                                     const ImmaParams p1, const ImmaParams p2, int first_ctas) {
    const int cta = static_cast<int>(blockIdx.x);
    if (cta < first_ctas) gemv_imma_body<FMT1, kBoxes, GROUPS>(wmap1, p1, cta);
    else gemv_imma_body<FMT2, kBoxes, GROUPS>(wmap2, p2, cta - first_ctas);
}

// ---------------------------------------------------------------- pre-pass: the activation image in global memory
// grid (ceil(nsb / 8), members): warp w of CTA (c, m) converts super-block 8c + w of member row m.
__global__ void __launch_bounds__(256) gemv_imma_image_kernel(const ImmaParams p, uint8_t* image) {
    __shared__ float partial[8];
    pdl_launch_dependents();
    pdl_wait_prior();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m = blockIdx.y;
    float inv_rms = 1.0f;
    if (p.mode == 1) {
        float part = partial_square_sum(p, m, static_cast<int>(threadIdx.x), 256);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
        if (lane == 0) partial[warp] = part;
        __syncthreads();
        float totalsq = 0.0f;
#pragma unroll
        for (int w = 0; w < 8; ++w) totalsq += partial[w];
        inv_rms = 1.0f / sqrtf(totalsq / static_cast<float>(p.k) + p.eps);
    }
    __half* sums = reinterpret_cast<__half*>(image + image_plane_bytes(p.members, p.nsb));
    float* scale = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(sums) + image_sums_bytes(p.members, p.nsb));
    const int sb = blockIdx.x * 8 + warp;
    if (sb < p.nsb) {
        float v[8], by[8];
        load_slice(p, m, sb, lane, v, by);
        apply_prologue(p, inv_rms, v, by);
        store_slice(p.rotated != 0, m, sb, lane, v, image + static_cast<size_t>(m) * p.nsb * kSliceBytes, sums + static_cast<size_t>(m) * p.nsb * 16, scale);
    }
}

constexpr size_t kSmemLimit = 227 * 1024;

int block_bytes(uint32_t value_type) { return value_type == kQ8_0 ? 34 : value_type == kQ4_K ? 144 : value_type == kQ5_K ? 176 : 210; }
int superblocks(int k) { return (k + kSuperBlock - 1) / kSuperBlock; }
unsigned long long encoded_row_bytes(uint32_t value_type, int k) {
    return value_type == kQ8_0 ? static_cast<unsigned long long>(k / 32) * 34 : static_cast<unsigned long long>(k / kSuperBlock) * block_bytes(value_type);
}
Fetch fetch_of(uint32_t value_type, int k) {
    const unsigned long long row = encoded_row_bytes(value_type, k);
    if (row % 16 == 0) return kBoxes;
    return row % 4 == 0 && value_type == kQ6_K ? kRowsEven : kRowsOdd;
}

// Rings, stages per ring and slots of a launch; stages = 0 when two stages do not fit.
struct Ring {
    int rings, stages, slots;
};
Ring ring_of(size_t stage_bytes, int members, int nsb, int tiles_per_cta, int wanted) {
    const int chunks = (nsb + kGroupWarps - 1) / kGroupWarps;
    // A group with a single stage waits for every copy it asks for.  Where the images leave no more than that, one group has all the
    // stages (4096 rows: Q4_K 4 x 12288 17.5 -> 13.5 us, 6 x 8192 14.7 -> 11.4; Q6_K 5 x 8192 18.1 -> 14.8).
    const int rings = tiles_per_cta > 1 && imma_fixed_bytes(members, nsb, (2 + chunks) / chunks) + 4 * stage_bytes <= kSmemLimit ? 2 : 1, least = 2;
    const int most = std::min(kMaxStages / rings, std::max(least, chunks * ((tiles_per_cta + rings - 1) / rings)));   // no more than the CTA has use for
    for (int stages = most; stages >= least; --stages) {
        if (wanted > 0 && stages * rings > wanted && stages > least) continue;
        // A warp that writes the slot of its group's tile T + slots has seen that tile's last stage, for which every warp of the group
        // gave the stage's last use back; that use is of tile T + 1 or later, begun when the sums of tile T were complete.
        const int slots = (stages + chunks) / chunks;
        if (imma_fixed_bytes(members, nsb, slots) + static_cast<size_t>(stages * rings) * stage_bytes <= kSmemLimit) return Ring{rings, stages, slots};
    }
    return Ring{0, 0, 0};
}
size_t stage_bytes_of(uint32_t value_type, Fetch fetch) {
    switch (value_type) {
        case kQ4_K: return ImmaPlan<kQ4_K, kBoxes>::kStageBytes;
        case kQ5_K: return ImmaPlan<kQ5_K, kBoxes>::kStageBytes;
        case kQ6_K: return fetch == kBoxes ? ImmaPlan<kQ6_K, kBoxes>::kStageBytes : ImmaPlan<kQ6_K, kRowsEven>::kStageBytes;
        default: return ImmaPlan<kQ8_0, kBoxes>::kStageBytes;
    }
}

ImmaParams params_of(const MmaGemvArgs& a) {
    ImmaParams p{};
    p.x = a.x;
    p.x_bf16 = a.x_bf16 ? 1 : 0;
    p.mode = a.mode;
    p.norm_weight = a.norm_weight;
    p.eps = a.eps;
    p.rotated = gemv_imma_rotates(a.value_type, a.k) ? 1 : 0;
    p.k = a.k;
    p.nsb = superblocks(a.k);
    p.members = a.members;
    return p;
}

// Parameters, tensor map and shared memory of a call on `ctas` CTAs.
template <uint32_t FMT, int FETCH>
cudaError_t plan(const MmaGemvArgs& a, int ctas, ImmaParams& p, CUtensorMap& wmap, size_t& smem) {
    using P = ImmaPlan<FMT, FETCH>;
    p = params_of(a);
    const int tiles = (a.n + kTileRows - 1) / kTileRows;
    p.tile_quotient = tiles / ctas;
    p.tile_remainder = tiles % ctas;
    const Ring ring = ring_of(P::kStageBytes, a.members, p.nsb, p.tile_quotient + (p.tile_remainder > 0 ? 1 : 0), a.stages);
    if (ring.stages == 0) return cudaErrorInvalidConfiguration;
    p.stages = ring.stages;
    p.rings = ring.rings;
    p.slots = ring.slots;
    smem = imma_fixed_bytes(a.members, p.nsb, p.slots) + static_cast<size_t>(p.stages * p.rings) * P::kStageBytes;
    p.row_bytes = encoded_row_bytes(FMT, a.k);
    p.weight_bytes = p.row_bytes * static_cast<unsigned long long>(a.n);
    if constexpr (FETCH == kBoxes) {
        EncodeTiledFn encode = encode_tiled_fn();
        if (encode == nullptr) return cudaErrorNotSupported;
        const cuuint64_t dims[2] = {static_cast<cuuint64_t>(p.row_bytes / 8), static_cast<cuuint64_t>(a.n)};
        const cuuint64_t strides[1] = {static_cast<cuuint64_t>(p.row_bytes)};
        const cuuint32_t box[2] = {static_cast<cuuint32_t>(P::kRowPitch / 8), static_cast<cuuint32_t>(kTileRows)};
        const cuuint32_t elem[2] = {1, 1};
        if (encode(&wmap, CU_TENSOR_MAP_DATA_TYPE_UINT64, 2, const_cast<uint8_t*>(a.weights), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return cudaErrorInvalidValue;
    }
    p.image = static_cast<const uint8_t*>(a.image);
    p.weights = a.weights;
    p.y = a.y;
    p.y_bf16 = a.y_bf16 ? 1 : 0;
    p.accumulate = a.accumulate ? 1 : 0;
    p.n = a.n;
    p.status = a.device_status;
    return cudaSuccess;
}

template <typename Kernel>
cudaError_t allow_shared_memory(Kernel kernel, int& configured_device) {
    int device = 0;
    cudaGetDevice(&device);
    if (configured_device == device) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSmemLimit));
    if (e == cudaSuccess) configured_device = device;
    return e;
}

template <uint32_t FMT, int FETCH, int GROUPS>
cudaError_t launch_groups(const MmaGemvArgs& a) {
    auto kernel = gemv_imma_kernel<FMT, FETCH, GROUPS>;
    static int configured_device = -1;
    cudaError_t e = allow_shared_memory(kernel, configured_device);
    if (e != cudaSuccess) return e;
    // One CTA per SM: its sixteen consumer warps share one image of the activations, and whole SMs divide the tiles more
    // evenly than halves do.
    const int tiles = (a.n + kTileRows - 1) / kTileRows;
    const int grid = tiles < a.sm_count ? tiles : a.sm_count;
    ImmaParams p;
    CUtensorMap wmap{};
    size_t smem = 0;
    e = plan<FMT, FETCH>(a, grid, p, wmap, smem);
    if (e != cudaSuccess) return e;
    return launch_kernel(kernel, dim3(grid), dim3(kThreads), smem, a.stream, wmap, p);
}

template <uint32_t FMT1, uint32_t FMT2, int GROUPS>
cudaError_t launch_pair_groups(const MmaGemvArgs& a, const MmaGemvArgs& b) {
    auto kernel = gemv_imma_pair_kernel<FMT1, FMT2, GROUPS>;
    static int configured_device = -1;
    cudaError_t e = allow_shared_memory(kernel, configured_device);
    if (e != cudaSuccess) return e;
    // SMs in proportion to the encoded bytes, so that both parts end together
    const int tiles1 = (a.n + kTileRows - 1) / kTileRows, tiles2 = (b.n + kTileRows - 1) / kTileRows;
    const double bytes1 = static_cast<double>(tiles1) * block_bytes(FMT1), bytes2 = static_cast<double>(tiles2) * block_bytes(FMT2);
    int ctas1 = static_cast<int>(a.sm_count * bytes1 / (bytes1 + bytes2) + 0.5);
    ctas1 = std::max(1, std::min(a.sm_count - 1, ctas1));
    const int ctas2 = std::min(tiles2, a.sm_count - ctas1);
    ctas1 = std::min(tiles1, ctas1);
    ImmaParams p1, p2;
    CUtensorMap wmap1{}, wmap2{};
    size_t smem1 = 0, smem2 = 0;
    e = plan<FMT1, kBoxes>(a, ctas1, p1, wmap1, smem1);
    if (e == cudaSuccess) e = plan<FMT2, kBoxes>(b, ctas2, p2, wmap2, smem2);
    if (e != cudaSuccess) return e;
    return launch_kernel(kernel, dim3(ctas1 + ctas2), dim3(kThreads), std::max(smem1, smem2), a.stream, wmap1, wmap2, p1, p2, ctas1);
}

template <uint32_t FMT1, uint32_t FMT2>
cudaError_t launch_pair(const MmaGemvArgs& a, const MmaGemvArgs& b) {
    switch ((a.members + 1) / 2) {
        case 1: return launch_pair_groups<FMT1, FMT2, 1>(a, b);
        case 2: return launch_pair_groups<FMT1, FMT2, 2>(a, b);
        case 3: return launch_pair_groups<FMT1, FMT2, 3>(a, b);
        default: return launch_pair_groups<FMT1, FMT2, 4>(a, b);
    }
}

template <uint32_t FMT, int FETCH>
cudaError_t launch_format(const MmaGemvArgs& a) {
    switch ((a.members + 1) / 2) {
        case 1: return launch_groups<FMT, FETCH, 1>(a);
        case 2: return launch_groups<FMT, FETCH, 2>(a);
        case 3: return launch_groups<FMT, FETCH, 3>(a);
        default: return launch_groups<FMT, FETCH, 4>(a);
    }
}

}  // namespace

bool gemv_imma_rotates(uint32_t value_type, int k) { return value_type == kQ8_0 && fetch_of(value_type, k) == kBoxes; }

bool gemv_imma_supports(uint32_t value_type, int k, int n, int members, const void* weights) {
    if (value_type != kQ4_K && value_type != kQ5_K && value_type != kQ6_K && value_type != kQ8_0) return false;
    if (members < 1 || members > kMaxMembers || k <= 0 || k % (value_type == kQ8_0 ? 32 : kSuperBlock) != 0 || n < kTileRows) return false;
    if (reinterpret_cast<uintptr_t>(weights) % 16 != 0) return false;
    return ring_of(stage_bytes_of(value_type, fetch_of(value_type, k)), members, superblocks(k), 2, 0).stages != 0;
}

bool gemv_imma_pairs(const MmaGemvArgs& a, const MmaGemvArgs& b) {
    return (a.value_type == kQ4_K || a.value_type == kQ5_K) && b.value_type == kQ6_K && fetch_of(kQ6_K, b.k) == kBoxes && a.k == b.k && a.x == b.x &&
           a.members == b.members && a.members <= kMaxMembers;
}

cudaError_t launch_gemv_imma_pair(const MmaGemvArgs& a, const MmaGemvArgs& b) {
    return a.value_type == kQ4_K ? launch_pair<kQ4_K, kQ6_K>(a, b) : launch_pair<kQ5_K, kQ6_K>(a, b);
}

size_t gemv_imma_image_bytes(int members, int k) { return (image_bytes(members, superblocks(k)) + 255) & ~static_cast<size_t>(255); }

cudaError_t launch_gemv_imma_image(const MmaGemvArgs& a, void* image) {
    const ImmaParams p = params_of(a);
    return launch_kernel(gemv_imma_image_kernel, dim3((p.nsb + 7) / 8, a.members), dim3(256), 0, a.stream, p, static_cast<uint8_t*>(image));
}

cudaError_t launch_gemv_imma(const MmaGemvArgs& a) {
    const Fetch fetch = fetch_of(a.value_type, a.k);
    switch (a.value_type) {
        case kQ4_K: return launch_format<kQ4_K, kBoxes>(a);
        case kQ5_K: return launch_format<kQ5_K, kBoxes>(a);
        case kQ6_K:
            return fetch == kBoxes      ? launch_format<kQ6_K, kBoxes>(a)
                   : fetch == kRowsEven ? launch_format<kQ6_K, kRowsEven>(a)
                                        : launch_format<kQ6_K, kRowsOdd>(a);
        case kQ8_0: return fetch == kBoxes ? launch_format<kQ8_0, kBoxes>(a) : launch_format<kQ8_0, kRowsOdd>(a);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace ribn
