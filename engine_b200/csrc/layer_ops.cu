// The operators of a dense-attention decoder layer that sit between the quantized GEMVs.
//
// They replace, for decode, these kernels of the reference (crates/nvidia/src/model_ops.rs and
// kernels/quantized/q4_k.cu):
//   q4_k_embedding{,_batch}   q4_k.cu:1-67          -> embedding_kernel (any of the four block formats)
//   strided_rms_norm          model_ops.rs:660-684  \
//   rope_neox                 model_ops.rs:393-422   > qk_norm_rope_append_kernel (one launch per token batch)
//   kv_append_f16             model_ops.rs:1256-1275 /
//   attn_score_gqa            model_ops.rs:439-562  -> attention_split_kernel + attention_combine_kernel
//   silu_mul                  model_ops.rs:316-328  -> silu_mul_kernel
//   residual_add              model_ops.rs:600-610  -> residual_add_kernel
//   argmax{,_batch}           model_ops.rs:201-314  -> argmax_kernel
// The arithmetic follows the reference's host model of the layer
// (crates/nvidia/src/qwen_reference.rs:368-470): per-head RMSNorm with raw weights, NEOX half-split
// rotary pairs (p, p + rot/2) with theta = pos * base^(-2p/rot), scores scaled by 1/sqrt(head_dim),
// softmax over all cached tokens, f32 accumulation; K and V are cached as f16.
//
// Layout of the KV cache (ours; the reference's is [token][kv_head][dim]):
//   [member][kv_head][token][dim] f16, max_context tokens per (member, head),
// so that one CTA streams the contiguous tokens of one head, shared by the query heads of its group.
//
// Positions are read from device memory (one int per member), so that a captured CUDA graph can be
// replayed for every decode step.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "formats.cuh"
#include "internal.h"
#include "pipeline.cuh"

namespace ribn {
namespace {

// ---------------------------------------------------------------- embedding
template <uint32_t FMT>
__global__ void __launch_bounds__(256) embedding_kernel(const uint8_t* __restrict__ w, const uint32_t* __restrict__ tokens,
                                                        float* __restrict__ out, int k, unsigned int vocabulary,
                                                        unsigned long long row_bytes, int nsb) {
    pdl_launch_dependents();
    pdl_wait_prior();   // inputs come from the kernels before this one in the stream
    using F = Format<FMT>;
    const int lane = threadIdx.x & 31;
    const int sb = blockIdx.x * 8 + (threadIdx.x >> 5);
    const unsigned int token = tokens[blockIdx.y];
    if (sb >= nsb || token >= vocabulary) return;   // as the reference: an out-of-range token leaves its row untouched
    int off_a, off_b;
    F::offsets(lane, off_a, off_b);
    const uint8_t* blk = w + static_cast<unsigned long long>(token) * row_bytes + static_cast<unsigned long long>(sb) * F::kBytes;
    float qa[4], qb[4], sa, ma, sb_scale, mb;
    F::quants(blk, lane, qa, qb);
    F::direct_scales(blk, lane, sa, ma, sb_scale, mb);
    float* dst = out + static_cast<size_t>(blockIdx.y) * k + static_cast<size_t>(sb) * kSuperBlock;
    *reinterpret_cast<float4*>(dst + off_a) = make_float4(dequant_value(sa, qa[0], ma), dequant_value(sa, qa[1], ma),
                                                          dequant_value(sa, qa[2], ma), dequant_value(sa, qa[3], ma));
    *reinterpret_cast<float4*>(dst + off_b) = make_float4(dequant_value(sb_scale, qb[0], mb), dequant_value(sb_scale, qb[1], mb),
                                                          dequant_value(sb_scale, qb[2], mb), dequant_value(sb_scale, qb[3], mb));
}

// ---------------------------------------------------------------- head norm + rope + cache append
// grid (ceil((q_heads + 2 kv_heads) / 8), members), a warp per head of 128 values, four per lane.  Heads [0, q_heads) rewrite a
// query head in place; [q_heads, q_heads + kv_heads) normalise and rotate a key head into the f16 cache; the rest convert a
// value head into the cache.  The angles depend on the member and the pair only: the CTA works them out once for its eight
// heads (a power, a sine and a cosine per pair).  A CTA per head, every thread with its own three of them, took 28 us for 512
// members of 48 heads.
constexpr int kHeadDim = 128;
constexpr int kRopeWarps = 8;

__global__ void __launch_bounds__(kRopeWarps * 32) qk_norm_rope_append_kernel(float* __restrict__ q, const float* __restrict__ k,
                                                                              const float* __restrict__ v, const float* __restrict__ q_norm,
                                                                              const float* __restrict__ k_norm, float eps,
                                                                              const int* __restrict__ positions, int q_heads, int kv_heads,
                                                                              int rot_pairs, float base, __half* __restrict__ k_cache,
                                                                              __half* __restrict__ v_cache, long long max_context, int shared_cache,
                                                                              int* __restrict__ status) {
    pdl_launch_dependents();
    pdl_wait_prior();   // inputs come from the kernels before this one in the stream
    __shared__ float sines[kHeadDim / 2], cosines[kHeadDim / 2];
    __shared__ float values[kRopeWarps][kHeadDim];
    const int member = blockIdx.y;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int head = blockIdx.x * kRopeWarps + warp;
    const int position = positions[member];
    const float* source = nullptr;
    const float* norm = nullptr;
    bool rotate = true;
    __half* cache = nullptr;
    float* in_place = nullptr;
    if (head < q_heads) {
        in_place = q + (static_cast<size_t>(member) * q_heads + head) * kHeadDim;
        source = in_place;
        norm = q_norm;
    } else if (head < q_heads + kv_heads) {
        head -= q_heads;
        source = k + (static_cast<size_t>(member) * kv_heads + head) * kHeadDim;
        norm = k_norm;
        cache = k_cache;
    } else if (head < q_heads + 2 * kv_heads) {
        head -= q_heads + kv_heads;
        source = v + (static_cast<size_t>(member) * kv_heads + head) * kHeadDim;
        rotate = false;
        cache = v_cache;
    }
    float x[4] = {0.0f, 0.0f, 0.0f, 0.0f};   // dims lane + 32 j
    if (source != nullptr) {
#pragma unroll
        for (int j = 0; j < 4; ++j) x[j] = source[lane + 32 * j];
    }
    if (threadIdx.x < rot_pairs) {
        const int pair = threadIdx.x;
        const float theta = static_cast<float>(position) * powf(base, -(2.0f * static_cast<float>(pair)) / (2.0f * static_cast<float>(rot_pairs)));
        sines[pair] = sinf(theta);
        cosines[pair] = cosf(theta);
    }
    __syncthreads();
    if (source == nullptr) return;
    if (norm != nullptr) {
        float total = 0.0f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float sum = x[j] * x[j];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            total += sum;
        }
        const float inverse = rsqrtf(total / static_cast<float>(kHeadDim) + eps);
#pragma unroll
        for (int j = 0; j < 4; ++j) x[j] = x[j] * inverse * norm[lane + 32 * j];
    }
    if (rotate && rot_pairs > 0) {
        float* own = values[warp];
#pragma unroll
        for (int j = 0; j < 4; ++j) own[lane + 32 * j] = x[j];
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int d = lane + 32 * j;
            if (d < 2 * rot_pairs) {
                const int pair = d < rot_pairs ? d : d - rot_pairs;
                const float sin_theta = sines[pair];
                const float cos_theta = cosines[pair];
                const float x0 = own[pair];
                const float x1 = own[pair + rot_pairs];
                x[j] = d < rot_pairs ? x0 * cos_theta - x1 * sin_theta : x0 * sin_theta + x1 * cos_theta;
            }
        }
    }
    if (in_place != nullptr) {
#pragma unroll
        for (int j = 0; j < 4; ++j) in_place[lane + 32 * j] = x[j];
    } else if (position >= 0 && position < max_context) {
        // a prefill chunk: the members are consecutive tokens of one sequence and append to the same cache
        const long long sequence = shared_cache ? 0 : member;
        __half* slot = cache + ((sequence * kv_heads + head) * max_context + position) * kHeadDim;
#pragma unroll
        for (int j = 0; j < 4; ++j) slot[lane + 32 * j] = __float2half_rn(x[j]);
    } else if (lane == 0) {
        // The position comes from device memory (a replayed graph advances it): outside the cache nothing is
        // stored and the context's status word says so.
        atomicExch(status, kDevicePositionOutOfRange);
    }
}

// ---------------------------------------------------------------- attention, one new token per member
// Split-KV ("flash decoding") on the warp-level tensor-core instruction: grid (kv_heads, members, splits), four warps.
// The query heads that share a KV head (up to eight) are the rows of one m16n8k16 A operand, so a K / V tile is read from
// shared memory once for the whole group (a kernel that lets every head read the tile with its own loads is bound by
// shared-memory bandwidth at 1/8 of what HBM delivers).  The CTA walks its token range in tiles of 64: cp.async brings K
// and V rows into padded shared-memory rows (272 bytes: ldmatrix of eight rows touches every bank once), warp w owns
// tokens 16 w .. 16 w + 15 of every tile and keeps its own running maximum, sum and 16 x 128 output accumulator; the four
// warps are merged through shared memory at the end.  The reference computes in f32 over the f16 cache
// (model_ops.rs:439-562); to stay at that accuracy the f32 queries and the probabilities enter the MMAs as two f16 parts
// each (hi + lo: about 22 bits), with f32 accumulation.
constexpr int kAttnTile = 64;
constexpr int kAttnHeadDim = 128;
constexpr int kAttnKStride = kAttnHeadDim + 8;   // halves; rows 272 bytes apart
constexpr int kAttnMaxGroup = 8;
constexpr int kAttnWarps = 4;
constexpr int kAttnTileBytes = kAttnTile * kAttnKStride * 2;
constexpr int kAttnSmemBytes = 4 * kAttnTileBytes;   // two stages of K and V; reused for the merge of the warps

__device__ __forceinline__ void ldmatrix_x4(uint32_t address, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(address));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t address, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(address));
}
__device__ __forceinline__ void mma_f16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_half2(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}
// (lo, hi) as f16 pair, and the f16 pair of what that rounding lost
__device__ __forceinline__ void split_half2(float lo, float hi, uint32_t& main, uint32_t& rest) {
    const __half2 h = __floats2half2_rn(lo, hi);
    const float2 back = __half22float2(h);
    main = *reinterpret_cast<const uint32_t*>(&h);
    rest = pack_half2(lo - back.x, hi - back.y);
}

__global__ void __launch_bounds__(kAttnWarps * 32, 3) attention_split_kernel(const float* __restrict__ q, const __half* __restrict__ k_cache,
                                                                             const __half* __restrict__ v_cache,
                                                                             const int* __restrict__ positions, float* __restrict__ part_o,
                                                                             float* __restrict__ part_ml, int q_heads, int kv_heads,
                                                                             long long max_context, int chunk, float scale, int active_context,
                                                                             int shared_cache, int* __restrict__ status) {
    pdl_launch_dependents();
    pdl_wait_prior();   // inputs come from the kernels before this one in the stream
    extern __shared__ __align__(128) uint8_t attn_smem[];
    const int kv_head = blockIdx.x;
    const int member = blockIdx.y;
    const int split = blockIdx.z;
    const int splits = gridDim.z;
    const int group = q_heads / kv_heads;
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;   // fragment coordinates: row g (and g + 8), column pair t
    // positions[] is device memory: the walk is clamped to the context the splits were planned for (at most the
    // cache size), and a position outside it is reported through the status word
    int tokens = positions[member] + 1;
    if (tokens < 1 || tokens > active_context) {
        if (threadIdx.x == 0 && split == 0 && kv_head == 0) atomicExch(status, kDevicePositionOutOfRange);
        tokens = max(0, min(tokens, active_context));
    }
    const int begin = split * chunk;
    const int end = min(tokens, begin + chunk);

    const long long sequence = shared_cache ? 0 : member;
    const __half* k_base = k_cache + (sequence * kv_heads + kv_head) * max_context * kAttnHeadDim;
    const __half* v_base = v_cache + (sequence * kv_heads + kv_head) * max_context * kAttnHeadDim;
    const uint32_t smem_base = static_cast<uint32_t>(__cvta_generic_to_shared(attn_smem));

    // Tile loads: 64 tokens x 128 halves of K and of V, 16 bytes per request; rows past the range are zero-filled.
    auto request_tile = [&](int buffer, int t0) {
        const int valid = min(kAttnTile, end - t0);
        for (int i = threadIdx.x; i < kAttnTile * (kAttnHeadDim / 8); i += blockDim.x) {
            const int row = i / (kAttnHeadDim / 8);
            const int piece = i % (kAttnHeadDim / 8);
            const uint32_t kd = smem_base + (2 * buffer) * kAttnTileBytes + (row * kAttnKStride + 8 * piece) * 2;
            const uint32_t vd = kd + kAttnTileBytes;
            if (row < valid) {
                const __half* ks = k_base + static_cast<long long>(t0 + row) * kAttnHeadDim + 8 * piece;
                const __half* vs = v_base + static_cast<long long>(t0 + row) * kAttnHeadDim + 8 * piece;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(kd), "l"(ks) : "memory");
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(vd), "l"(vs) : "memory");
            } else {
                asm volatile("st.shared.v4.b32 [%0], {%1,%1,%1,%1};" ::"r"(kd), "r"(0) : "memory");
                asm volatile("st.shared.v4.b32 [%0], {%1,%1,%1,%1};" ::"r"(vd), "r"(0) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (begin < end) request_tile(0, begin);   // in flight while the queries are fetched and split below

    // The group's queries as A fragments, times scale * log2(e) (the softmax runs on exp2), hi and lo parts: rows = heads
    // (rows from `group` on are zero), eight K steps of 16 dims.
    uint32_t q_hi[8][4], q_lo[8][4];
    {
        const float factor = scale * 1.4426950408889634f;
        const float* q_group = q + (static_cast<size_t>(member) * q_heads + static_cast<size_t>(kv_head) * group) * kAttnHeadDim;
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
#pragma unroll
            for (int part = 0; part < 4; ++part) {
                const int row = g + 8 * (part & 1), column = 16 * ks + 2 * t + 8 * (part >> 1);
                float2 v = make_float2(0.0f, 0.0f);
                if (row < group) v = *reinterpret_cast<const float2*>(q_group + row * kAttnHeadDim + column);
                split_half2(v.x * factor, v.y * factor, q_hi[ks][part], q_lo[ks][part]);
            }
        }
    }

    float out[16][4];   // rows g, g + 8; dims 8 n + 2 t, + 1
#pragma unroll
    for (int n = 0; n < 16; ++n) out[n][0] = out[n][1] = out[n][2] = out[n][3] = 0.0f;
    float running_max[2] = {-INFINITY, -INFINITY}, running_sum[2] = {0.0f, 0.0f};
    // ldmatrix row addresses of this lane inside a tile: K as B operand (not transposed), V as B operand (transposed)
    const uint32_t k_lane = ((16 * warp + (lane & 7) + 8 * (lane >> 4)) * kAttnKStride + 8 * ((lane >> 3) & 1)) * 2;
    const uint32_t v_lane = ((16 * warp + (lane & 7) + 8 * ((lane >> 3) & 1)) * kAttnKStride + 8 * (lane >> 4)) * 2;

    int buffer = 0;
    for (int t0 = begin; t0 < end; t0 += kAttnTile, buffer ^= 1) {
        if (t0 + kAttnTile < end) {
            request_tile(buffer ^ 1, t0 + kAttnTile);   // its previous contents were consumed before the barrier that ended the last round
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();   // this tile has landed for every thread
        const int first = t0 + 16 * warp;    // this warp's sixteen tokens
        if (first < end) {
            const uint32_t k_tile = smem_base + (2 * buffer) * kAttnTileBytes, v_tile = k_tile + kAttnTileBytes;
            // scores: S[16 heads][16 tokens] = Q K^T, two n-tiles of eight tokens
            float s[2][4] = {{0.0f, 0.0f, 0.0f, 0.0f}, {0.0f, 0.0f, 0.0f, 0.0f}};
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) {
                uint32_t b[4];   // (tokens 0-7: dims lo, hi), (tokens 8-15: dims lo, hi) of this K step
                ldmatrix_x4(k_tile + k_lane + 32 * ks, b);
                mma_f16(s[0], q_hi[ks], b[0], b[1]);
                mma_f16(s[1], q_hi[ks], b[2], b[3]);
                mma_f16(s[0], q_lo[ks], b[0], b[1]);
                mma_f16(s[1], q_lo[ks], b[2], b[3]);
            }
            // mask the tokens past the range, then the online softmax of rows g and g + 8
            const int valid = end - first;
#pragma unroll
            for (int n = 0; n < 2; ++n) {
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (8 * n + 2 * t + (c & 1) >= valid) s[n][c] = -INFINITY;
            }
            uint32_t p_hi[4], p_lo[4];
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                float tile_max = fmaxf(fmaxf(s[0][2 * r], s[0][2 * r + 1]), fmaxf(s[1][2 * r], s[1][2 * r + 1]));
                tile_max = fmaxf(tile_max, __shfl_xor_sync(0xffffffffu, tile_max, 1));
                tile_max = fmaxf(tile_max, __shfl_xor_sync(0xffffffffu, tile_max, 2));
                const float new_max = fmaxf(running_max[r], tile_max);   // finite: the warp has at least one valid token
                const float rescale = exp2f(running_max[r] - new_max);   // 0 the first time round
                running_max[r] = new_max;
                const float p0 = exp2f(s[0][2 * r] - new_max), p1 = exp2f(s[0][2 * r + 1] - new_max);
                const float p2 = exp2f(s[1][2 * r] - new_max), p3 = exp2f(s[1][2 * r + 1] - new_max);
                running_sum[r] = running_sum[r] * rescale + ((p0 + p1) + (p2 + p3));   // this lane's share; lanes are added at the end
#pragma unroll
                for (int n = 0; n < 16; ++n) {
                    out[n][2 * r] *= rescale;
                    out[n][2 * r + 1] *= rescale;
                }
                // A fragment of P: a[r] = tokens 2t, 2t+1 of row g + 8 r; a[2 + r] = tokens 8 + 2t, + 1
                split_half2(p0, p1, p_hi[r], p_lo[r]);
                split_half2(p2, p3, p_hi[2 + r], p_lo[2 + r]);
            }
            // O += P V: one K step of sixteen tokens, sixteen n-tiles of eight dims
#pragma unroll
            for (int pair = 0; pair < 8; ++pair) {
                uint32_t b[4];   // dims 16 pair .. + 7: (tokens 0-7, 8-15), dims 16 pair + 8 .. + 15: (tokens 0-7, 8-15)
                ldmatrix_x4_trans(v_tile + v_lane + 32 * pair, b);
                mma_f16(out[2 * pair], p_hi, b[0], b[1]);
                mma_f16(out[2 * pair + 1], p_hi, b[2], b[3]);
                mma_f16(out[2 * pair], p_lo, b[0], b[1]);
                mma_f16(out[2 * pair + 1], p_lo, b[2], b[3]);
            }
        }
        __syncthreads();   // every warp is done with this buffer before the next round refills it
    }

    // merge the four warps: [warp][row] maximum and sum, [warp][row][dim] output, in the tile buffers
    float* merge_o = reinterpret_cast<float*>(attn_smem);                        // [4][8][128]
    float* merge_m = merge_o + kAttnWarps * kAttnMaxGroup * kAttnHeadDim;         // [4][8]
    float* merge_l = merge_m + kAttnWarps * kAttnMaxGroup;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        running_sum[r] += __shfl_xor_sync(0xffffffffu, running_sum[r], 1);
        running_sum[r] += __shfl_xor_sync(0xffffffffu, running_sum[r], 2);
    }
    if (g < kAttnMaxGroup) {   // rows g + 8 are padding: at most eight heads share a KV head
        if (t == 0) {
            merge_m[warp * kAttnMaxGroup + g] = running_max[0];
            merge_l[warp * kAttnMaxGroup + g] = running_sum[0];
        }
#pragma unroll
        for (int n = 0; n < 16; ++n)
            *reinterpret_cast<float2*>(merge_o + (warp * kAttnMaxGroup + g) * kAttnHeadDim + 8 * n + 2 * t) = make_float2(out[n][0], out[n][1]);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < group * kAttnHeadDim; i += blockDim.x) {
        const int row = i / kAttnHeadDim, dim = i % kAttnHeadDim;
        float top = -INFINITY;
#pragma unroll
        for (int w = 0; w < kAttnWarps; ++w) top = fmaxf(top, merge_m[w * kAttnMaxGroup + row]);
        float total = 0.0f, value = 0.0f;
#pragma unroll
        for (int w = 0; w < kAttnWarps; ++w) {
            const float m = merge_m[w * kAttnMaxGroup + row];
            const float weight = m == -INFINITY ? 0.0f : exp2f(m - top);
            total = fmaf(merge_l[w * kAttnMaxGroup + row], weight, total);
            value = fmaf(merge_o[(w * kAttnMaxGroup + row) * kAttnHeadDim + dim], weight, value);
        }
        const size_t slot = (static_cast<size_t>(member) * q_heads + static_cast<size_t>(kv_head) * group + row) * splits + split;
        part_o[slot * kAttnHeadDim + dim] = value;
        if (dim == 0) {
            part_ml[slot * 2] = top * 0.6931471805599453f;   // back to natural-log units for the merge of the splits
            part_ml[slot * 2 + 1] = total;
        }
    }
}

// ---------------------------------------------------------------- attention of a prompt chunk
// The members are consecutive tokens of one sequence, so their queries share the keys and values they read.  The kernel above
// walks the cache once per token with at most eight of the sixteen rows of its MMAs in use (310 us on average for 512 tokens
// behind 0, 512, 1024 and 1536 others at 32 query and 8 key-value heads).  Here a CTA owns 48 rows = (token, head of the group)
// pairs of one KV head and one walk serves them all: bound by the MMAs, which are twice as many as a plain f16 product needs
// because queries and probabilities keep their hi + lo parts.  Warp = (row tile of 16, sixteen tokens of every tile of 64): the
// same sums in the same order as above, so that a token's result does not depend on which kernel ran.  Three row tiles: twelve
// warps of 168 registers fill the register file.  Grid (kv_heads, row tiles); the last tokens, which walk furthest, start first.
constexpr int kChunkRowTiles = 3;
constexpr int kChunkRows = 16 * kChunkRowTiles;
constexpr int kChunkWarps = kAttnWarps * kChunkRowTiles;
constexpr int kChunkMergeBytes = kAttnWarps * kChunkRows * (kAttnHeadDim + 2) * 4;
constexpr int kChunkSmemBytes = kAttnSmemBytes > kChunkMergeBytes ? kAttnSmemBytes : kChunkMergeBytes;

template <bool OUT_BF16>
__global__ void __launch_bounds__(kChunkWarps * 32, 1) attention_chunk_kernel(const float* __restrict__ q, const __half* __restrict__ k_cache,
                                                                              const __half* __restrict__ v_cache, const int* __restrict__ positions,
                                                                              void* __restrict__ out, int members, int q_heads, int kv_heads,
                                                                              long long max_context, float scale, int active_context,
                                                                              int* __restrict__ status) {
    pdl_launch_dependents();
    pdl_wait_prior();   // inputs come from the kernels before this one in the stream
    extern __shared__ __align__(128) uint8_t attn_smem[];
    __shared__ int warp_limit[kChunkWarps];
    const int kv_head = blockIdx.x;
    const int group = q_heads / kv_heads;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = warp / kAttnWarps, part = warp % kAttnWarps;   // row tile; which sixteen tokens of every 64
    const int g = lane >> 2, t = lane & 3;
    const int cta_row = static_cast<int>(gridDim.y - 1 - blockIdx.y) * kChunkRows;   // of members * group rows of this KV head

    // Tokens each of this thread's two rows may look at; positions[] is device memory: clamped and reported like above.
    int limit[2];
    const float* q_row[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int row = cta_row + tile * 16 + g + 8 * r;
        const int member = row / group;
        limit[r] = 0;
        q_row[r] = nullptr;
        if (member < members) {
            limit[r] = positions[member] + 1;
            if (limit[r] < 1 || limit[r] > active_context) {
                if (t == 0) atomicExch(status, kDevicePositionOutOfRange);
                limit[r] = max(0, min(limit[r], active_context));
            }
            q_row[r] = q + (static_cast<size_t>(member) * q_heads + static_cast<size_t>(kv_head) * group + (row - member * group)) * kAttnHeadDim;
        }
    }
    const int tile_end = __reduce_max_sync(0xffffffffu, max(limit[0], limit[1]));
    if (lane == 0) warp_limit[warp] = tile_end;
    __syncthreads();
    int end = 0;
#pragma unroll
    for (int w = 0; w < kChunkWarps; ++w) end = max(end, warp_limit[w]);

    const __half* k_base = k_cache + static_cast<long long>(kv_head) * max_context * kAttnHeadDim;
    const __half* v_base = v_cache + static_cast<long long>(kv_head) * max_context * kAttnHeadDim;
    const uint32_t smem_base = static_cast<uint32_t>(__cvta_generic_to_shared(attn_smem));
    auto request_tile = [&](int buffer, int t0) {
        const int valid = min(kAttnTile, end - t0);
        for (int i = threadIdx.x; i < kAttnTile * (kAttnHeadDim / 8); i += kChunkWarps * 32) {
            const int row = i / (kAttnHeadDim / 8);
            const int piece = i % (kAttnHeadDim / 8);
            const uint32_t kd = smem_base + (2 * buffer) * kAttnTileBytes + (row * kAttnKStride + 8 * piece) * 2;
            const uint32_t vd = kd + kAttnTileBytes;
            if (row < valid) {
                const __half* ks = k_base + static_cast<long long>(t0 + row) * kAttnHeadDim + 8 * piece;
                const __half* vs = v_base + static_cast<long long>(t0 + row) * kAttnHeadDim + 8 * piece;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(kd), "l"(ks) : "memory");
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(vd), "l"(vs) : "memory");
            } else {
                asm volatile("st.shared.v4.b32 [%0], {%1,%1,%1,%1};" ::"r"(kd), "r"(0) : "memory");
                asm volatile("st.shared.v4.b32 [%0], {%1,%1,%1,%1};" ::"r"(vd), "r"(0) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (end > 0) request_tile(0, 0);   // in flight while the queries are fetched and split below

    uint32_t q_hi[8][4], q_lo[8][4];
    {
        const float factor = scale * 1.4426950408889634f;
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
#pragma unroll
            for (int piece = 0; piece < 4; ++piece) {
                float2 v = make_float2(0.0f, 0.0f);
                if (q_row[piece & 1] != nullptr) v = *reinterpret_cast<const float2*>(q_row[piece & 1] + 16 * ks + 2 * t + 8 * (piece >> 1));
                split_half2(v.x * factor, v.y * factor, q_hi[ks][piece], q_lo[ks][piece]);
            }
        }
    }
    float acc[16][4];   // rows g, g + 8; dims 8 n + 2 t, + 1
#pragma unroll
    for (int n = 0; n < 16; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.0f;
    float running_max[2] = {-INFINITY, -INFINITY}, running_sum[2] = {0.0f, 0.0f};
    const uint32_t k_lane = ((16 * part + (lane & 7) + 8 * (lane >> 4)) * kAttnKStride + 8 * ((lane >> 3) & 1)) * 2;
    const uint32_t v_lane = ((16 * part + (lane & 7) + 8 * ((lane >> 3) & 1)) * kAttnKStride + 8 * (lane >> 4)) * 2;

    int buffer = 0;
    for (int t0 = 0; t0 < end; t0 += kAttnTile, buffer ^= 1) {
        if (t0 + kAttnTile < end) {
            request_tile(buffer ^ 1, t0 + kAttnTile);   // its previous contents were consumed before the barrier that ended the last round
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();   // this tile has landed for every thread
        const int first = t0 + 16 * part;
        if (first < tile_end) {
            const uint32_t k_tile = smem_base + (2 * buffer) * kAttnTileBytes, v_tile = k_tile + kAttnTileBytes;
            float s[2][4] = {{0.0f, 0.0f, 0.0f, 0.0f}, {0.0f, 0.0f, 0.0f, 0.0f}};
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) {
                uint32_t b[4];
                ldmatrix_x4(k_tile + k_lane + 32 * ks, b);
                mma_f16(s[0], q_hi[ks], b[0], b[1]);
                mma_f16(s[1], q_hi[ks], b[2], b[3]);
                mma_f16(s[0], q_lo[ks], b[0], b[1]);
                mma_f16(s[1], q_lo[ks], b[2], b[3]);
            }
            uint32_t p_hi[4], p_lo[4];
#pragma unroll
            for (int r = 0; r < 2; ++r) {
#pragma unroll
                for (int n = 0; n < 2; ++n) {
#pragma unroll
                    for (int c = 2 * r; c < 2 * r + 2; ++c)
                        if (first + 8 * n + 2 * t + (c & 1) >= limit[r]) s[n][c] = -INFINITY;
                }
                float tile_max = fmaxf(fmaxf(s[0][2 * r], s[0][2 * r + 1]), fmaxf(s[1][2 * r], s[1][2 * r + 1]));
                tile_max = fmaxf(tile_max, __shfl_xor_sync(0xffffffffu, tile_max, 1));
                tile_max = fmaxf(tile_max, __shfl_xor_sync(0xffffffffu, tile_max, 2));
                const float new_max = fmaxf(running_max[r], tile_max);
                const float shift = new_max == -INFINITY ? 0.0f : new_max;   // a row that sees none of these tokens
                const bool moved = new_max != running_max[r];
                const float rescale = exp2f(running_max[r] - shift);          // 0 the first time round
                running_max[r] = new_max;
                const float p0 = exp2f(s[0][2 * r] - shift), p1 = exp2f(s[0][2 * r + 1] - shift);
                const float p2 = exp2f(s[1][2 * r] - shift), p3 = exp2f(s[1][2 * r + 1] - shift);
                running_sum[r] = running_sum[r] * rescale + ((p0 + p1) + (p2 + p3));   // this lane's share; lanes are added at the end
                if (__any_sync(0xffffffffu, moved)) {   // rare after the first tiles; the factor is one otherwise
#pragma unroll
                    for (int n = 0; n < 16; ++n) {
                        acc[n][2 * r] *= rescale;
                        acc[n][2 * r + 1] *= rescale;
                    }
                }
                split_half2(p0, p1, p_hi[r], p_lo[r]);
                split_half2(p2, p3, p_hi[2 + r], p_lo[2 + r]);
            }
#pragma unroll
            for (int pair = 0; pair < 8; ++pair) {
                uint32_t b[4];
                ldmatrix_x4_trans(v_tile + v_lane + 32 * pair, b);
                mma_f16(acc[2 * pair], p_hi, b[0], b[1]);
                mma_f16(acc[2 * pair + 1], p_hi, b[2], b[3]);
                mma_f16(acc[2 * pair], p_lo, b[0], b[1]);
                mma_f16(acc[2 * pair + 1], p_lo, b[2], b[3]);
            }
        }
        __syncthreads();   // every warp is done with this buffer before the next round refills it
    }

    // merge the four token parts: [part][row] maximum and sum, [part][row][dim] output, in the tile buffers
    float* merge_o = reinterpret_cast<float*>(attn_smem);                    // [4][48][128]
    float* merge_m = merge_o + kAttnWarps * kChunkRows * kAttnHeadDim;        // [4][48]
    float* merge_l = merge_m + kAttnWarps * kChunkRows;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        running_sum[r] += __shfl_xor_sync(0xffffffffu, running_sum[r], 1);
        running_sum[r] += __shfl_xor_sync(0xffffffffu, running_sum[r], 2);
        const int row = part * kChunkRows + tile * 16 + g + 8 * r;
        if (t == 0) {
            merge_m[row] = running_max[r];
            merge_l[row] = running_sum[r];
        }
#pragma unroll
        for (int n = 0; n < 16; ++n)
            *reinterpret_cast<float2*>(merge_o + row * kAttnHeadDim + 8 * n + 2 * t) = make_float2(acc[n][2 * r], acc[n][2 * r + 1]);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kChunkRows * kAttnHeadDim; i += kChunkWarps * 32) {
        const int row = i / kAttnHeadDim, dim = i % kAttnHeadDim;
        const int member = (cta_row + row) / group;
        if (member >= members) break;
        float top = -INFINITY;
#pragma unroll
        for (int w = 0; w < kAttnWarps; ++w) top = fmaxf(top, merge_m[w * kChunkRows + row]);
        float total = 0.0f, value = 0.0f;
#pragma unroll
        for (int w = 0; w < kAttnWarps; ++w) {
            const float m = merge_m[w * kChunkRows + row];
            const float weight = m == -INFINITY ? 0.0f : exp2f(m - top);
            total = fmaf(merge_l[w * kChunkRows + row], weight, total);
            value = fmaf(merge_o[(w * kChunkRows + row) * kAttnHeadDim + dim], weight, value);
        }
        const size_t index = (static_cast<size_t>(member) * q_heads + static_cast<size_t>(kv_head) * group + (cta_row + row - member * group)) * kAttnHeadDim + dim;
        if constexpr (OUT_BF16) static_cast<__nv_bfloat16*>(out)[index] = __float2bfloat16_rn(value / total);
        else static_cast<float*>(out)[index] = value / total;
    }
}

// grid (q_heads, members), 128 threads: merges the splits of one query head.  Lane s of every warp holds split s (at most 32
// splits): the maximum, the sum and the weights come out of two warp reductions, and a thread then has sixteen partial rows
// of its output dimension in flight at a time.
template <bool OUT_BF16>
__global__ void __launch_bounds__(kAttnHeadDim) attention_combine_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml,
                                                                         void* __restrict__ out, int q_heads, int splits) {
    pdl_launch_dependents();
    pdl_wait_prior();   // inputs come from the kernels before this one in the stream
    const int lane = threadIdx.x & 31;
    const size_t base = (static_cast<size_t>(blockIdx.y) * q_heads + blockIdx.x) * splits;
    float m = -INFINITY, l = 0.0f;
    if (lane < splits) {
        const float2 ml = *reinterpret_cast<const float2*>(part_ml + (base + lane) * 2);
        m = ml.x;
        l = ml.y;
    }
    float global_max = m;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) global_max = fmaxf(global_max, __shfl_xor_sync(0xffffffffu, global_max, o));
    const float weight = m == -INFINITY ? 0.0f : expf(m - global_max);
    float total = l * weight;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
    const float* column = part_o + base * kAttnHeadDim + threadIdx.x;
    float value = 0.0f;
    for (int s0 = 0; s0 < splits; s0 += 16) {
        float part[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) part[u] = s0 + u < splits ? column[static_cast<size_t>(s0 + u) * kAttnHeadDim] : 0.0f;
#pragma unroll
        for (int u = 0; u < 16; ++u) value = fmaf(part[u], __shfl_sync(0xffffffffu, weight, (s0 + u) & 31), value);
    }
    const size_t index = (static_cast<size_t>(blockIdx.y) * q_heads + blockIdx.x) * kAttnHeadDim + threadIdx.x;
    if constexpr (OUT_BF16) static_cast<__nv_bfloat16*>(out)[index] = __float2bfloat16_rn(value / total);
    else static_cast<float*>(out)[index] = value / total;
}

// ---------------------------------------------------------------- elementwise
// out[m][i] = silu(gate[m][i]) * up[m][i]; gate and up rows are `in_stride` floats apart (they may be the two
// halves of one [members][2 * length] GEMV output), out rows are `length` apart.  Grid (pieces of a row, members); four
// neighbouring values per thread where rows keep 16-byte boundaries (VECTOR), one otherwise.  Bound by memory: 512 rows of
// 12288 took 22.8 us with one value and one 64-bit division per thread and step.
template <bool OUT_BF16, bool VECTOR>
__global__ void __launch_bounds__(256) silu_mul_kernel(const float* __restrict__ gate, const float* __restrict__ up, void* __restrict__ out,
                                                       unsigned long long length, unsigned long long in_stride, unsigned int first_member) {
    pdl_launch_dependents();
    pdl_wait_prior();   // inputs come from the kernels before this one in the stream
    constexpr int kWidth = VECTOR ? 4 : 1;
    const unsigned long long member = static_cast<unsigned long long>(first_member) + blockIdx.y;
    const float* gate_row = gate + member * in_stride;
    const float* up_row = up + member * in_stride;
    for (unsigned long long i = (static_cast<unsigned long long>(blockIdx.x) * blockDim.x + threadIdx.x) * kWidth; i < length;
         i += static_cast<unsigned long long>(gridDim.x) * blockDim.x * kWidth) {
        float g[kWidth], u[kWidth], product[kWidth];
        if constexpr (VECTOR) {
            const float4 gv = *reinterpret_cast<const float4*>(gate_row + i), uv = *reinterpret_cast<const float4*>(up_row + i);
            g[0] = gv.x; g[1] = gv.y; g[2] = gv.z; g[3] = gv.w;
            u[0] = uv.x; u[1] = uv.y; u[2] = uv.z; u[3] = uv.w;
        } else {
            g[0] = gate_row[i];
            u[0] = up_row[i];
        }
#pragma unroll
        for (int j = 0; j < kWidth; ++j) product[j] = (g[j] / (1.0f + expf(-g[j]))) * u[j];
        if constexpr (OUT_BF16) {
            __nv_bfloat16* target = static_cast<__nv_bfloat16*>(out) + member * length + i;
            if constexpr (VECTOR) {
                const __nv_bfloat162 low = __floats2bfloat162_rn(product[0], product[1]), high = __floats2bfloat162_rn(product[2], product[3]);
                *reinterpret_cast<uint2*>(target) = make_uint2(*reinterpret_cast<const uint32_t*>(&low), *reinterpret_cast<const uint32_t*>(&high));
            } else {
                *target = __float2bfloat16_rn(product[0]);
            }
        } else {
            float* target = static_cast<float*>(out) + member * length + i;
            if constexpr (VECTOR) *reinterpret_cast<float4*>(target) = make_float4(product[0], product[1], product[2], product[3]);
            else *target = product[0];
        }
    }
}

// y += x, four values per thread and a scalar tail (both pointers are 16-byte aligned)
__global__ void __launch_bounds__(256) residual_add_kernel(float* __restrict__ y, const float* __restrict__ x, unsigned long long total) {
    pdl_launch_dependents();
    pdl_wait_prior();   // inputs come from the kernels before this one in the stream
    const unsigned long long quads = total / 4;
    const unsigned long long thread = static_cast<unsigned long long>(blockIdx.x) * blockDim.x + threadIdx.x;
    for (unsigned long long i = thread; i < quads; i += static_cast<unsigned long long>(gridDim.x) * blockDim.x) {
        const float4 a = reinterpret_cast<const float4*>(y)[i], b = reinterpret_cast<const float4*>(x)[i];
        reinterpret_cast<float4*>(y)[i] = make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
    }
    if (thread < total - 4 * quads) y[4 * quads + thread] += x[4 * quads + thread];
}

// ---------------------------------------------------------------- argmax
// NaN never wins, ties go to the lowest index, a row of NaNs gives 0 -- the reference's rules (model_ops.rs:201-258).
// A candidate is one 64-bit word: the monotone unsigned image of its value above the complement of its index, so that the
// largest word is the answer and 0 means "none".
//
// Grid (parts, members).  A row is a vocabulary, 128 K values and more, and one CTA reads it at what a single SM can have in
// flight: 69 us for one row of 151936 values.  Sixteen values per thread and one CTA per 4096 put the whole row in flight at
// once; the CTAs of a row meet in an atomic maximum and the last to arrive writes the index and leaves the words zero.
constexpr int kArgmaxThreads = 256;
constexpr int kArgmaxPerThread = 16;
constexpr int kArgmaxWordsPerMember = 4;   // of the context's zero-initialised counters: the maximum (two words), arrivals

__device__ __forceinline__ unsigned int logit_key(float value) {
    const unsigned int bits = __float_as_uint(value);
    return (bits >> 31) ? ~bits : (bits ^ 0x80000000u);
}

__global__ void __launch_bounds__(kArgmaxThreads) argmax_kernel(const float* __restrict__ logits, unsigned int* __restrict__ out,
                                                                unsigned long long length, unsigned int* counters) {
    pdl_launch_dependents();
    pdl_wait_prior();   // inputs come from the kernels before this one in the stream
    __shared__ unsigned long long warp_best[kArgmaxThreads / 32];
    const float* row = logits + static_cast<size_t>(blockIdx.y) * length;
    unsigned long long best = 0ull;
    const unsigned long long stride = static_cast<unsigned long long>(gridDim.x) * (kArgmaxThreads * kArgmaxPerThread);
    for (unsigned long long first = static_cast<unsigned long long>(blockIdx.x) * (kArgmaxThreads * kArgmaxPerThread) + threadIdx.x; first < length;
         first += stride) {
        float value[kArgmaxPerThread];
#pragma unroll
        for (int u = 0; u < kArgmaxPerThread; ++u) {
            const unsigned long long i = first + static_cast<unsigned long long>(u) * kArgmaxThreads;
            value[u] = i < length ? row[i] : __int_as_float(0x7fc00000);
        }
#pragma unroll
        for (int u = 0; u < kArgmaxPerThread; ++u) {
            const unsigned int index = static_cast<unsigned int>(first) + static_cast<unsigned int>(u * kArgmaxThreads);
            const unsigned long long candidate = (static_cast<unsigned long long>(logit_key(value[u])) << 32) | (~index);
            if (value[u] == value[u] && candidate > best) best = candidate;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
        best = other > best ? other : best;
    }
    if ((threadIdx.x & 31) == 0) warp_best[threadIdx.x >> 5] = best;
    __syncthreads();
    if (threadIdx.x != 0) return;
#pragma unroll
    for (int w = 1; w < kArgmaxThreads / 32; ++w) best = warp_best[w] > best ? warp_best[w] : best;
    if (gridDim.x > 1) {
        unsigned int* words = counters + static_cast<size_t>(blockIdx.y) * kArgmaxWordsPerMember;
        unsigned long long* maximum = reinterpret_cast<unsigned long long*>(words);
        if (best != 0ull) atomicMax(maximum, best);
        __threadfence();
        if (atomicAdd(words + 2, 1u) != gridDim.x - 1) return;
        __threadfence();
        best = atomicExch(maximum, 0ull);   // ready for the next launch
        words[2] = 0u;
    }
    out[blockIdx.y] = best == 0ull ? 0u : ~static_cast<unsigned int>(best);
}

}  // namespace

// Whether an operator over `rows` rows is launched as a dependent of the kernel before it.  A decode step's operators are not (unless
// option "pdl" is 1): resident early, they keep the SMs from the projection behind them, whose weights could already be on their
// way (a step of one row: 1910 us without, 2020 with; 32 rows 1374 and 1385).  A prompt chunk's kernels are long and fill the SMs,
// and the launch between them is what a dependent start hides (1987 tokens, four layers: 6645 us without, 6540 with).
static bool dependent_launch(uint64_t rows) { return pdl_switch() == 1 || (pdl_switch() == 2 && rows > 64); }

cudaError_t launch_embedding(const uint8_t* weights, uint32_t value_type, int k, unsigned int vocabulary, const uint32_t* tokens,
                             int members, float* out, cudaStream_t stream) {
    const int nsb = k / kSuperBlock;
    const dim3 grid((nsb + 7) / 8, members);
    const unsigned long long blocks_per_row = value_type == kQ8_0 ? k / 32 : nsb;
    switch (value_type) {
        case kQ4_K: return launch_kernel_if(pdl_switch() == 1, embedding_kernel<kQ4_K>, grid, dim3(256), 0, stream, weights, tokens, out, k, vocabulary, blocks_per_row * 144ull, nsb);
        case kQ5_K: return launch_kernel_if(pdl_switch() == 1, embedding_kernel<kQ5_K>, grid, dim3(256), 0, stream, weights, tokens, out, k, vocabulary, blocks_per_row * 176ull, nsb);
        case kQ6_K: return launch_kernel_if(pdl_switch() == 1, embedding_kernel<kQ6_K>, grid, dim3(256), 0, stream, weights, tokens, out, k, vocabulary, blocks_per_row * 210ull, nsb);
        case kQ8_0: return launch_kernel_if(pdl_switch() == 1, embedding_kernel<kQ8_0>, grid, dim3(256), 0, stream, weights, tokens, out, k, vocabulary, blocks_per_row * 34ull, nsb);
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t launch_qk_norm_rope_append(const LayerAttentionArgs& a) {
    if (a.head_dim != kHeadDim) return cudaErrorInvalidValue;
    const dim3 grid((a.q_heads + 2 * a.kv_heads + kRopeWarps - 1) / kRopeWarps, a.members);
    return launch_kernel_if(dependent_launch(a.members), qk_norm_rope_append_kernel, grid, dim3(kRopeWarps * 32), 0, a.stream, a.q, a.k, a.v, a.q_norm, a.k_norm,
                            a.eps, a.positions, a.q_heads, a.kv_heads, a.rot_dims / 2, a.rope_base, static_cast<__half*>(a.k_cache),
                            static_cast<__half*>(a.v_cache), a.max_context, a.shared_cache ? 1 : 0, a.device_status);
}

// Consecutive tokens of one sequence go to the chunk kernel once the token-by-token walk has enough CTAs to leave the context
// unsplit (four per SM) and the chunk's row tiles occupy at least half of the SMs.  Above the first line both give the same bits;
// below it the walk merges splits, which rounds differently.  The line is not where the times cross, which is earlier: 8 key/value
// heads of four query heads, behind 512 tokens, walk and chunk: 32 tokens 22.0 and 26.4 us, 64 tokens 36.1 and 26.7, 96 tokens 48.9 and
// 27.9 (the walk is taken), 112 tokens 58.4 and 28.1, 512 tokens 270 and 91.9 (the chunk is).  The second line is where a shard's
// two heads are: 128 tokens 27.0 and 28.1, 173 tokens 34.2 and 29.7, 512 tokens 85.5 and 55.5.
static bool attention_is_chunk(const LayerAttentionArgs& a, int sm_count) {
    const long long tiles = (static_cast<long long>(a.members) * (a.q_heads / a.kv_heads) + kChunkRows - 1) / kChunkRows;
    return a.shared_cache && static_cast<long long>(a.members) * a.kv_heads > 4ll * sm_count && 2 * tiles * a.kv_heads >= sm_count;
}

int attention_splits(const LayerAttentionArgs& a, int sm_count) {
    if (attention_is_chunk(a, sm_count)) return 0;   // no partial results
    // About eight CTAs per SM: a CTA walks its tiles one after the other, so the memory latency is hidden by
    // the CTAs that share its SM.
    int splits = (8 * sm_count) / (a.members * a.kv_heads);
    if (splits < 1) splits = 1;
    if (splits > 32) splits = 32;
    const long long tiles = (a.active_context + kAttnTile - 1) / kAttnTile;
    if (splits > tiles) splits = static_cast<int>(tiles < 1 ? 1 : tiles);
    return splits;
}

size_t attention_scratch_bytes(int members, int q_heads, int splits) {
    return static_cast<size_t>(members) * q_heads * splits * (kAttnHeadDim + 2) * sizeof(float);
}

static cudaError_t launch_attention_chunk(const LayerAttentionArgs& a, void* out, bool out_bf16) {
    const float scale = 1.0f / sqrtf(static_cast<float>(a.head_dim));
    auto kernel = out_bf16 ? attention_chunk_kernel<true> : attention_chunk_kernel<false>;
    static int configured_device = -1;
    int device = 0;
    cudaGetDevice(&device);
    if (configured_device != device) {
        cudaError_t attribute = cudaFuncSetAttribute(attention_chunk_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kChunkSmemBytes);
        if (attribute == cudaSuccess)
            attribute = cudaFuncSetAttribute(attention_chunk_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kChunkSmemBytes);
        if (attribute != cudaSuccess) return attribute;
        configured_device = device;
    }
    const int tiles = (a.members * (a.q_heads / a.kv_heads) + kChunkRows - 1) / kChunkRows;
    return launch_kernel_if(dependent_launch(a.members), kernel, dim3(a.kv_heads, tiles), dim3(kChunkWarps * 32), kChunkSmemBytes, a.stream,
                            static_cast<const float*>(a.q), static_cast<const __half*>(a.k_cache), static_cast<const __half*>(a.v_cache), a.positions, out,
                            a.members, a.q_heads, a.kv_heads, a.max_context, scale, static_cast<int>(a.active_context), a.device_status);
}

cudaError_t launch_attention_decode(const LayerAttentionArgs& a, void* out, bool out_bf16, void* scratch, int splits) {
    if (a.head_dim != kAttnHeadDim || a.q_heads % a.kv_heads != 0 || a.q_heads / a.kv_heads > kAttnMaxGroup) return cudaErrorInvalidValue;
    if (splits == 0) return launch_attention_chunk(a, out, out_bf16);
    long long chunk = (a.active_context + splits - 1) / splits;
    chunk = (chunk + kAttnTile - 1) / kAttnTile * kAttnTile;
    float* part_o = static_cast<float*>(scratch);
    float* part_ml = part_o + static_cast<size_t>(a.members) * a.q_heads * splits * kAttnHeadDim;
    const float scale = 1.0f / sqrtf(static_cast<float>(a.head_dim));
    static int configured_device = -1;
    int device = 0;
    cudaGetDevice(&device);
    if (configured_device != device) {
        const cudaError_t attribute = cudaFuncSetAttribute(attention_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kAttnSmemBytes);
        if (attribute != cudaSuccess) return attribute;
        configured_device = device;
    }
    cudaError_t e = launch_kernel_if(pdl_switch() == 1, attention_split_kernel, dim3(a.kv_heads, a.members, splits), dim3(kAttnWarps * 32), kAttnSmemBytes, a.stream,
                                  static_cast<const float*>(a.q), static_cast<const __half*>(a.k_cache), static_cast<const __half*>(a.v_cache),
                                  a.positions, part_o, part_ml, a.q_heads, a.kv_heads, a.max_context, static_cast<int>(chunk), scale,
                                  static_cast<int>(a.active_context), a.shared_cache ? 1 : 0, a.device_status);
    if (e != cudaSuccess) return e;
    if (out_bf16)
        return launch_kernel_if(pdl_switch() == 1, attention_combine_kernel<true>, dim3(a.q_heads, a.members), dim3(kAttnHeadDim), 0, a.stream,
                                static_cast<const float*>(part_o), static_cast<const float*>(part_ml), out, a.q_heads, splits);
    return launch_kernel_if(pdl_switch() == 1, attention_combine_kernel<false>, dim3(a.q_heads, a.members), dim3(kAttnHeadDim), 0, a.stream,
                            static_cast<const float*>(part_o), static_cast<const float*>(part_ml), out, a.q_heads, splits);
}

cudaError_t launch_silu_mul(const float* gate, const float* up, void* out, bool out_bf16, uint64_t members, uint64_t length, uint64_t in_stride,
                            int sm_count, cudaStream_t stream) {
    // rows that all start on 16-byte boundaries: the API checks the pointers, the halves of one row may still be anywhere
    const bool vector = length % 4 == 0 && in_stride % 4 == 0 && reinterpret_cast<uintptr_t>(gate) % 16 == 0 && reinterpret_cast<uintptr_t>(up) % 16 == 0;
    const uint64_t per_block = 256 * (vector ? 4 : 1);
    uint64_t pieces = (length + per_block - 1) / per_block;
    if (pieces > static_cast<uint64_t>(sm_count) * 8) pieces = static_cast<uint64_t>(sm_count) * 8;
    auto kernel = out_bf16 ? (vector ? silu_mul_kernel<true, true> : silu_mul_kernel<true, false>)
                           : (vector ? silu_mul_kernel<false, true> : silu_mul_kernel<false, false>);
    for (uint64_t first = 0; first < members; first += 65535) {   // members are the grid's y dimension
        const uint64_t rows = members - first < 65535 ? members - first : 65535;
        const cudaError_t e = launch_kernel_if(dependent_launch(members), kernel, dim3(static_cast<unsigned>(pieces), static_cast<unsigned>(rows)), dim3(256), 0,
                                               stream, gate, up, out, static_cast<unsigned long long>(length), static_cast<unsigned long long>(in_stride),
                                               static_cast<unsigned int>(first));
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_residual_add(float* y, const float* x, uint64_t rows, uint64_t total, int sm_count, cudaStream_t stream) {
    unsigned long long blocks = (total / 4 + 255) / 256;
    if (blocks > static_cast<unsigned long long>(sm_count) * 8) blocks = static_cast<unsigned long long>(sm_count) * 8;
    return launch_kernel_if(dependent_launch(rows), residual_add_kernel, dim3(static_cast<unsigned>(blocks ? blocks : 1)), dim3(256), 0, stream, y, x,
                         static_cast<unsigned long long>(total));
}

cudaError_t launch_argmax(const float* logits, int members, uint64_t length, uint32_t* out, unsigned int* counters, int counter_count, int sm_count,
                          cudaStream_t stream) {
    if (members <= 0) return cudaErrorInvalidValue;
    // As many CTAs as the rows have pieces of 4096 values, at most four per SM over all rows; one per row where the counters
    // do not reach.
    const uint64_t pieces = (length + kArgmaxThreads * kArgmaxPerThread - 1) / (kArgmaxThreads * kArgmaxPerThread);
    uint64_t parts = (4ull * sm_count + members - 1) / members;
    if (parts > pieces) parts = pieces;
    if (static_cast<int64_t>(members) * kArgmaxWordsPerMember > counter_count) parts = 1;
    // members is the grid's y dimension
    for (int first = 0; first < members; first += 65535) {
        const int rows = members - first < 65535 ? members - first : 65535;
        const cudaError_t e = launch_kernel_if(pdl_switch() == 1, argmax_kernel, dim3(static_cast<unsigned>(parts), rows), dim3(kArgmaxThreads), 0, stream,
                                               logits + static_cast<size_t>(first) * length, out + first, static_cast<unsigned long long>(length),
                                               counters);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace ribn
