// Host-side helpers shared by the tensor-core kernels: kernel parameter block, tensor-map encoding
// through the runtime's driver entry point, split-K choice.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace ribn {

struct TcParams {
    const uint8_t* w;
    unsigned long long w_bytes;
    unsigned long long row_bytes;
    void* y;                 // [m][n] f32 or bf16
    float* partial;          // split-K scratch: [ksplit][m][n] f32
    const float* x_scale;    // decode kernel: power-of-two factor per member row (activations were divided by it)
    unsigned int* tickets;   // one counter per (n tile, m tile), zero between launches
    int k, n, m;
    int nsb;                 // super-blocks per row
    int ksplit;
    int y_bf16;
    int accumulate;          // decode kernel: add to y instead of overwriting it
    int* status;
    // Diagnostics: when non-null, CTA (0,0,0) of the decode kernel records SM clock stamps of its
    // pipeline events here: trace[(role * 64 + step) * 8 + event], 4 roles x 64 steps x 8 events.
    long long* trace;
};

// cuTensorMapEncodeTiled through the runtime's driver entry point (the library does not link libcuda).
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                   const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_tiled_fn() {
    static EncodeTiledFn fn = nullptr;
    if (fn == nullptr) {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult result;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &result) == cudaSuccess &&
            result == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(sym);
    }
    return fn;
}

// The GEMM's split factor: waves of tiles of 128 rows x (K work per CTA + a fixed cost of about one and a half super-blocks for
// pipeline fill, TMEM allocation and the epilogue), minimised.  The kernel works on pairs of CTAs and cuts tokens finer than the
// tiles counted here.  Against the best of eleven forced factors: within 1 % at six of nine shapes of 96..256 tokens (Q5_K 5120 x
// 5120, 173 tokens: 24.1 us in three, 36.4 unsplit); behind it at Q4_K 24576 x 4096, 200 tokens (66.9 us, 57.6 unsplit), 12288 x 4096,
// 128 tokens (33.2, 30.6 unsplit) and Q6_K 1024 x 4096, 256 tokens (21.5 in sixteen, 18.0 in four to eight).
inline int choose_ksplit(int tiles, int nsb, int sm_count, size_t plane_bytes, size_t scratch_bytes, int max_tickets) {
    if (tiles > max_tickets) return 1;
    int best = 1;
    double best_cost = 1e30;
    const int limit = nsb < 16 ? nsb : 16;
    for (int ks = 1; ks <= limit; ++ks) {
        if (ks > 1 && plane_bytes * ks > scratch_bytes) break;
        const int waves = (tiles * ks + sm_count - 1) / sm_count;
        const double per_cta = static_cast<double>((nsb + ks - 1) / ks) + 1.5 + (ks > 1 ? 0.5 : 0.0);
        const double cost = waves * per_cta;
        if (cost < best_cost - 1e-9) {
            best_cost = cost;
            best = ks;
        }
    }
    return best;
}

// The f16-tile decode kernel's split factor (qgemv_tc.cu; times in units of one 128-row super-block, ~1.45 us): a CTA costs its K
// share plus ~5 units of launch, pipeline fill and epilogue; every split adds a partial tile the last CTA of the tile has to add,
// ~0.33 units per 16 tokens.  Ties go to the smaller factor.  Q8_0, against the best forced factor: within 1 % from nine to 32 rows
// (12288 x 4096, sixteen rows: 32.9 us unsplit, 39.6 in two; 4096 x 12288 31.4 in four, 37.2 in three); at 64 rows one split too many
// (4096 x 4096 29.4 in four, 21.6 in three; 4096 x 12288 47.6 and 43.6).
inline int choose_ksplit_decode(int tiles, int nsb, int sm_count, size_t plane_bytes, size_t scratch_bytes, int max_tickets,
                                int tokens_per_tile) {
    if (tiles > max_tickets) return 1;
    int best = 1;
    double best_cost = 1e30;
    const int limit = nsb < 16 ? nsb : 16;
    for (int ks = 1; ks <= limit; ++ks) {
        if (ks > 1 && plane_bytes * ks > scratch_bytes) break;
        const int waves = (tiles * ks + sm_count - 1) / sm_count;
        const double per_cta = static_cast<double>((nsb + ks - 1) / ks) + 5.0;
        const double reduce = ks > 1 ? ks * 0.33 * (tokens_per_tile / 16.0) : 0.0;
        const double cost = waves * per_cta + reduce;
        if (cost < best_cost - 1e-9) {
            best_cost = cost;
            best = ks;
        }
    }
    return best;
}

}  // namespace ribn
