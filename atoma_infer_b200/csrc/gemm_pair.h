// Products on CTA pairs (gemm_pair.cu): what its callers fill in.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace atoma {

constexpr int kPairClamped = 3;   // activation of GemmPairArgs::act beyond hybrid::glu_act's 0 silu, 1 relu, 2 gelu

struct GemmPairArgs {
    void *y;                      // [rows, N], row stride ldy
    int64_t ldy;
    // gated activation: act 0..2: act(gate) up;  kPairClamped: glu_clamped on gate + bias[n], up + bias[N + n] (bias may be null)
    int act, round_products;      // round_products: the two products are rounded to the output's type first
    const float *bias;
    float limit, alpha, shift;
    // dense: `chunks` runs of `width` tokens (a multiple of 32, at most 256)
    int width, chunks;
    // grouped (plan not null): plan[0] chunks; from plan[4] on four ints per chunk: expert, first row, rows, width (a multiple of 32, at most 256)
    const int32_t *plan;
    const int32_t *row_pair;      // with out_weight: row r is scaled by out_weight[row_pair[r]] (negative: zero)
    const float *out_weight;
    int tiles, max_width;         // grouped: upper bounds of the tiles and of a chunk's width (a multiple of 32)
    int w_once;                   // the weights are read once: they need not stay in L2
    // filled in by launch_gemm_pair
    unsigned int *late;           // set to 1 when a wait ran out (late_word())
    int T, N, K, is_bf16, w_tiles, stages, stage_bytes, kbs, k_blocked;
};

// Tokens per chunk for T tokens.
int gemm_pair_width(int64_t T, int64_t N, int64_t K, bool glu);
int gemm_pair_w_tiles(int64_t N, bool glu);
bool gemm_pair_ok(const void *x, const void *w, int64_t N, int64_t K, int64_t ldx, int64_t ldw);
bool launch_gemm_pair(GemmPairArgs a, const void *x, const void *w, int64_t rows, int64_t N, int64_t K, int64_t ldx, int64_t ldw, int64_t experts, bool glu,
                      bool is_bf16, cudaStream_t stream);

}  // namespace atoma
