// Device-side parameter block shared by the attention kernels.  Field meaning follows the
// reference's Flash_fwd_params (csrc/kernels/flash.h:18-134) for the live subset only; strides are
// in elements, widened to 64-bit here.
#pragma once
#include <cstdint>

namespace atoma {

struct MhaParams {
    const void *q;
    const void *k;
    const void *v;
    void *o;
    float *lse;           // may be null
    const float *alibi;   // may be null; [h] or [b,h] (alibi_bs = 0 / row stride)
    const int *cu_q;      // may be null (dense batch layout)
    const int *cu_k;      // may be null
    const int *seqused_k; // may be null
    const int *block_table;  // may be null (contiguous K/V)

    int64_t q_bs, k_bs, v_bs, o_bs;  // batch strides (k_bs/v_bs = page stride when paged)
    int64_t q_rs, k_rs, v_rs, o_rs;  // row (token) strides
    int64_t q_hs, k_hs, v_hs, o_hs;  // head strides
    int64_t alibi_bs;
    int64_t bt_bs;  // block_table row stride

    int b, h, h_k, d;
    int seqlen_q, seqlen_k;
    int page;  // page_block_size (tokens per KV block)
    float scale;
    float scale_log2;
    int is_causal;
    int k_cumulative;  // cu_k holds b+1 cumulative offsets (1) or b per-sequence lengths (0)
    int unpadded_lse;
    // tcgen05 prefill kernel only (zero = off): causal sliding window (query i sees the window_left keys up to its own), a
    // per-head softmax sink (one more term exp(sink[h]) of the denominator, not scaled), and sequences with fewer than
    // min_len_q query rows are left alone (nothing is read or written for them)
    int window_left;
    int min_len_q;
    const float *sink;
    // tcgen05 prefill kernel only (null = off): a bias by query-key distance, dist_bias[min(i + shift - j, dist_rows - 1) * dist_heads + head],
    // added to the scaled score
    const float *dist_bias;
    int dist_rows, dist_heads;
    // tcgen05 prefill kernel only: entries of a query / key head when they differ from the value head's d (0: the same), and a gate on the
    // outputs (null = none): out times sigmoid(gate[(first row of the sequence + i) * gate_rs + head * d + c]), rows as cu_q counts them
    int d_k;
    const void *gate;
    int64_t gate_rs;
    // ... for rows at positions below gate_below only (0: all rows); key_lo: position of every sequence's first key (null: 0)
    int gate_below;
    const int *key_lo;
    // tcgen05 prefill kernel only: neighbouring key heads that share one value head (0: 1); v then has h_k / v_share heads per row
    int v_share;
    // a paged step that both prompt kernels serve: attn_tile_kernel the sequences with short_for_prefill(), prefill_attn_kernel the others
    int split_short;
    int64_t rows_q;       // query rows of all sequences (0: unknown)
    int k_batched;        // tcgen05 prefill kernel on gathered keys only: sequence b's start at b k_bs also where cu_k holds offsets; so many rows there are
    unsigned int *late;   // set by the prefill kernel's launcher: where it says that a wait ran out (late_word())
};

// Sequences of a paged step of many (sequence, head) pairs that are faster on the 64-row tiles, several of which share an SM, than on
// prefill_attn_kernel, whose CTA fills one: few query rows over few keys (no longer sequence is short if one is not).  64 sequences of 32 heads,
// tiles / prefill kernel, us: heads of 128, 64 rows over 64, 164, 264, 364 keys 64 / 115, 127 / 164, 188 / 195, 235 / 191, 100 rows over 100 and 200 keys 146 / 129,
// 277 / 172; heads of 64, 64 rows over 64, 564, 1064 keys 36 / 98, 180 / 210, 328 / 306, 128 rows over 128, 192, 328 keys 82 / 109, 116 / 139, 217 / 164.
__host__ __device__ inline bool short_for_prefill(int d, int len_q, int len_k) {
    return d <= 64 ? (len_q <= 64 ? len_k <= 1024 : len_q <= 128 && len_k <= 192) : len_q <= 64 && len_k <= 256;
}

}  // namespace atoma
