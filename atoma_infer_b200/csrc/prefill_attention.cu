// Prefill / dense attention forward on the 5th-generation tensor cores (tcgen05 + TMEM) for
// sm_100a: contiguous or paged K/V, head dim 64 or 128, causal or not, varlen or batched, GQA.
// This is the path `flash_attn_varlen` takes at prefill (reference csrc/src/lib.rs:606-1103 ->
// run_mha -> flash_fwd_kernel, csrc/kernels/flash_fwd_kernel.h:56-500) and `flash_attn` (:31-343).
//
// Same contract as the reference (fp32 scores, exp2-domain online softmax, P rounded to the io type
// before P.V, fp32 accumulation, one final 1/rowsum, bottom-right aligned causal mask mask.h:171-172,
// rows without a visible key -> 0); the execution model is new:
//  * one CTA = one 128-row query tile of one head; K/V tiles of 128 keys stream through a 2-stage
//    TMA ring (128-byte swizzle boxes straight from the [tokens, heads, d] layout);
//  * warp 1 issues S = Q K^T (tcgen05.mma, A and B from shared memory, 128x128 fp32 accumulator in
//    TENSOR MEMORY, double buffered) and O += P V (A = P read from tensor memory, B = V from shared
//    memory as an MN-major operand, 128 x D fp32 accumulator in tensor memory);
//  * the softmax warps own one query row per thread (TMEM lane = row), or half of its keys (SPLIT 2): tcgen05.ld the scores of the row,
//    softmax them with a LAZY running maximum (the reference maximum is only moved, and O rescaled in
//    tensor memory, when a row's maximum grows by more than 2^8 — otherwise exp2 stays in range and
//    no correction pass is needed), write P back over S as packed 16-bit pairs (tcgen05.st);
//  * QK^T of tile j+1 is issued before P.V of tile j, so the tensor pipe works while tile j is being
//    exponentiated; the epilogue reads O from tensor memory, scales by 1/rowsum and stores 16-byte
//    vectors;
//  * tiles that stick out of their sequence (ragged tails) are loaded with cp.async + zero fill in
//    the same swizzled layout instead of TMA, so nothing outside a sequence is ever multiplied in;
//  * query / key heads may be longer than value heads (KH 64-column pieces of them, zero-filled behind their
//    last entry): 128 columns over values of 64, 192 over values of 128 (one key stage instead of two there:
//    two query tiles, one key and two value stages take 208 KB of shared memory);
//  * every wait is bounded: a wait that runs out stops the CTA's loads and lets its other roles run through,
//    its copies in flight are waited for (again with a bound), tensor memory is freed and a counter is
//    raised that the host can read (atoma_prefill_timeouts, atoma_kernel_timeouts); the CTA's outputs mean nothing then.
//
//  * paged keys and values (PAGED): three warps look the pages up and copy rows of 16-byte pieces with cp.async into the same
//    swizzled tiles (a page's rows of one head are strided: no box of a tensor map covers a tile of pages in any order), or, in long steps, all keys and values are
//    gathered first (try_launch_gathered);
//  * a quarter of the exponentials is a polynomial on the FMA pipe (exp2_poly2), and all heads' heaviest tiles start first;
//  * an output gate is applied in the epilogue (fetched before the last P.V is waited for), so no pass over the outputs follows.
//
// Bound: a tile's chain of products (S, then P V: 1300 to 1600 cycles, Q K^T at 100 instead of 64 per 128 x 128 x 16 since both operands come from
// shared memory) and softmax (1700 to 2000), which the two query tiles of a CTA run in turn: 3500 cycles per 128 keys of 256 rows; without any
// softmax the products alone take 3000.  Algorithmic flops: 4 * sum_b(visible (q,k) pairs) * D per head.
//  * Causal 8192 tokens, float16, 32 heads of 128: 627 -> 576 us by the share of polynomial exponentials and the order of the tiles (none, 3/8 and 1/2
//    of them were slower), 575 -> 562 with the maximum beside the exponentials (kEager).
//  * Portions of 1500 tokens and less over prefixes in pages: 765 us on the mma.sync tiles, 190 with one thread a row and two loading warps, 154 with two threads a
//    row, which halve the corrections, and three loading warps that hand a tile on at once.
//  * Window of 4096 tokens with a distance table and a gate: 310 us with one thread a row and clamps on the diagonal and across the table's end, 208 with two (more
//    of the biases' reads in flight) and none.
#include "common.cuh"
#include "mha_params.h"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <type_traits>
#include <vector>

namespace atoma {

bool launch_attention_tile(const MhaParams &p, bool is_bf16, cudaStream_t stream);   // attention_tile.cu

namespace {

// Threads: warpgroup 0 loads (warp 0) and issues the products (warp 1); then SPLIT softmax warpgroups per query tile, each of which takes 128 / SPLIT keys of a tile.
template <int SPLIT>
constexpr int kPfThreads = 128 + 256 * SPLIT;
constexpr int kPfM = 128, kPfN = 128;
constexpr int kQTiles = 2;       // two 128-row query tiles per CTA
constexpr int kVStages = 2;
constexpr int kPfWaitTries = 1 << 18;   // milliseconds at least (a try may also suspend the thread for a hardware-chosen time)
constexpr int kTmemCols = 512;   // S_A 0..127 | S_B 128..255 | O_A 256.. | O_B 384..
template <int SPLIT>
constexpr int kPfIssueRegs = SPLIT == 1 ? 56 : 64;
template <int SPLIT>
constexpr int kPfSoftmaxRegs = SPLIT == 1 ? 224 : 104;  // setmaxnreg: 168 * 384 = 56 * 128 + 224 * 256; 96 * 640 = 64 * 128 + 104 * 512
constexpr float kRescaleThreshold = 8.f;  // log2 units: P <= 2^8 between corrections
constexpr int kPfBiasSmem = 2048;         // distances whose bias (this head's column of the table) is kept in shared memory
// ... behind copies of its first row and in front of copies of its last (of a longer table: the rows that follow), so that a tile on the diagonal (distances
// from -254 on), across the table's end or within a longer table's first rows reads its biases without a clamp: with one, such a tile took 9000 to 12000
// cycles where others take 3000 (4000 tokens under a table of 4096 rows, heads of 64 and 128: 651 and 686 us with clamps in all tiles, 432 and 471).
constexpr int kPfBiasFront = 256, kPfBiasBack = 160;

__device__ unsigned int g_prefill_late;   // CTAs that gave up waiting, since the library was loaded

template <int D, int KH>
struct PfCfg {
    static constexpr int kHalfBytes = 128 * 128;             // 128 rows of 128 bytes
    static constexpr int kQkBytes = KH * kHalfBytes;         // one Q / K tile
    static constexpr int kVBytes = (D / 64) * kHalfBytes;    // one V tile
    static constexpr int kKStages = KH > 2 ? 1 : 2;
    static constexpr int kSmem = kQkBytes * (kQTiles + kKStages) + kVBytes * kVStages + 1024;
};

// A bounded wait; `late` (shared) is raised when the bound is reached.  The MMA and softmax warps then run on through their loops on
// whatever is in shared and tensor memory (every access stays in bounds, every arrival they owe is made); only the loads stop
// (pf_wait_all).
__device__ __forceinline__ void pf_wait(uint64_t *bar, uint32_t parity, volatile int *late) {
#pragma unroll 1
    for (int i = 0; !mbar_try_wait(bar, parity);)
        if (++i == kPfWaitTries) {
            *late = 1;
            break;
        }
}
// The same for a whole (converged) warp, with one answer for all lanes: false when the wait, or any other wait of the CTA, ran out.
__device__ __forceinline__ bool pf_wait_all(uint64_t *bar, uint32_t parity, volatile int *late) {
    pf_wait(bar, parity, late);
    return !__any_sync(0xffffffffu, *late != 0);
}

// ---- the exponential of the softmax, on packed float32 pairs ----
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
// 2^x of a pair on the FMA pipe: x = n + f, n the nearest integer (the sum with 1.5 * 2^23 holds it in its low bits), 2^f by a degree-6
// polynomial with constant term 1, the least-maximum fit over [-1/2, 1/2] by reweighted least squares, times 2^n: 7.4e-8 off at most, 2.6e-8 in the mean
// square (ex2.approx 1.45e-7 and 5.8e-8, measured over [-126, 8]; degree 5 1.65e-7 and 6.6e-8).  As with ex2.approx.ftz what is below
// 2^-126 is 0 (n = -127 gives the factor 0), and NaN stays NaN.
__device__ __forceinline__ void exp2_poly2(uint64_t x2, float &p0, float &p1) {
    float x0, x1;
    upk2(x2, x0, x1);
    asm("max.NaN.f32 %0, %0, 0fC2FE0000;" : "+f"(x0));   // -127
    asm("max.NaN.f32 %0, %0, 0fC2FE0000;" : "+f"(x1));
    x2 = pk2(x0, x1);
    const uint64_t big = pk2(12582912.f, 12582912.f), minus_big = pk2(-12582912.f, -12582912.f), minus = pk2(-1.f, -1.f);
    const uint64_t t = add2(x2, big), f = fma2(add2(t, minus_big), minus, x2);
    uint64_t y = fma2(f, pk2(0.00015353361959569156f, 0.00015353361959569156f), pk2(0.0013398875016719103f, 0.0013398875016719103f));
    y = fma2(y, f, pk2(0.00961843691766262f, 0.00961843691766262f));
    y = fma2(y, f, pk2(0.055503327399492264f, 0.055503327399492264f));
    y = fma2(y, f, pk2(0.24022646248340607f, 0.24022646248340607f));
    y = fma2(y, f, pk2(0.6931471824645996f, 0.6931471824645996f));
    y = fma2(y, f, pk2(1.f, 1.f));
    float t0, t1;
    upk2(t, t0, t1);
    const uint64_t scale = pk2(__uint_as_float((__float_as_uint(t0) << 23) + 0x3f800000u), __uint_as_float((__float_as_uint(t1) << 23) + 0x3f800000u));
    upk2(mul2_ftz(y, scale), p0, p1);
}
// P = 2^(s sc - m) of 32 scores as packed 16-bit pairs, and their sum.  MIX: every fourth pair leaves the special-function unit for the FMA
// pipe (the unit's 16 results a cycle and SM are what bounds the softmax of heads of 64 and 128).  Tiles with masked scores, and tiles whose FMA pipe
// adds a bias to every score, take the unit for all.
// MAX: the scores' maximum is taken beside them.
template <typename T, bool MIX, bool MAX>
__device__ __forceinline__ void softmax_chunk(const uint32_t *sv, uint64_t sc2, uint64_t mm2, uint64_t (&ls)[2], uint32_t (&pk)[16], float (&mx)[4]) {
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        if (MAX) mx[i & 3] = max3(mx[i & 3], __uint_as_float(sv[2 * i]), __uint_as_float(sv[2 * i + 1]));
        const uint64_t x2 = fma2(pk2(__uint_as_float(sv[2 * i]), __uint_as_float(sv[2 * i + 1])), sc2, mm2);
        float p0, p1;
        if (MIX && (i & 3) == 3) {
            exp2_poly2(x2, p0, p1);
        } else {
            upk2(x2, p0, p1);
            p0 = fast_exp2(p0);
            p1 = fast_exp2(p1);
        }
        ls[i & 1] = add2(ls[i & 1], pk2(p0, p1));
        pk[i] = pack2<T>(p0, p1);
    }
}
// ... of a thread's N scores, P to tensor memory.
template <typename T, int N, bool MIX, bool MAX>
__device__ __forceinline__ void softmax_scores(const uint32_t *sv, uint64_t sc2, uint64_t mm2, float &l, float (&mx)[4], uint32_t tmem_p) {
    uint64_t ls[2] = {0ull, 0ull};
#pragma unroll
    for (int c = 0; c < N / 32; ++c) {
        uint32_t pk[16];
        softmax_chunk<T, MIX, MAX>(sv + c * 32, sc2, mm2, ls, pk, mx);
        tmem_st_32x32b_x16(tmem_p + c * 16, pk);
    }
    float l0, l1;
    upk2(add2(ls[0], ls[1]), l0, l1);
    l = l0 + l1;
}

struct PfSeq {
    int len_q, len_k;
    int q_row0, k_row0;      // TMA row coordinate of the sequence's first token
    int q_batch, k_batch;    // TMA batch coordinate
    int64_t q_off, o_off, k_off, v_off;  // element offsets of the sequence's first token
    int q_start;             // cu_q[b] or -1
};

template <bool ROWS>   // gathered keys: sequence b's start at b k_bs, and there are k_batched of them
__device__ __forceinline__ PfSeq pf_seq(const MhaParams &p, int bidb) {
    PfSeq s;
    // reference block_info.h:14-36
    s.q_start = p.cu_q ? p.cu_q[bidb] : -1;
    s.len_q = p.cu_q ? p.cu_q[bidb + 1] - s.q_start : p.seqlen_q;
    const int k_first = (p.cu_k && p.k_cumulative) ? p.cu_k[bidb] : -1, k_start = ROWS ? -1 : k_first;
    const int len_k_cache = p.cu_k ? (p.k_cumulative ? p.cu_k[bidb + 1] - k_first : p.cu_k[bidb]) : p.seqlen_k;
    s.len_k = p.seqused_k ? p.seqused_k[bidb] : len_k_cache;
    if (ROWS) s.len_k = min(s.len_k, p.k_batched);   // the rows that there are
    s.q_off = s.q_start < 0 ? bidb * p.q_bs : static_cast<int64_t>(s.q_start) * p.q_rs;
    s.o_off = s.q_start < 0 ? bidb * p.o_bs : static_cast<int64_t>(s.q_start) * p.o_rs;
    s.k_off = k_start < 0 ? bidb * p.k_bs : static_cast<int64_t>(k_start) * p.k_rs;
    s.v_off = k_start < 0 ? bidb * p.v_bs : static_cast<int64_t>(k_start) * p.v_rs;
    s.q_row0 = s.q_start < 0 ? 0 : s.q_start;
    s.q_batch = s.q_start < 0 ? bidb : 0;
    s.k_row0 = k_start < 0 ? 0 : k_start;
    s.k_batch = k_start < 0 ? bidb : 0;
    return s;
}

// SPLIT: softmax threads per query row.
// BIASED: a bias by query-key distance is added to the scaled scores (MhaParams::dist_bias).  Instantiations of their own, so
// that the unbiased kernel keeps its register allocation.
// PAGED: keys and values lie in pages behind a block table (MhaParams::block_table).
// EXACT: the results of a paged step, to the bit, where its keys and values have been gathered (paged_rows_kernel).
template <typename T, int D, int KH, bool BIASED, bool PAGED, int SPLIT, bool EXACT>
__global__ void __launch_bounds__(kPfThreads<SPLIT>, 1)
prefill_attn_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                    const __grid_constant__ CUtensorMap map_v, const MhaParams p) {
    using C = PfCfg<D, KH>;
    constexpr int kKStages = C::kKStages;
    extern __shared__ unsigned char smem_dyn[];
    unsigned char *tiles = smem_dyn + ((1024u - (smem_u32(smem_dyn) & 1023u)) & 1023u);
    unsigned char *sq = tiles;                            // [q tile]
    unsigned char *sk = sq + kQTiles * C::kQkBytes;       // [stage]
    unsigned char *sv = sk + kKStages * C::kQkBytes;      // [stage]
    __shared__ __align__(8) uint64_t q_full[kQTiles], k_full[kKStages], k_empty[kKStages], v_full[kVStages],
        v_empty[kVStages], s_full[kQTiles], p_full[kQTiles], pv_done[kQTiles];
    __shared__ uint32_t tmem_base_smem;
    __shared__ int late_s;
    volatile int *late = &late_s;
    constexpr int N = kPfN / SPLIT;   // keys of a tile per softmax thread
    // Paged steps correct by every new maximum: a row's largest weight is then 1, which rounding to 16 bits leaves alone, as on the tile kernel, whose steps
    // these are (error against 64 bits of bfloat16 portions, queries of 1 and 4 times unit size: 2.08e-3 and 1.73e-3 there, 2.09e-3 and 1.74e-3 here,
    // 2.13e-3 and 2.09e-3 with corrections from 2^8 on; the portions of prompts over prefixes 180 -> 190 us).
    constexpr float kThreshold = PAGED || EXACT ? 0.f : kRescaleThreshold;
    // Where most tiles correct nothing (8192 tokens of 32 heads, float16: 575 us without, 562 so).  A thread of half the keys would have to learn of the other's
    // maximum all the same; heads of 64 gain nothing (414 us, 428).
    constexpr bool kEager = SPLIT == 1 && !PAGED && !EXACT && D == 128;
    constexpr int kCorrect = SPLIT == 1 ? 32 : 16;   // columns of O that a correction holds
    __shared__ float bias_s[BIASED ? kPfBiasFront + kPfBiasSmem + kPfBiasBack : 1];
    __shared__ float swap_s[2][kQTiles][2][SPLIT == 2 ? kPfM : 1];         // a row's maximum (at the end: its sum) over either half of the keys

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // Heads, then sequences, then query tiles from the last (causal: heaviest) one down, so that the SMs run out of light tiles together
    // (head by head, one prompt of 8192 x 32 heads kept them 0.86 busy; under a window of 256, 1024 and 4096 4000 tokens of 32 heads of 128 take 108,
    // 154 and 242 us head by head, 105, 145 and 206 so).  Tiles behind a sequence's end leave at once.
    const int m_block = gridDim.z - 1 - blockIdx.z, head = blockIdx.x, bidb = blockIdx.y;
    pdl_wait();
    const PfSeq si = pf_seq<EXACT>(p, bidb);
    if (m_block * kQTiles * kPfM >= si.len_q || (PAGED && p.split_short && short_for_prefill(D, si.len_q, si.len_k))) return;

    if (tid == 0) {
        late_s = 0;
        for (int i = 0; i < kKStages; ++i) {
            mbar_init(&k_full[i], 1);
            mbar_init(&k_empty[i], 1);
        }
        for (int i = 0; i < kVStages; ++i) {
            mbar_init(&v_full[i], 1);
            mbar_init(&v_empty[i], 1);
        }
        for (int i = 0; i < kQTiles; ++i) {
            mbar_init(&q_full[i], 1);
            mbar_init(&s_full[i], 1);
            mbar_init(&p_full[i], 4 * SPLIT);  // one arrival per softmax warp
            mbar_init(&pv_done[i], 1);
        }
        fence_mbar_init();
        tma_prefetch_desc(&map_q);
        tma_prefetch_desc(&map_k);
        tma_prefetch_desc(&map_v);
    }
    const int bias_n = BIASED ? min(p.dist_rows, kPfBiasSmem) : 0;
    if (BIASED)
        for (int i = tid; i < kPfBiasFront + bias_n + kPfBiasBack; i += kPfThreads<SPLIT>)
            bias_s[i] = p.dist_bias[static_cast<int64_t>(min(max(i - kPfBiasFront, 0), p.dist_rows - 1)) * p.dist_heads + head] * 1.4426950408889634f;
    if (warp == 1) tmem_alloc(&tmem_base_smem, kTmemCols);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = tmem_base_smem;
    pdl_launch_dependents();

    const int len_q = si.len_q, len_k = si.len_k;
    const int shift = len_k - len_q;  // mask.h:171-172: key j visible to query i iff j <= i + shift
    const bool skip = p.min_len_q > 0 && len_q < p.min_len_q;   // the caller serves this sequence elsewhere
    const int window = (p.is_causal && p.window_left > 0) ? p.window_left : 0;
    // Query tile t of this CTA covers rows m0[t] .. m0[t] + 127 and needs the first nt[t] key tiles.
    int m0[kQTiles], nt[kQTiles];
#pragma unroll
    for (int t = 0; t < kQTiles; ++t) {
        m0[t] = (m_block * kQTiles + t) * kPfM;
        nt[t] = 0;
        if (m0[t] < len_q && !skip) {
            nt[t] = (len_k + kPfN - 1) / kPfN;
            if (p.is_causal) {
                const int lim = min(m0[t] + kPfM, len_q) + shift;  // one past the last visible key of the tile
                nt[t] = min(nt[t], lim <= 0 ? 0 : (lim + kPfN - 1) / kPfN);
            }
        }
    }
    const int n_max = max(nt[0], nt[1]);
    // Sliding window: the CTA starts at the key tile that holds the lowest key its first row can see (both query tiles
    // start there: the later one's extra tiles are masked out, which the running softmax takes like any masked tile).
    // Stage indices and barrier parities below count tiles from n_lo.
    int n_lo = 0;
    if (window > 0) {
        const int first_key = m0[0] + shift - window + 1;
        n_lo = first_key > 0 ? first_key / kPfN : 0;
    }
    const int kvh = head / (p.h / p.h_k);  // flash_fwd_kernel.h:593

    // ================================ paged loads: warps 2, 3 and, behind the queries, 0 ================================
    // Pages are a few rows each, too small for a copy by the TMA unit each (a warp starts about six a microsecond); the 16-byte pieces of a tile of keys
    // or values go by cp.async.  The tiles, K V K V .., go round the three warps; a warp hands a tile on as soon as its pieces have landed, while the
    // others' tiles are under way (two warps that handed a tile on only behind their next one's copies, which wait for a free stage, made a tile
    // of 128 keys cost 6700 cycles instead of 3500).  A lane looks up the rows 32 i + lane of a tile, and every piece asks for its row's place by shuffle.
    [[maybe_unused]] auto paged_loads = [&](int worker) {
        constexpr int kPieces = D / 8, kRowsPer = 32 / kPieces, kStages = 2;
        static_assert(!PAGED || (kKStages == 2 && kVStages == 2 && KH == D / 64), "keys and values are loaded alike");
        const int *table = p.block_table + static_cast<int64_t>(bidb) * p.bt_bs;
        const int piece = lane % kPieces, sub = lane / kPieces;
        for (int u = worker; u < 2 * (n_max - n_lo); u += 3) {
            const bool keys = (u & 1) == 0;
            const int jj = u >> 1, j = n_lo + jj, st = jj % kStages, left = len_k - j * kPfN;   // rows of the sequence from this tile on
            const T *base = static_cast<const T *>(keys ? p.k : p.v) + static_cast<int64_t>(kvh) * (keys ? p.k_hs : p.v_hs) + piece * 8;
            const int64_t bs = keys ? p.k_bs : p.v_bs, rs = keys ? p.k_rs : p.v_rs;
            int64_t place[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int r = 32 * i + lane, key = j * kPfN + r;
                const int pg = key / p.page;   // entries past the sequence's end are never read
                place[i] = r < left ? static_cast<int64_t>(table[pg]) * bs + static_cast<int64_t>(key - pg * p.page) * rs : 0;
            }
            if (!pf_wait_all(keys ? &k_empty[st] : &v_empty[st], ((jj / kStages) & 1) ^ 1, late)) break;
            const uint32_t dst = smem_u32((keys ? sk : sv) + st * C::kVBytes) + (piece >> 3) * C::kHalfBytes;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
#pragma unroll 4
                for (int q = 0; q < kPieces; ++q) {
                    const int rr = q * kRowsPer + sub, r = 32 * i + rr;
                    const int64_t at = __shfl_sync(0xffffffffu, place[i], rr);
                    cp_async_16(dst + r * 128 + (((piece & 7) ^ (r & 7)) << 4), base + at, r < left ? 16 : 0);
                }
            }
            cp_async_commit();
            cp_async_wait_all();
            fence_proxy_async();       // generic-proxy writes -> visible to the tensor core's async reads
            __syncwarp();
            if (lane == 0) mbar_arrive(keys ? &k_full[st] : &v_full[st]);
        }
    };

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kPfIssueRegs<SPLIT>));
        if (warp == 0 && n_max > 0) {
            // ================================ loads ================================
            // A tile that lies completely inside its sequence is one TMA transaction (kHalves boxes);
            // a ragged one is filled with cp.async + zero fill in the same 128-byte-swizzled layout.
            // Q and K tiles are KH pieces of 64 columns, V tiles D / 64; columns from `cols` on are zero (TMA's fill).
            [[maybe_unused]] auto load_tile = [&](auto pieces, int cols, unsigned char *dst, const CUtensorMap *map, uint64_t *bar, const T *gbase,
                                 int64_t rs, int row0, int len, int tma_row, int tma_head, int tma_batch,
                                 uint64_t policy) {
                constexpr int NP = decltype(pieces)::value;
                if (row0 + 128 <= len) {
                    if (elect_one_sync()) {
                        mbar_arrive_expect_tx(bar, NP * C::kHalfBytes);
#pragma unroll
                        for (int hf = 0; hf < NP; ++hf)
                            tma_load_4d(dst + hf * C::kHalfBytes, map, bar, hf * 64, tma_head, tma_row, tma_batch, policy);
                    }
                    __syncwarp();
                } else {
                    for (int idx = lane; idx < 128 * NP * 8; idx += 32) {
                        const int r = idx / (NP * 8), c = idx % (NP * 8);
                        const bool ok = row0 + r < len && c * 8 < cols;
                        const T *src = ok ? gbase + static_cast<int64_t>(row0 + r) * rs + c * 8 : gbase;
                        cp_async_16(smem_u32(dst + (c >> 3) * C::kHalfBytes + r * 128 + (((c & 7) ^ (r & 7)) << 4)), src,
                                    ok ? 16 : 0);
                    }
                    cp_async_commit();
                    cp_async_wait_all();
                    fence_proxy_async();  // generic-proxy writes -> visible to the tensor core's async reads
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar);
                }
            };
            using QkPieces = std::integral_constant<int, KH>;
            using VPieces = std::integral_constant<int, D / 64>;
            const int d_k = p.d_k > 0 ? p.d_k : D;
            const T *qg = static_cast<const T *>(p.q) + si.q_off + static_cast<int64_t>(head) * p.q_hs;
            const T *kg = static_cast<const T *>(p.k) + si.k_off + static_cast<int64_t>(kvh) * p.k_hs;
            const int vh = p.v_share > 1 ? kvh / p.v_share : kvh;
            const T *vg = static_cast<const T *>(p.v) + si.v_off + static_cast<int64_t>(vh) * p.v_hs;
#pragma unroll
            for (int t = 0; t < kQTiles; ++t)
                if (nt[t] > 0)
                    load_tile(QkPieces(), d_k, sq + t * C::kQkBytes, &map_q, &q_full[t], qg, p.q_rs, m0[t], len_q, si.q_row0 + m0[t],
                              head, si.q_batch, kL2EvictFirst);
            const int there = EXACT ? 1 << 30 : len_k;   // gathered rows are whole tiles
            int k_issued = 0, v_issued = 0;
            if constexpr (PAGED) paged_loads(2);
            for (int j = n_lo; !PAGED && j < n_max; ++j) {
                const int jj = j - n_lo, ks = jj % kKStages, vs = jj % kVStages;
                if (!pf_wait_all(&k_empty[ks], ((jj / kKStages) & 1) ^ 1, late)) break;
                load_tile(QkPieces(), d_k, sk + ks * C::kQkBytes, &map_k, &k_full[ks], kg, p.k_rs, j * kPfN, there,
                          si.k_row0 + j * kPfN, kvh, si.k_batch, kL2EvictLast);
                ++k_issued;
                if (!pf_wait_all(&v_empty[vs], ((jj / kVStages) & 1) ^ 1, late)) break;
                load_tile(VPieces(), D, sv + vs * C::kVBytes, &map_v, &v_full[vs], vg, p.v_rs, j * kPfN, there,
                          si.k_row0 + j * kPfN, vh, si.k_batch, kL2EvictLast);
                ++v_issued;
            }
            // whatever happens to the other roles, the copies have landed before this warp leaves
            auto landed = [&](uint64_t *bar, uint32_t parity) {
                for (int i = 0; i < kPfWaitTries && !mbar_try_wait(bar, parity); ++i) {
                }
            };
            for (int t = 0; t < kQTiles; ++t)
                if (nt[t] > 0) landed(&q_full[t], 0);
            for (int i = max(0, k_issued - kKStages); i < k_issued; ++i) landed(&k_full[i % kKStages], (i / kKStages) & 1);
            for (int i = max(0, v_issued - kVStages); i < v_issued; ++i) landed(&v_full[i % kVStages], (i / kVStages) & 1);
        } else if (PAGED && warp >= 2 && n_max > 0) {
            paged_loads(warp - 2);
        } else if (warp == 1 && n_max > 0) {
            // ================================ MMA issue ================================
            // The whole warp runs this role converged on warp-uniform values; only the tcgen05
            // instructions sit under elect.sync.  (Under `if (lane == 0)` the loop took ~70 cycles per
            // product against the 64 cycles a 128x128x16 product occupies the tensor pipe — the issue
            // thread, not the pipe, was the limit of a first version: tensor pipe 49 % active.)
            // Order per key tile j:  P.V(A,j)  QK(A,j+1)  P.V(B,j)  QK(B,j+1)
            // so while one query tile is being exponentiated the tensor pipe works for the other.
            constexpr bool kBf16 = std::is_same<T, __nv_bfloat16>::value;
            const uint32_t idesc_qk = umma_idesc_f16(kPfM, kPfN, kBf16, false);
            const uint32_t idesc_pv = umma_idesc_f16(kPfM, D, kBf16, true);
            auto issue_qk = [&](int t, int j) {
                const uint32_t q_addr = smem_u32(sq + t * C::kQkBytes);
                const uint32_t k_addr = smem_u32(sk + (j - n_lo) % kKStages * C::kQkBytes);
                const uint32_t tmem_s = tmem_base + t * 128;
                if (elect_one_sync()) {
#pragma unroll
                    for (int kk = 0; kk < KH * 4; ++kk) {
                        const uint32_t off = (kk >> 2) * C::kHalfBytes + (kk & 3) * 32;
                        umma_f16_ss(tmem_s, umma_desc_k_sw128(q_addr + off), umma_desc_k_sw128(k_addr + off), idesc_qk,
                                    kk != 0 ? 1u : 0u);
                    }
                    umma_commit(&s_full[t]);
                }
                __syncwarp();
            };
            auto issue_pv = [&](int t, int j) {
                const uint32_t v_addr = smem_u32(sv + (j - n_lo) % kVStages * C::kVBytes);
                const uint32_t tmem_p = tmem_base + t * 128;
                const uint32_t tmem_o = tmem_base + 256 + t * 128;
                if (elect_one_sync()) {
#pragma unroll
                    for (int kk = 0; kk < kPfN / 16; ++kk) {
                        // 16 keys = 16 rows of 128 bytes of V; 16 P values = 8 packed 32-bit columns
                        umma_f16_ts(tmem_o, tmem_p + kk * 8, umma_desc_mn_sw128(v_addr + kk * 16 * 128, C::kHalfBytes),
                                    idesc_pv, ((j - n_lo) | kk) != 0 ? 1u : 0u);
                    }
                    umma_commit(&pv_done[t]);
                }
                __syncwarp();
            };
            // first key tile: both query tiles
            pf_wait(&k_full[0], 0, late);
#pragma unroll
            for (int t = 0; t < kQTiles; ++t) {
                if (nt[t] > 0) {
                    pf_wait(&q_full[t], 0, late);
                    tc_fence_after_sync();
                    issue_qk(t, n_lo);
                }
            }
            if (elect_one_sync()) umma_commit(&k_empty[0]);
            __syncwarp();
            for (int j = n_lo; j < n_max; ++j) {
                const int jj = j - n_lo;
                const int s = jj % kVStages, sn = (jj + 1) % kKStages;
                pf_wait(&v_full[s], (jj / kVStages) & 1, late);
                bool k_next_ready = false;
#pragma unroll
                for (int t = 0; t < kQTiles; ++t) {
                    if (j < nt[t]) {
                        pf_wait(&p_full[t], jj & 1, late);
                        tc_fence_after_sync();
                        issue_pv(t, j);
                    }
                    if (j + 1 < nt[t]) {
                        if (!k_next_ready) {
                            pf_wait(&k_full[sn], ((jj + 1) / kKStages) & 1, late);
                            k_next_ready = true;
                        }
                        tc_fence_after_sync();
                        issue_qk(t, j + 1);
                    }
                }
                if (elect_one_sync()) {
                    umma_commit(&v_empty[s]);                       // both P.V of tile j are issued
                    if (k_next_ready) umma_commit(&k_empty[sn]);    // ... and every QK^T of tile j + 1
                }
                __syncwarp();
            }
        }
    } else {
        // ================================ softmax / epilogue warpgroups ================================
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kPfSoftmaxRegs<SPLIT>));
        const int t = (warp - 4) / (4 * SPLIT), half = SPLIT == 2 ? ((warp - 4) >> 2) & 1 : 0;   // query tile and half of its keys of this warpgroup
        const int quad = warp & 3;
        const int row = quad * 32 + lane;       // query row of this thread within the tile
        const int m0t = t ? m0[1] : m0[0];
        const int grow = m0t + row;             // ... within the sequence
        const int n_tiles = t ? nt[1] : nt[0];
        const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
        const uint32_t tmem_s = tmem_base + lane_addr + t * 128;
        const uint32_t tmem_o = tmem_base + lane_addr + 256 + t * 128 + half * (D / SPLIT);   // this half corrects and stores half of O's columns
        T *og = static_cast<T *>(p.o) + si.o_off + static_cast<int64_t>(head) * p.o_hs +
                static_cast<int64_t>(grow) * p.o_rs + half * (D / SPLIT);
        int64_t lse_idx = 0;
        if (p.lse && grow < len_q) {
            if (p.unpadded_lse && p.cu_q) lse_idx = static_cast<int64_t>(head) * p.cu_q[p.b] + si.q_start + grow;
            else lse_idx = (static_cast<int64_t>(bidb) * p.h + head) * p.seqlen_q + grow;
        }
        // The two warps of a row quad tell each other a value per row (both run the same tiles).  The exchanges of a row take two cells in turn: a cell is stored
        // to again behind the barrier of the exchange between, where the other warp arrives with the value that it read.
        [[maybe_unused]] auto swap = [&](int turn, float mine) {
            swap_s[turn & 1][t][half][row] = mine;
            tc_fence_before_sync();
            asm volatile("bar.sync %0, 64;" ::"r"(1 + t * 4 + quad) : "memory");
            tc_fence_after_sync();
            return swap_s[turn & 1][t][half ^ 1][row];
        };
        if (n_tiles > 0) {
            float m_ref = -INFINITY, l_run = 0.f;
            [[maybe_unused]] float l_high = 0.f;   // EXACT: the second half of the keys apart, as two threads sum them
            if (p.sink) {   // the sink is one more term of the denominator: the running state starts from it
                m_ref = p.sink[head] * 1.4426950408889634f;
                l_run = half ? 0.f : 1.f;
            }
            for (int j = n_lo; j < n_tiles; ++j) {
                pf_wait(&s_full[t], (j - n_lo) & 1, late);
                tc_fence_after_sync();
                uint32_t sv_[N];
#pragma unroll
                for (int c = 0; c < N / 32; ++c) tmem_ld_32x32b_x32(tmem_s + half * N + c * 32, sv_ + c * 32);
                tmem_ld_wait();
                const int col0 = j * kPfN + half * N;
                // ---- bias by distance: the scores move to the scaled log2 domain here, and `sc` below becomes 1; where all of the warp's keys lie
                // beyond the table's last row the bias is one value, which goes into the exponent with the maximum ----
                float sc = p.scale_log2, far_bias = 0.f;
                bool far = !BIASED;
                if constexpr (BIASED) {
                    const int d0 = grow + shift - col0, last = p.dist_rows - 1;   // distance of this row to the half's first key
                    const float sl2 = sc;
                    if (__all_sync(0xffffffffu, d0 - (N - 1) >= last) && last < bias_n) {
                        far = true;
                        far_bias = bias_s[kPfBiasFront + last];
                    } else if (__all_sync(0xffffffffu, d0 - (N - 1) >= -kPfBiasFront && d0 < bias_n + kPfBiasBack)) {
                        // every distance of the tile is a row of the shared-memory copy: no clamps, constant offsets from one address
                        const float *bp = bias_s + kPfBiasFront + d0;
#pragma unroll
                        for (int c = 0; c < N; ++c) sv_[c] = __float_as_uint(fmaf(__uint_as_float(sv_[c]), sl2, bp[-c]));
                    } else {
#pragma unroll
                        for (int c = 0; c < N; ++c) {
                            const int dist = min(max(d0 - c, 0), last);
                            const float bv = dist < bias_n ? bias_s[kPfBiasFront + dist]
                                                           : __ldg(p.dist_bias + static_cast<int64_t>(dist) * p.dist_heads + head) * 1.4426950408889634f;
                            sv_[c] = __float_as_uint(fmaf(__uint_as_float(sv_[c]), sl2, bv));
                        }
                    }
                }
                if (!far) sc = 1.f;
                // ---- masks: only tiles that touch the sequence end or the causal diagonal ----
                const bool tail = col0 + N > len_k;
                const bool diag = p.is_causal && (col0 + N - 1 > m0t + shift);
                const bool low = window > 0 && col0 < m0t + kPfM + shift - window;   // some row's window starts inside or after this tile
                if (tail || diag || low) {
                    const int lim = p.is_causal ? min(len_k, grow + shift + 1) : len_k;  // first masked column
                    const int lb = window > 0 ? grow + shift - window + 1 : -(1 << 30);  // first visible column
#pragma unroll
                    for (int c = 0; c < N; ++c)
                        if (col0 + c >= lim || col0 + c < lb) sv_[c] = 0xff800000u;  // -inf
                }
                const bool masked = tail || diag || low;
                const uint64_t sc2 = pk2(sc, sc);
                const uint32_t tmem_p = tmem_s + half * (N / 2);
                // ---- P = exp2(S * scale - m), row sum, packed 16-bit pairs back over S ----
                // Most tiles move no row's reference maximum: the exponentials start from the one at hand and the tile's maximum is taken beside them.
                float l_tile = 0.f, mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
                bool done = false;
                if (kEager && j > n_lo && !masked) {
                    const float m_use = m_ref == -INFINITY ? 0.f : m_ref;
                    softmax_scores<T, N, true, true>(sv_, sc2, pk2(-m_use, -m_use), l_tile, mx4, tmem_p);
                    const float m_tile = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * sc;
                    done = !__any_sync(0xffffffffu, m_tile > m_ref + kThreshold);
                    if (!done) tmem_st_wait();   // P is written once more
                }
                if (!done) {
                    // eight independent chains: a single running maximum is a chain of dependent operations
                    float mx8[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) mx8[i] = max3(__uint_as_float(sv_[i]), __uint_as_float(sv_[8 + i]), __uint_as_float(sv_[16 + i]));
#pragma unroll
                    for (int c = 24; c + 15 < N; c += 16)
#pragma unroll
                        for (int i = 0; i < 8; ++i) mx8[i] = max3(mx8[i], __uint_as_float(sv_[c + i]), __uint_as_float(sv_[c + 8 + i]));
#pragma unroll
                    for (int i = 0; i < 8; ++i) mx8[i] = fmaxf(mx8[i], __uint_as_float(sv_[N - 8 + i]));
                    const float mx = fmaxf(max3(mx8[0], mx8[1], mx8[2]), fmaxf(max3(mx8[3], mx8[4], mx8[5]), fmaxf(mx8[6], mx8[7])));
                    float m_tile = BIASED ? fmaf(mx, sc, far_bias) : mx * sc;  // scale_log2 > 0 (checked on the host)
                    if constexpr (SPLIT == 2) m_tile = fmaxf(m_tile, swap(j - n_lo, m_tile));   // both halves' scores are in registers: P may be written over them
                    // ---- running maximum ----
                    const bool need = m_tile > m_ref + kThreshold;  // also the first finite tile (m_ref = -inf)
                    if (__any_sync(0xffffffffu, need)) {
                        const float alpha = need ? (m_ref == -INFINITY ? 0.f : fast_exp2(m_ref - m_tile)) : 1.f;
                        if (need) m_ref = m_tile;
                        l_run *= alpha;
                        if (EXACT) l_high *= alpha;
                        if (j > n_lo) {
                            // O of this row lives in tensor memory: wait until P.V of the previous tile has
                            // been accumulated, rescale, write back.  Rare after the first tiles.
                            pf_wait(&pv_done[t], (j - 1 - n_lo) & 1, late);
                            tc_fence_after_sync();
#pragma unroll 1
                            for (int c = 0; c < D / SPLIT; c += kCorrect) {       // the scores hold most registers
                                uint32_t ov[kCorrect];
#pragma unroll
                                for (int i = 0; i < kCorrect; i += 16) tmem_ld_32x32b_x16(tmem_o + c + i, *reinterpret_cast<uint32_t (*)[16]>(ov + i));
                                tmem_ld_wait();
#pragma unroll
                                for (int i = 0; i < kCorrect; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * alpha);
#pragma unroll
                                for (int i = 0; i < kCorrect; i += 16) tmem_st_32x32b_x16(tmem_o + c + i, ov + i);
                            }
                            tmem_st_wait();
                        }
                    }
                    const float m_use = m_ref == -INFINITY ? 0.f : m_ref;
                    const float off = BIASED ? far_bias - m_use : -m_use;
                    const uint64_t mm2 = pk2(off, off);
                    if constexpr (EXACT) {   // half by half, each by its own masks, as two threads a row have it
                        static_assert(SPLIT == 1 && !BIASED, "one thread a row");
                        constexpr int M = N / 2;
                        const bool diag0 = p.is_causal && (col0 + M - 1 > m0t + shift), masked0 = col0 + M > len_k || diag0 || low, masked1 = tail || diag || (window > 0 && col0 + M < m0t + kPfM + shift - window);
                        float l_half = 0.f;
                        if (masked0) softmax_scores<T, M, false, false>(sv_, sc2, mm2, l_tile, mx4, tmem_p);
                        else softmax_scores<T, M, true, false>(sv_, sc2, mm2, l_tile, mx4, tmem_p);
                        if (masked1) softmax_scores<T, M, false, false>(sv_ + M, sc2, mm2, l_half, mx4, tmem_p + M / 2);
                        else softmax_scores<T, M, true, false>(sv_ + M, sc2, mm2, l_half, mx4, tmem_p + M / 2);
                        l_high += l_half;
                    } else if (masked || !far) softmax_scores<T, N, false, false>(sv_, sc2, mm2, l_tile, mx4, tmem_p);
                    else softmax_scores<T, N, true, false>(sv_, sc2, mm2, l_tile, mx4, tmem_p);
                }
                l_run += l_tile;
                tmem_st_wait();
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&p_full[t]);
            }
            // ---- epilogue: O / rowsum -> global ----
            const bool gated = p.gate && grow < len_q && (p.gate_below <= 0 || grow + shift + (p.key_lo ? p.key_lo[bidb] : 0) < p.gate_below);
            if constexpr (SPLIT == 2) {   // both halves' sums of a row, in the same order on both sides
                const float other = swap(n_tiles - n_lo, l_run);
                l_run = half ? other + l_run : l_run + other;
            }
            if (EXACT) l_run += l_high;
            // this half's part of the row's gate, 32 columns at a time: the first are under way while the last products run
            const T *gg = gated ? static_cast<const T *>(p.gate) + static_cast<int64_t>(si.q_row0 + grow) * p.gate_rs + static_cast<int64_t>(head) * D + half * (D / SPLIT) : nullptr;
            uint4 gv[4];
            if (gated) {
#pragma unroll
                for (int i = 0; i < 4; ++i) gv[i] = *reinterpret_cast<const uint4 *>(gg + i * 8);
            }
            pf_wait(&pv_done[t], (n_tiles - 1 - n_lo) & 1, late);
            tc_fence_after_sync();
            const bool empty = (l_run == 0.f || l_run != l_run);
            const float inv = empty ? 0.f : 1.f / l_run;
#pragma unroll
            for (int c = 0; c < D / 32 / SPLIT; ++c) {
                uint32_t ov[32];
                tmem_ld_32x32b_x32(tmem_o + c * 32, ov);
                tmem_ld_wait();
                if (grow < len_q) {
                    if (gated) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const T *ge = reinterpret_cast<const T *>(&gv[i]);
#pragma unroll
                            for (int e = 0; e < 8; ++e)
                                ov[8 * i + e] = __float_as_uint(over_one_plus(__uint_as_float(ov[8 * i + e]), expf(-static_cast<float>(ge[e]))));
                            if (c + 1 < D / 32 / SPLIT) gv[i] = *reinterpret_cast<const uint4 *>(gg + (c + 1) * 32 + i * 8);
                        }
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        uint4 w;
                        w.x = pack2<T>(__uint_as_float(ov[8 * i + 0]) * inv, __uint_as_float(ov[8 * i + 1]) * inv);
                        w.y = pack2<T>(__uint_as_float(ov[8 * i + 2]) * inv, __uint_as_float(ov[8 * i + 3]) * inv);
                        w.z = pack2<T>(__uint_as_float(ov[8 * i + 4]) * inv, __uint_as_float(ov[8 * i + 5]) * inv);
                        w.w = pack2<T>(__uint_as_float(ov[8 * i + 6]) * inv, __uint_as_float(ov[8 * i + 7]) * inv);
                        *reinterpret_cast<uint4 *>(og + c * 32 + i * 8) = w;
                    }
                }
            }
            if (p.lse && half == 0 && grow < len_q)
                p.lse[lse_idx] = empty ? INFINITY : m_ref * 0.6931471805599453f + __logf(l_run);
        } else if (grow < len_q && !skip) {
            // No visible key for any row of this tile: O = 0, LSE = +inf (flash_fwd_kernel.h:543-582).
#pragma unroll
            for (int c = 0; c < D / 8 / SPLIT; ++c) *reinterpret_cast<uint4 *>(og + c * 8) = make_uint4(0, 0, 0, 0);
            if (p.lse && half == 0) p.lse[lse_idx] = INFINITY;
        }
    }

    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, kTmemCols);
    }
    if (tid == 0 && *late) {
        atomicAdd(&g_prefill_late, 1u);
        if (p.late) *reinterpret_cast<volatile unsigned int *>(p.late) = 1;
    }
}

// Keys and values of a paged step into rows of their own: sequence b's from b * pitch on, all heads of a row together, and zeros up to a whole tile.  One warp per key; bound by
// the bytes (16-byte pieces).
constexpr int kPfGatherWarps = 8;
__global__ void __launch_bounds__(32 * kPfGatherWarps) paged_rows_kernel(const MhaParams p, uint4 *__restrict__ k_out, uint4 *__restrict__ v_out, int pitch) {
    pdl_launch_dependents();
    pdl_wait();
    const int b = blockIdx.y, key = blockIdx.x * kPfGatherWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    const PfSeq si = pf_seq<false>(p, b);
    const int keys = min(si.len_k, pitch), per = p.d / 8, pieces = p.h_k * per;
    if (key >= (keys + kPfN - 1) / kPfN * kPfN || si.len_q <= 0) return;
    if (key >= keys) {
        const int64_t row = (static_cast<int64_t>(b) * pitch + key) * pieces;
        for (int c = lane; c < pieces; c += 32) k_out[row + c] = v_out[row + c] = make_uint4(0, 0, 0, 0);
        return;
    }
    const int pg = key / p.page;
    const int64_t page = p.block_table[static_cast<int64_t>(b) * p.bt_bs + pg], in = key - pg * p.page, row = (static_cast<int64_t>(b) * pitch + key) * pieces;
    const uint16_t *k = static_cast<const uint16_t *>(p.k) + page * p.k_bs + in * p.k_rs, *v = static_cast<const uint16_t *>(p.v) + page * p.v_bs + in * p.v_rs;
#pragma unroll 4
    for (int c = lane; c < pieces; c += 32) {
        const int g = c / per, at = (c - g * per) * 8;
        const uint4 kv = *reinterpret_cast<const uint4 *>(k + g * p.k_hs + at), vv = *reinterpret_cast<const uint4 *>(v + g * p.v_hs + at);
        k_out[row + c] = kv;
        v_out[row + c] = vv;
    }
}

// ---------------------------------------------------------------------------------------------
struct Map4Key {
    const void *ptr;
    int64_t hs, rs, bs, rows, batches;
    int d, heads, bf16;
    bool operator==(const Map4Key &o) const { return std::memcmp(this, &o, sizeof(Map4Key)) == 0; }
};
struct Map4Entry {
    Map4Key key;
    CUtensorMap map;
};

// [batches][rows][heads][d] view with element strides; box = 128 rows x 64 d of one head.
bool make_attn_map(CUtensorMap *out, const void *ptr, int d, int heads, int64_t rows, int64_t batches,
                   int64_t hs, int64_t rs, int64_t bs, bool is_bf16) {
    static thread_local std::vector<Map4Entry> cache;
    Map4Key key;
    std::memset(&key, 0, sizeof(key));
    key.ptr = ptr; key.hs = hs; key.rs = rs; key.bs = bs; key.rows = rows; key.batches = batches;
    key.d = d; key.heads = heads; key.bf16 = is_bf16;
    for (const Map4Entry &e : cache)
        if (e.key == key) { *out = e.map; return true; }
    EncodeTiledFn enc = get_encode_tiled();
    if (!enc) return false;
    const cuuint64_t dims[4] = {static_cast<cuuint64_t>(d), static_cast<cuuint64_t>(heads),
                                static_cast<cuuint64_t>(rows), static_cast<cuuint64_t>(batches)};
    const cuuint64_t strides[3] = {static_cast<cuuint64_t>(hs) * 2, static_cast<cuuint64_t>(rs) * 2,
                                   static_cast<cuuint64_t>(bs) * 2};
    const cuuint32_t box[4] = {64, 1, 128, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = enc(out, is_bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4,
                     const_cast<void *>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_status(kErrDriver, "prefill: cuTensorMapEncodeTiled failed (CUresult %d)", static_cast<int>(r));
        return false;
    }
    if (cache.size() >= 256) cache.clear();
    cache.push_back(Map4Entry{key, *out});
    return true;
}

template <typename T, int D, int KH, bool BIASED, bool PAGED = false, bool EXACT = false>
bool launch_prefill_b(const CUtensorMap &mq, const CUtensorMap &mk, const CUtensorMap &mv, const MhaParams &p, cudaStream_t stream) {
    constexpr int SPLIT = BIASED || PAGED ? 2 : 1;
    constexpr size_t smem = PfCfg<D, KH>::kSmem;
    static thread_local int attr_dev = -1;
    const DeviceInfo &di = current_device_info();
    if (attr_dev != di.ordinal) {
        cudaError_t e = cudaFuncSetAttribute(prefill_attn_kernel<T, D, KH, BIASED, PAGED, SPLIT, EXACT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             static_cast<int>(smem));
        if (e != cudaSuccess) {
            set_status(static_cast<int>(e), "prefill: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
            return false;
        }
        attr_dev = di.ordinal;
    }
    MhaParams pp = p;
    pp.late = late_word();
    const dim3 grid(p.h, p.b, (p.seqlen_q + kQTiles * kPfM - 1) / (kQTiles * kPfM));
    prefill_attn_kernel<T, D, KH, BIASED, PAGED, SPLIT, EXACT><<<grid, kPfThreads<SPLIT>, smem, stream>>>(mq, mk, mv, pp);
    note_launch();
    return check_launch("prefill_attn_kernel");
}

template <typename T, int D>
bool launch_prefill(const CUtensorMap &mq, const CUtensorMap &mk, const CUtensorMap &mv, const MhaParams &p,
                    cudaStream_t stream) {
    return p.dist_bias && p.dist_rows > 0 ? launch_prefill_b<T, D, D / 64, true>(mq, mk, mv, p, stream) : launch_prefill_b<T, D, D / 64, false>(mq, mk, mv, p, stream);
}

// A paged step whose keys and values are gathered first, so that the kernel for contiguous ones serves it, with the same bits: 1 = launched, 0 = not taken, -1 = error.
// A tile of keys that TMA copies and one thread a row works on is faster than one that three warps copy and two threads a row work on; the gather reads and writes every key
// of every sequence once.  So it is taken where what the tiles save is sure to pay for it (gather_pays).  Heads of 64 gain nothing (123 / 123, 99 / 102).
constexpr int64_t kPfGatherBytes = 256ll << 20;   // of scratch at most; longer steps stay with the pages
constexpr int kPfGatherQ = 256, kPfGatherK = 2048;

// Whether the gather pays for itself however the step's rows lie on its sequences: the host knows their number, their sum (rows, or, unknown, 0: one portion is sure) and the longest
// portion and sequence.  Saved, us, fitted to 200 steps: 0.38 a tile of keys and wave of CTAs where they fill the SMs, 0.30 a tile of the longest CTA; the gather 4 and its bytes at
// 8 TB/s.  The least that m portions of a mean length can save: they are new prompts, or all lie behind as many keys as there can be, and the other sequences' keys are gathered for
// one row each.
// Pages / rows, us, of steps taken: 32 heads on 8: 2048, 1500 and 531 tokens behind 0, 1003 and 37 160.8 / 154.6, 2048, 2030 and 1 behind 0, 0 and 2502 168 / 163, 4096 205 / 190, 8192 681 / 615,
// 1024 behind 8000 211 / 206, 256 behind 3000 88 / 85; 8 on 1: 512 behind 4000 111 / 103, 3000 78 / 78; 16 on 16: 8192 357 / 339.
// Of steps left: 300 tokens beside seven decoded behind up to 4000 keys 168 / 179 and (8 on 1) 84 / 87, four portions of 256 behind 4000 117 / 128, 256 beside fifteen decoded behind 4095
// 317 / 339; 16 on 16: 1024 behind 1100 62 / 67, eight of 256 behind 2000 74 / 114.
bool gather_pays(const MhaParams &p, int sms) {
    const double longest_q = p.rows_q > 0 ? static_cast<double>(std::min<int64_t>(p.rows_q, p.seqlen_q)) : p.seqlen_q;
    const double longest_k = std::max<double>(p.seqlen_k, longest_q), rows = p.rows_q > 0 ? static_cast<double>(p.rows_q) : longest_q;
    auto pays = [&](double m, double q, double c, double keys) {
        const double blocks = std::max(1.0, q / (kQTiles * kPfM));
        const double saved = std::max(0.30 * (q + c) / kPfN, 0.38 * m * p.h * (blocks * (blocks + 1.0) + blocks * c / kPfN) / sms);
        return saved >= 4.0 + keys * p.h_k * p.d * 8.0 / 8e6;
    };
    if (p.b == 1) return pays(1.0, longest_q, longest_k - longest_q, longest_k);
    const int most = p.rows_q > 0 ? p.b : 1;
    for (int m = std::max(1, static_cast<int>(std::min<double>(p.b, std::ceil(rows / longest_q)))); m <= most; ++m) {
        const double q = std::min(longest_q, rows / m), behind = std::max(0.0, longest_k - q);
        for (const double c : {0.0, behind})
            if (!pays(m, q, c, rows + m * c + (p.b - m) * longest_k)) return false;
    }
    return true;
}

int try_launch_gathered(const MhaParams &p, bool is_bf16, const CUtensorMap &mq, cudaStream_t stream) {
    // whole tiles of rows for whatever a block table can name: a sequence may be longer than the caller's bound, as it may on the pages
    const int64_t row = static_cast<int64_t>(p.h_k) * p.d, named = std::max<int64_t>(p.seqlen_k, p.bt_bs * p.page), pitch = (named + kPfN - 1) / kPfN * kPfN;
    const int64_t bytes = static_cast<int64_t>(p.b) * pitch * row * 2;
    if (p.d != 128 || p.seqlen_q < kPfGatherQ || p.seqlen_k < kPfGatherK || named > (1 << 24) || 2 * bytes > kPfGatherBytes || !gather_pays(p, current_device_info().sm_count)) return 0;
    // A graph may be replayed on any stream, where the scratch of the stream that it was captured on is not its own.
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &capturing) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    if (capturing != cudaStreamCaptureStatusNone) return 0;
    // The copy and the kernel that reads it are enqueued together: another thread may use this stream and its scratch.
    static std::mutex together;
    std::lock_guard<std::mutex> lock(together);
    unsigned char *space = static_cast<unsigned char *>(try_workspace(stream, static_cast<size_t>(2 * bytes), kWorkspacePrefillKeys));
    if (!space) return 0;
    MhaParams pp = p;
    pp.block_table = nullptr;
    pp.k = space, pp.v = space + bytes;
    pp.k_hs = pp.v_hs = p.d, pp.k_rs = pp.v_rs = row, pp.k_bs = pp.v_bs = pitch * row;
    pp.k_batched = static_cast<int>(pitch);
    CUtensorMap mk, mv;
    if (!make_attn_map(&mk, pp.k, p.d, p.h_k, pitch, p.b, pp.k_hs, pp.k_rs, pp.k_bs, is_bf16)) return -1;
    if (!make_attn_map(&mv, pp.v, p.d, p.h_k, pitch, p.b, pp.v_hs, pp.v_rs, pp.v_bs, is_bf16)) return -1;
    const dim3 grid(static_cast<unsigned>((pitch + kPfGatherWarps - 1) / kPfGatherWarps), static_cast<unsigned>(p.b));
    const cudaError_t e = launch_ex(paged_rows_kernel, grid, dim3(32 * kPfGatherWarps), 0, stream, p, reinterpret_cast<uint4 *>(space), reinterpret_cast<uint4 *>(space + bytes), static_cast<int>(pitch));
    note_launch();
    if (e != cudaSuccess) {
        set_status(static_cast<int>(e), "paged_rows_kernel: %s", cudaGetErrorString(e));
        return -1;
    }
    const bool done = is_bf16 ? launch_prefill_b<__nv_bfloat16, 128, 2, false, false, true>(mq, mk, mv, pp, stream)
                              : launch_prefill_b<__half, 128, 2, false, false, true>(mq, mk, mv, pp, stream);
    return done ? 1 : -1;
}

}  // namespace

// 1 = launched, 0 = outside this kernel's envelope (caller uses the general tile kernel), -1 = error.
int try_launch_prefill_tc(const MhaParams &p, bool is_bf16, cudaStream_t stream) {
    if (p.alibi) return 0;
    if (p.block_table && (p.page <= 0 || p.d_k > 0 || p.gate || p.dist_bias || p.v_share > 1)) return 0;
    if (p.d != 64 && p.d != 128) return 0;
    if (p.seqlen_q < 32) return 0;  // a 128-row tile would be mostly padding
    if (!(p.scale_log2 > 0.f)) return 0;
    if (p.h_k <= 0 || p.h % p.h_k != 0 || p.h > 65535 || p.b > 65535 || p.seqlen_q > 65535 * kQTiles * kPfM) return 0;
    if (p.d_k > 0 && (p.d_k % 8 || p.d_k > p.d + 64 || (p.d_k > p.d && (!is_bf16 || p.dist_bias)))) return 0;
    if (p.gate && (!p.cu_q || p.gate_rs % 8 || (reinterpret_cast<uintptr_t>(p.gate) & 15))) return 0;
    const DeviceInfo &di = current_device_info();
    if (di.cc_major != 10) return 0;
    // Pages: where all sequences are short (by the longest portion and the longest sequence), the tile kernel takes the step: from two pairs of a
    // sequence and a head per SM on by short_for_prefill(), below that up to 64 keys (4 sequences of 8 heads of 64 over 32, 64, 96 keys, tiles /
    // prefill kernel: 5 / 7, 6 / 8, 8 / 8 us).  Heads of 64 with six pairs per SM and more: each kernel takes its sequences of a mixed step.  A second
    // launch costs 10 to 18 us there: one portion of 64 tokens beside 63 decoded ones over 64, 264 and 564 keys, 32 heads, tiles alone / prefill kernel alone:
    // 30 / 90, 82 / 123, 160 / 171 us.  With heads of 128 it gives back less than that (41 / 107, 152 / 145, 302 / 210).
    const int64_t pairs = p.block_table ? static_cast<int64_t>(p.b) * p.h : 0;
    if (p.block_table && (pairs >= 2 * di.sm_count ? short_for_prefill(p.d, p.seqlen_q, p.seqlen_k) : p.seqlen_k <= 64)) return 0;
    // TMA: 16-byte aligned bases and strides (run_mha already checked pointers and strides % 8)
    const bool q_varlen = p.cu_q != nullptr;
    const bool k_varlen = p.cu_k != nullptr && p.k_cumulative;
    const int64_t huge_rows = 1ll << 26;
    auto stride_ok = [](int64_t s) { return s > 0 && s * 2 < (1ll << 40); };
    if (!stride_ok(p.q_rs) || !stride_ok(p.k_rs) || !stride_ok(p.v_rs) || !stride_ok(p.q_hs) ||
        !stride_ok(p.k_hs) || !stride_ok(p.v_hs))
        return 0;
    if (!q_varlen && p.b > 1 && !stride_ok(p.q_bs)) return 0;
    if (!p.block_table && !k_varlen && p.b > 1 && (!stride_ok(p.k_bs) || !stride_ok(p.v_bs))) return 0;

    CUtensorMap mq, mk, mv;
    const int64_t q_rows = q_varlen ? huge_rows : p.seqlen_q, q_b = q_varlen ? 1 : p.b;
    const int64_t k_rows = k_varlen ? huge_rows : p.seqlen_k, k_b = k_varlen ? 1 : p.b;
    const int64_t q_bs = (q_varlen || p.b == 1 || p.q_bs == 0) ? p.q_rs : p.q_bs;
    const int64_t k_bs = (k_varlen || p.b == 1 || p.k_bs == 0) ? p.k_rs : p.k_bs;
    const int64_t v_bs = (k_varlen || p.b == 1 || p.v_bs == 0) ? p.v_rs : p.v_bs;
    const int d_k = p.d_k > 0 ? p.d_k : p.d;
    if (!make_attn_map(&mq, p.q, d_k, p.h, q_rows, q_b, p.q_hs, p.q_rs, q_bs, is_bf16)) return -1;
    if (p.block_table) {
        MhaParams pp = p;
        pp.split_short = p.d == 64 && p.b > 1 && pairs >= 6 * di.sm_count ? 1 : 0;
        bool done;
        const int gathered = try_launch_gathered(pp, is_bf16, mq, stream);
        if (gathered != 0) return gathered;
        if (is_bf16) done = p.d == 128 ? launch_prefill_b<__nv_bfloat16, 128, 2, false, true>(mq, mq, mq, pp, stream)
                                       : launch_prefill_b<__nv_bfloat16, 64, 1, false, true>(mq, mq, mq, pp, stream);
        else done = p.d == 128 ? launch_prefill_b<__half, 128, 2, false, true>(mq, mq, mq, pp, stream)
                               : launch_prefill_b<__half, 64, 1, false, true>(mq, mq, mq, pp, stream);
        if (done && pp.split_short) done = launch_attention_tile(pp, is_bf16, stream);
        return done ? 1 : -1;
    }
    if (!make_attn_map(&mk, p.k, d_k, p.h_k, k_rows, k_b, p.k_hs, p.k_rs, k_bs, is_bf16)) return -1;
    if (!make_attn_map(&mv, p.v, p.d, p.v_share > 1 ? p.h_k / p.v_share : p.h_k, k_rows, k_b, p.v_hs, p.v_rs, v_bs, is_bf16)) return -1;
    bool ok;
    if (p.d == 128 && d_k <= 64 && is_bf16 && !p.dist_bias)   // shorter query / key heads: one 64-column piece
        ok = launch_prefill_b<__nv_bfloat16, 128, 1, false>(mq, mk, mv, p, stream);
    else if ((d_k + 63) / 64 > p.d / 64)   // longer query / key heads than value heads
        ok = p.d == 128 ? launch_prefill_b<__nv_bfloat16, 128, 3, false>(mq, mk, mv, p, stream)
                        : launch_prefill_b<__nv_bfloat16, 64, 2, false>(mq, mk, mv, p, stream);
    else if (is_bf16) ok = p.d == 128 ? launch_prefill<__nv_bfloat16, 128>(mq, mk, mv, p, stream)
                                 : launch_prefill<__nv_bfloat16, 64>(mq, mk, mv, p, stream);
    else ok = p.d == 128 ? launch_prefill<__half, 128>(mq, mk, mv, p, stream)
                         : launch_prefill<__half, 64>(mq, mk, mv, p, stream);
    return ok ? 1 : -1;
}

}  // namespace atoma

extern "C" int atoma_prefill_timeouts(void) {
    unsigned int n = 0;
    if (cudaMemcpyFromSymbol(&n, atoma::g_prefill_late, sizeof(n)) != cudaSuccess) return -1;
    return static_cast<int>(n);
}
