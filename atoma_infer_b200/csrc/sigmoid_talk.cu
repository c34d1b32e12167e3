// Sigmoid attention whose heads talk, for prompt portions (include/atoma_hybrid.h, atoma_sigmoid_attention_paged with a talk matrix): bfloat16 caches, 16 or
// 32 heads of up to 64 entries.
//
// Every head's weight of a (query, key) pair must exist before any head can apply it: per tile of 16 queries x 32 keys,
//   1. scores and weights: a warp takes two heads (mma.sync on the staged keys; cap, distance, bias and sigmoid in float32),
//   2. the talk matrix: mixed[h, pair] = sum_g talk[h, g] a[g, pair], a product of its own over the heads,
//   3. values: a warp applies its two heads' mixed weights (bfloat16, as before).
// What bounded the mix on CUDA cores was shared memory (32 float32 weights read per pair and head; 4000 warp instructions per tile and
// warp), so it runs on the tensor cores too, at float32's precision: weights and talk are each split into three bfloat16 pieces of 8 bits, which
// hold all of a float32's 24 and its whole range, and the six products of pieces down to 2^-16 of a term are summed in float32 (what is dropped is
// 2^-25 of a term).  mma.sync and not tcgen05: the products per tile are 16 rows or one head-square deep.
// One CTA holds all heads (64 accumulator registers per thread for two heads), so there is no cluster exchange, and the keys are cut into segments,
// whose float32 sums simply add (no softmax): 128 row blocks of one prompt over 74 CTA pairs left the SMs idle half of the time.  A
// segment is 512 keys from a multiple of 512 on whatever the step looks like, so a position's sums depend on its keys alone.  A CTA takes one
// segment, or, in steps whose row blocks fill the SMs without, all of its rows' segments one after the other; the sums between take at most 256 MiB
// (kStScratch), and longer steps go in runs of tokens.  Keys of the next tile are copied under the mix, values under the scores.
// A tile of 2048 tokens, 32 heads of 64 on 8, takes 14000 cycles: scores and weights 6000 (four results of the special-function unit per weight are 4100 of them),
// the mix 5000 (3100 of the tensor pipe), values 2000.  With 27000: every copy waited for its own block-table entry (5000), a branch per weight kept
// their chains from overlapping, quotients and exponentials took denormal numbers into account, and registers spilled.
// 2048 tokens, 32 heads of 64 on 8: 1218 us on the CUDA-core mix (hybrid_attention.cu), 507 with those, 283 here; 2000 tokens of 16 heads 328 and 169.  Prompts of up to
// some 40 tokens are slower than on CUDA cores, since all heads wait for each other in one CTA (33 tokens of 16 and 32 heads 15.9 and 24.2 us, there 14.3 and 19.1;
// 64 tokens 16.4 and 26.6, there 22.6 and 32.8); they stay here, so that a position's bits do not follow the step.
#include "common.cuh"
#include "hybrid_common.cuh"

#include "atoma_hybrid.h"

#include <algorithm>
#include <type_traits>

namespace atoma {
namespace {

using namespace hybrid;

constexpr int kStRows = 16, kStKeys = 32, kStSegKeys = 512, kStPieces = 3;
constexpr int64_t kStScratch = 256ll << 20;

// sigmoid(cap tanh(s / cap) - slope dist + bias), tanh(y) = 1 - 2 / (1 + e^2y).  The unit's estimates of 2^x and of the reciprocal are within 2 and 1 units of the last
// place.  The logit keeps its own unit until it is whole: slopes in units of log 2 would carry their rounding times the distance (rms 1.4e-7 off where this is 4e-8).
template <bool CAP>
__device__ __forceinline__ float st_weight(float dot, float scale, float in, float cap, float slope, float dist, float head_bias) {
    auto ex2 = [](float x) {
        float y;
        asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
        return y;
    };
    auto rcp = [](float x) {
        float y;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
        return y;
    };
    const float s = CAP ? fmaf(-2.f, rcp(1.f + ex2(dot * in)), 1.f) * cap : dot * scale;
    return rcp(1.f + ex2(-1.4426950408889634f * (fmaf(-slope, dist, s) + head_bias)));
}

template <int HT>   // heads = 16 HT
struct StLayout {
    static constexpr int H = 16 * HT, kPair = 4 * H + 32, kRow = kStKeys * kPair + 16;   // bytes of a pair's float32 weights, of a query row's
    static constexpr int kMixRow = 2 * kStKeys + 16, kMixHead = kStRows * kMixRow + 16;
    static constexpr int kTalkRow = 2 * H + 16, kTalk = H * kTalkRow;                    // one piece of the talk matrix
    static constexpr int w_off = 0, m_off = kStRows * kRow, t_off = m_off + H * kMixHead, kv_off = t_off + kStPieces * kTalk;
    __host__ __device__ static size_t total(int G, int D, int DV) { return kv_off + static_cast<size_t>(G) * kStKeys * (D + 8 + DV + 8) * 2; }
};

// a float32's three bfloat16 pieces, the largest first
__device__ __forceinline__ void st_split(float x, float (&piece)[kStPieces]) {
#pragma unroll
    for (int i = 0; i < kStPieces; ++i) {
        piece[i] = __bfloat162float(__float2bfloat16_rn(x));
        x -= piece[i];
    }
}

// Row blocks of every sequence that start on the step's tokens lo .. hi - 1.  slots: segments that have a place of their own in `partial` for every token
// (blockIdx.z: which segment this CTA takes; sigmoid_talk_sum_kernel adds them), or 1: this CTA takes them all and keeps the running sum there.  Both add the
// segments in order, so they give the same bits.  No scratch: one chain over all keys.
template <int HT>
__global__ void __launch_bounds__(256 * HT, 1) sigmoid_talk_kernel(const atoma_sigmoid_attn_args a, int lo, int hi, int slots, float *__restrict__ partial) {
    using L = StLayout<HT>;
    constexpr int H = L::H, NW = 8 * HT, NT = 256 * HT;
    extern __shared__ __align__(16) unsigned char sm[];
    pdl_launch_dependents();
    pdl_wait();
    const int G = static_cast<int>(a.G), D = static_cast<int>(a.dim), DV = static_cast<int>(a.vdim), bs = static_cast<int>(a.block_size);
    const int b = blockIdx.y, seg = blockIdx.z;
    const int t_begin = a.query_start[b], n_q = a.query_start[b + 1] - t_begin;
    const int first = max(0, lo - t_begin + kStRows - 1) / kStRows, last = (min(n_q, hi - t_begin) + kStRows - 1) / kStRows - 1;   // this run's row blocks
    const int blk = last - static_cast<int>(blockIdx.x);   // the rows with the most keys first
    if (n_q <= 0 || blk < first) return;
    const int r0 = blk * kStRows, rows = min(kStRows, n_q - r0), tok0 = t_begin + r0;
    const int ctx = static_cast<int>(a.positions[t_begin]), p0 = ctx + r0, total = ctx + n_q;
    const int all_end = p0 + rows, j_begin = seg * kStSegKeys, j_end = seg == slots - 1 ? all_end : min(all_end, j_begin + kStSegKeys);
    if (j_begin >= all_end) return;
    const int32_t *bt = a.block_tables + static_cast<int64_t>(b) * a.max_blocks;
    unsigned char *weights = sm + L::w_off, *mix = sm + L::m_off, *talk = sm + L::t_off;
    __nv_bfloat16 *Ks = reinterpret_cast<__nv_bfloat16 *>(sm + L::kv_off), *Vs = Ks + G * kStKeys * (D + 8);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, t4 = lane & 3, rq = lane >> 2;
    const __nv_bfloat16 *kc = static_cast<const __nv_bfloat16 *>(a.k_cache), *vc = static_cast<const __nv_bfloat16 *>(a.v_cache);
    // Cache rows of a tile's keys (-1: behind the sequence's end, zero-filled), looked up one tile ahead by one warp: a copy that waits for its own table
    // entry costs a round trip to memory.
    __shared__ int32_t slot_s[2][kStKeys];
    const int bs_shift = (bs & (bs - 1)) == 0 ? __ffs(bs) - 1 : -1;
    auto look_up = [&](int j) {
        const int pg = bs_shift >= 0 ? j >> bs_shift : j / bs;
        return j < total ? bt[pg] * bs + (j - pg * bs) : -1;
    };
    static_assert(kStKeys == 32, "a lane per key");
    if (warp == 0) slot_s[0][lane] = look_up(j_begin + lane);
    __syncthreads();
    // a thread's piece of a row is the same for all its keys when the CTA takes whole rows at a time
    auto stage = [&](const __nv_bfloat16 *cache, __nv_bfloat16 *dst, int n, const int32_t *slots) {
        const int pieces = G * n / 8;
        auto put = [&](int jj, int e, int g) {
            const int slot = slots[jj];
            cp_async_16(smem_u32(dst + (g * kStKeys + jj) * (n + 8) + e * 8 - g * n), cache + static_cast<int64_t>(max(slot, 0)) * G * n + e * 8, slot >= 0 ? 16 : 0);
        };
        if (NT % pieces == 0) {
            const int e = tid % pieces, g = e * 8 / n;
            for (int jj = tid / pieces; jj < kStKeys; jj += NT / pieces) put(jj, e, g);
        } else {
            for (int i = tid; i < kStKeys * pieces; i += NT) {
                const int jj = i / pieces, e = i - jj * pieces;
                put(jj, e, e * 8 / n);
            }
        }
        cp_async_commit();
    };
    stage(kc, Ks, D, slot_s[0]);
    // ---- the talk matrix in three pieces ----
    for (int i = tid; i < H * H; i += NT) {
        float piece[kStPieces];
        st_split(a.talk[i], piece);
#pragma unroll
        for (int k = 0; k < kStPieces; ++k)
            *reinterpret_cast<__nv_bfloat16 *>(talk + k * L::kTalk + i / H * L::kTalkRow + i % H * 2) = __float2bfloat16_rn(piece[k]);
    }
    // ---- this warp's heads: query fragments, constants ----
    const int h0 = 2 * warp, rep = H / G;
    uint32_t qf[32];   // [head][16 of its entries][fragment]
    float slope[2], hb[2];
#pragma unroll
    for (int x = 0; x < 2; ++x) {
        slope[x] = a.slopes ? a.slopes[h0 + x] : 0.f;
        hb[x] = a.head_bias[h0 + x];
        const __nv_bfloat16 *q = static_cast<const __nv_bfloat16 *>(a.q) + static_cast<int64_t>(tok0) * H * D + (h0 + x) * D;
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int row = rq + (e & 1) * 8, col = kk * 16 + 2 * t4 + (e >> 1) * 8;
                qf[x * 16 + kk * 4 + e] = kk * 16 < D && row < rows ? *reinterpret_cast<const uint32_t *>(q + static_cast<int64_t>(row) * H * D + col) : 0u;
            }
    }
    // Of 32 heads, a thread's 64 sums, 32 queries and the mix do not fit its 128 registers (spilled, 81 KB a tile passed through an L1 of 28 KB: 386 us, 308 without):
    // the queries and, between tiles, the sums lie in tensor memory, from where a phase takes them in one or two loads.
    __shared__ uint32_t tmem_base_s;
    uint32_t tmem_q = 0, tmem_o = 0;
    if constexpr (HT == 2) {
        if (warp == 0) tmem_alloc(&tmem_base_s, 512);
        tc_fence_before_sync();
        __syncthreads();
        tc_fence_after_sync();
        tmem_q = tmem_base_s + (static_cast<uint32_t>((warp & 3) * 32) << 16) + (warp >> 2) * 32;
        tmem_o = tmem_base_s + (static_cast<uint32_t>((warp & 3) * 32) << 16) + 128 + (warp >> 2) * 64;
        tmem_st_32x32b_x32(tmem_q, qf);
        tmem_st_wait();
    }
    float o[2][8][4];
    auto clear = [&] {
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int i = 0; i < 8; ++i) o[x][i][0] = o[x][i][1] = o[x][i][2] = o[x][i][3] = 0.f;
    };
    clear();
    bool fresh = true;   // nothing has been summed since the start, or since a segment went out
    const float in = a.softcap > 0.f ? a.scale * 2.8853900817779268f / a.softcap : 0.f;   // e^(2 s / cap) = 2^(in dot)
    // the sums of a segment, out of the accumulators: into its place, onto the running sum, or, where no other segment follows or precedes, out
    bool more = false;   // a running sum waits in this token's place
    auto put = [&](bool last) {
        const bool out = last && (slots == 1 || all_end <= kStSegKeys);
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int nt = 0; nt < 8; ++nt) {
                if (nt * 8 >= DV) continue;
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int row = rq + 8 * e, col = (h0 + x) * DV + nt * 8 + 2 * t4;
                    if (row >= rows) continue;
                    float2 s = make_float2(o[x][nt][2 * e], o[x][nt][2 * e + 1]);
                    float2 *place = reinterpret_cast<float2 *>(partial + (static_cast<int64_t>(tok0 + row - lo) * slots + seg) * H * DV + col);
                    if (more) s = make_float2(place->x + s.x, place->y + s.y);
                    if (out) *reinterpret_cast<uint32_t *>(static_cast<__nv_bfloat16 *>(a.out) + static_cast<int64_t>(tok0 + row) * H * DV + col) = pack2<__nv_bfloat16>(s.x, s.y);
                    else *place = s;
                }
            }
    };

    for (int j0 = j_begin; j0 < j_end; j0 += kStKeys) {
        cp_async_wait_all();
        __syncthreads();   // the keys are there; everyone is done with the last tile's values and mixed weights
        const int cur = (j0 - j_begin) / kStKeys & 1;
        stage(vc, Vs, DV, slot_s[cur]);
        int next_slot = 0;
        if (warp == 0) next_slot = look_up(j0 + kStKeys + lane);
        // ---- 1. scores and weights of two heads; both heads' weights of a pair go out together ----
        if constexpr (HT == 2) {
            tmem_ld_32x32b_x32(tmem_q, qf);
            tmem_ld_wait();
        }
        // 16 keys at a time: the accumulators of the values and the queries leave few registers
#pragma unroll
        for (int np = 0; np < 2; ++np) {
            float w0[2][4];
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                float s[2][4];
#pragma unroll
                for (int i = 0; i < 2; ++i) s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.f;
                const __nv_bfloat16 *kb = Ks + ((h0 + x) / rep * kStKeys + (lane >> 4) * 8 + (lane & 7)) * (D + 8) + ((lane >> 3) & 1) * 8;
#pragma unroll
                for (int kk = 0; kk < 4; ++kk)
                    if (kk * 16 < D) {
                        uint32_t r[4];
                        ldmatrix_x4(r, smem_u32(kb + np * 16 * (D + 8) + kk * 16));
                        const uint32_t(&qk)[4] = *reinterpret_cast<const uint32_t(*)[4]>(qf + x * 16 + kk * 4);
                        Mma16816<__nv_bfloat16>::run(s[0], qk, r[0], r[1]);
                        Mma16816<__nv_bfloat16>::run(s[1], qk, r[2], r[3]);
                    }
                // weights of hidden pairs are formed too and dropped: without a branch per weight their chains of exponentials and quotients overlap
                const float base = static_cast<float>(p0 + rq - j0 - 2 * t4);
                auto weigh = [&](auto with_cap) {
#pragma unroll
                    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            s[nt][e] = st_weight<decltype(with_cap)::value>(s[nt][e], a.scale, in, a.softcap, slope[x],
                                                                            base - static_cast<float>((2 * np + nt) * 8 + (e & 1) - (e >> 1) * 8), hb[x]);
                };
                if (a.softcap > 0.f) weigh(std::true_type{});
                else weigh(std::false_type{});
#pragma unroll
                for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int row = rq + (e >> 1) * 8, key = (2 * np + nt) * 8 + 2 * t4 + (e & 1);
                        const float w = row < rows && p0 + row >= j0 + key ? s[nt][e] : 0.f;
                        if (x == 0) w0[nt][e] = w;
                        else *reinterpret_cast<float2 *>(weights + row * L::kRow + key * L::kPair + h0 * 4) = make_float2(w0[nt][e], w);
                    }
            }
        }
        if (warp == 0) slot_s[cur ^ 1][lane] = next_slot;
        __syncthreads();   // all heads' weights are there, and the keys are done with
        if (j0 + kStKeys < j_end) stage(kc, Ks, D, slot_s[cur ^ 1]);
        else cp_async_commit();   // an empty group: the values' is always the one before the last
        // ---- 2. the heads talk: a warp takes whole query rows, eight (32 heads; thirty-two: 286 us for 286) or thirty-two (16 heads; eight: 179 us for 169) keys at a time ----
        constexpr int kN = HT == 2 ? 1 : 4;
        for (int row = warp; row < kStRows; row += NW)
#pragma unroll 1
            for (int n2 = 0; n2 < kStKeys / 8; n2 += kN) {
                uint32_t wb[kN][kStPieces][HT][2];
#pragma unroll
                for (int i = 0; i < kN; ++i)
#pragma unroll
                    for (int kk = 0; kk < HT; ++kk)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const float2 w = *reinterpret_cast<const float2 *>(weights + row * L::kRow + ((n2 + i) * 8 + rq) * L::kPair + (kk * 16 + 8 * e + 2 * t4) * 4);
                            float x = w.x, y = w.y;   // two values' pieces at a time
#pragma unroll
                            for (int k = 0; k < kStPieces; ++k) {
                                const uint32_t piece = pack2<__nv_bfloat16>(x, y);
                                wb[i][k][kk][e] = piece;
                                x -= __uint_as_float(piece << 16);
                                y -= __uint_as_float(piece & 0xffff0000u);
                            }
                        }
#pragma unroll
                for (int mt = 0; mt < HT; ++mt) {
                    // products of one order in a sum of their own, a shorter chain; the smallest are added first
                    float co[kN][kStPieces][4];
#pragma unroll
                    for (int i = 0; i < kN; ++i)
#pragma unroll
                        for (int order = 0; order < kStPieces; ++order)
#pragma unroll
                            for (int e = 0; e < 4; ++e) co[i][order][e] = 0.f;
#pragma unroll
                    for (int k = 0; k < kStPieces; ++k) {
                        uint32_t ta[HT][4];
#pragma unroll
                        for (int kk = 0; kk < HT; ++kk)
                            ldmatrix_x4(ta[kk], smem_u32(talk + k * L::kTalk + (mt * 16 + (lane & 15)) * L::kTalkRow + (kk * 16 + (lane >> 4) * 8) * 2));
#pragma unroll
                        for (int i = 0; i < kN; ++i)
#pragma unroll
                            for (int kk = 0; kk < HT; ++kk)
#pragma unroll
                                for (int order = k; order < kStPieces; ++order) Mma16816<__nv_bfloat16>::run(co[i][order], ta[kk], wb[i][order - k][kk][0], wb[i][order - k][kk][1]);
                    }
#pragma unroll
                    for (int i = 0; i < kN; ++i) {
                        float c[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) c[e] = co[i][0][e] + (co[i][1][e] + co[i][2][e]);
                        unsigned char *m = mix + (mt * 16 + rq) * L::kMixHead + row * L::kMixRow + ((n2 + i) * 8 + 2 * t4) * 2;
                        *reinterpret_cast<uint32_t *>(m) = pack2<__nv_bfloat16>(c[0], c[1]);
                        *reinterpret_cast<uint32_t *>(m + 8 * L::kMixHead) = pack2<__nv_bfloat16>(c[2], c[3]);
                    }
                }
            }
        asm volatile("cp.async.wait_group 1;" ::: "memory");   // the values
        __syncthreads();
        // ---- 3. values ----
        if constexpr (HT == 2) {
            if (fresh) {
                clear();
            } else {
                uint32_t *r = reinterpret_cast<uint32_t *>(&o[0][0][0]);
                tmem_st_wait();
                tmem_ld_32x32b_x32(tmem_o, r);
                tmem_ld_32x32b_x32(tmem_o + 32, r + 32);
                tmem_ld_wait();
            }
        }
        fresh = false;
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            const __nv_bfloat16 *vb = Vs + ((h0 + x) / rep * kStKeys + ((lane >> 3) & 1) * 8 + (lane & 7)) * (DV + 8) + (lane >> 4) * 8;
#pragma unroll
            for (int kk = 0; kk < 2; ++kk) {
                uint32_t af[4];
                ldmatrix_x4(af, smem_u32(mix + (h0 + x) * L::kMixHead + (lane & 15) * L::kMixRow + (kk * 16 + (lane >> 4) * 8) * 2));
#pragma unroll
                for (int n2 = 0; n2 < 4; ++n2)
                    if (n2 * 16 < DV) {
                        uint32_t r[4];
                        ldmatrix_x4_trans(r, smem_u32(vb + kk * 16 * (DV + 8) + n2 * 16));
                        Mma16816<__nv_bfloat16>::run(o[x][2 * n2], af, r[0], r[1]);
                        Mma16816<__nv_bfloat16>::run(o[x][2 * n2 + 1], af, r[2], r[3]);
                    }
            }
        }
        if (slots == 1 && partial && j0 + kStKeys < j_end && (j0 + kStKeys) % kStSegKeys == 0) {   // a segment ends here
            put(false);
            more = true;
            fresh = true;
            clear();
        } else if constexpr (HT == 2) {
            const uint32_t *r = reinterpret_cast<const uint32_t *>(&o[0][0][0]);
            tmem_st_32x32b_x32(tmem_o, r);
            tmem_st_32x32b_x32(tmem_o + 32, r + 32);
        }
    }
    cp_async_wait_all();
    put(true);
    if constexpr (HT == 2) {
        tmem_st_wait();
        tc_fence_before_sync();
        __syncthreads();
        tc_fence_after_sync();
        if (warp == 0) tmem_dealloc(tmem_base_s, 512);
    }
}

// A token's segments, in order; tokens of one segment are out already.
__global__ void __launch_bounds__(256) sigmoid_talk_sum_kernel(const atoma_sigmoid_attn_args a, const float *__restrict__ partial, int lo, int hi, int segs) {
    pdl_launch_dependents();
    pdl_wait();
    const int64_t t = lo + static_cast<int64_t>(blockIdx.x);
    const int b = a.token_seq[t], t_begin = a.query_start[b], n_q = a.query_start[b + 1] - t_begin;
    const int r0 = static_cast<int>(t - t_begin) / kStRows * kStRows, end = static_cast<int>(a.positions[t_begin]) + min(r0 + kStRows, n_q);
    const int n = min(segs, (end + kStSegKeys - 1) / kStSegKeys), row = static_cast<int>(a.H * a.vdim);
    if (n < 2 || t_begin + r0 < lo || t_begin + r0 >= hi) return;
    const float *p = partial + (t - lo) * segs * row;
    for (int i = threadIdx.x * 4; i < row; i += 1024) {
        float4 s = *reinterpret_cast<const float4 *>(p + i);
        for (int k = 1; k < n; ++k) {
            const float4 v = *reinterpret_cast<const float4 *>(p + k * row + i);
            s.x += v.x, s.y += v.y, s.z += v.z, s.w += v.w;
        }
        *reinterpret_cast<uint2 *>(static_cast<__nv_bfloat16 *>(a.out) + t * row + i) = make_uint2(pack2<__nv_bfloat16>(s.x, s.y), pack2<__nv_bfloat16>(s.z, s.w));
    }
}

}  // namespace

// Prompt portions (decode-only batches split their keys in hybrid_attention.cu) of 16 or 32 talking heads whose staged tiles fit shared memory.
bool hyb_sigmoid_talk_ok(const atoma_sigmoid_attn_args &a) {
    auto al = [](const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    if (a.dtype != ATOMA_DTYPE_BF16 || !a.talk || a.max_query_len < 2 || !a.query_start || (a.H != 16 && a.H != 32) || a.dim % 16 || a.vdim % 16 || a.dim > 64 || a.vdim > 64 ||
        !al(a.q) || !al(a.k_cache) || !al(a.v_cache) || !al(a.out) || current_device_info().cc_major != 10 || a.B > 65535)
        return false;
    const int G = static_cast<int>(a.G), D = static_cast<int>(a.dim), DV = static_cast<int>(a.vdim);
    return (a.H == 16 ? StLayout<1>::total(G, D, DV) : StLayout<2>::total(G, D, DV)) <= 225 * 1024;
}

bool hyb_sigmoid_talk(const atoma_sigmoid_attn_args &a, cudaStream_t stream) {
    const int64_t longest = a.max_seq_len > 0 ? a.max_seq_len : a.max_blocks * a.block_size;
    const int64_t segs = std::min<int64_t>(65535, (longest + kStSegKeys - 1) / kStSegKeys), blocks = (a.T + kStRows - 1) / kStRows;
    const int64_t place = a.H * a.vdim * 4;   // bytes of a token's sums
    int64_t slots = 1, run = a.T;
    float *partial = nullptr;
    if (segs > 1) {
        // a segment per CTA unless the row blocks are four per SM and more, or two and the segments' sums do not fit at once
        auto fits = [&](int64_t n) { return std::max<int64_t>(kStRows, kStScratch / (n * place) / kStRows * kStRows); };
        const int64_t sms = current_device_info().sm_count;
        slots = blocks >= 4 * sms || (blocks >= 2 * sms && fits(segs) < a.T) ? 1 : segs;
        run = std::min(a.T, fits(slots));
        partial = static_cast<float *>(try_workspace(stream, static_cast<size_t>((run + kStRows) * slots * place), kWorkspaceHybridAttn));   // a run's last row block may end behind it
        if (!partial) slots = 1, run = a.T;   // no scratch: one chain needs none
    }
    const int G = static_cast<int>(a.G), D = static_cast<int>(a.dim), DV = static_cast<int>(a.vdim);
    auto kernel = a.H == 16 ? sigmoid_talk_kernel<1> : sigmoid_talk_kernel<2>;
    const size_t smem = a.H == 16 ? StLayout<1>::total(G, D, DV) : StLayout<2>::total(G, D, DV);
    const cudaError_t attr = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 225 * 1024);
    if (attr != cudaSuccess) return hybrid::launched(attr, "sigmoid_talk_kernel");
    for (int64_t lo = 0; lo < a.T; lo += run) {
        const int64_t hi = std::min(a.T, lo + run), rows = (std::min<int64_t>(hi - lo, a.max_query_len) + kStRows - 1) / kStRows + 1;
        const dim3 grid(static_cast<unsigned>(rows), static_cast<unsigned>(a.B), static_cast<unsigned>(slots));
        if (!hybrid::launched(launch_ex(kernel, grid, dim3(16 * static_cast<unsigned>(a.H)), smem, stream, a, static_cast<int>(lo), static_cast<int>(hi),
                                        static_cast<int>(slots), partial),
                              "sigmoid_talk_kernel"))
            return false;
        if (slots > 1 && !hybrid::launched(launch_ex(sigmoid_talk_sum_kernel, dim3(static_cast<unsigned>(std::min(a.T, hi + kStRows) - lo)), dim3(256), 0, stream, a,
                                                    static_cast<const float *>(partial), static_cast<int>(lo), static_cast<int>(hi), static_cast<int>(slots)),
                                          "sigmoid_talk_sum_kernel"))
            return false;
    }
    return true;
}

}  // namespace atoma
