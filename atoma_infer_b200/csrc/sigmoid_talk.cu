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
// 2^-25 of a term).
// One CTA holds all heads (64 accumulator registers per thread for two heads), so there is no cluster exchange, and the keys are cut into segments,
// whose float32 sums simply add (no softmax): 128 row blocks of one prompt over 74 CTA pairs left the SMs idle half of the time.  A
// segment is 512 keys (sigmoid_talk32_kernel: 256) from a multiple of that on whatever the step looks like, so a position's sums depend on its keys alone.  A CTA takes one
// segment (of the shorter ones two neighbours in steps of many), or, in steps whose row blocks fill the SMs without, all of its rows' segments one after the other; the sums between take
// at most 256 MiB (kStScratch), and longer steps go in runs of tokens.  Keys of the next tile are copied under the mix, values under the scores.
// 32 heads of 64 in pages of whole runs of eight keys go by sigmoid_talk32_kernel, all others by sigmoid_talk_kernel, whose figures these are.  A tile of 2048 tokens, 32 heads
// of 64 on 8, takes 14000 cycles: scores and weights 6000 (four results of the special-function unit per weight are 4100 of them),
// the mix 5000 (3100 of the tensor pipe), values 2000.  With 27000: every copy waited for its own block-table entry (5000), a branch per weight kept
// their chains from overlapping, quotients and exponentials took denormal numbers into account, and registers spilled.
// 2048 tokens, 32 heads of 64 on 8: 1218 us on the CUDA-core mix (hybrid_attention.cu), 507 with those, 283 now; 2000 tokens of 16 heads 328 and 169.  Prompts of up to
// some 40 tokens are slower than on CUDA cores, since all heads wait for each other in one CTA (33 tokens of 16 and 32 heads 15.9 and 24.2 us, there 14.3 and 19.1;
// 64 tokens 16.4 and 26.6, there 22.6 and 32.8); they stay, so that a position's bits do not follow the step.
#include "common.cuh"
#include "hybrid_common.cuh"

#include "atoma_hybrid.h"

#include <algorithm>
#include <type_traits>

namespace atoma {
namespace {

using namespace hybrid;

constexpr int kStRows = 16, kStKeys = 32, kStPieces = 3;
// Keys of a segment, of sigmoid_talk_kernel and of sigmoid_talk32_kernel.  Shorter ones put short prompts on more SMs and cost long ones more sums.  The first, 512 / 256: 16 heads,
// 2000 tokens 166 / 171 us; 32 heads of 32 and 48 on 16, 1000 and 4000 tokens 153 / 89, 1015 / 1143.  The second: 600 and 1000 tokens 117 / 66, 119 / 68, long ones faster than on the
// first all the same; 128 lose from 1000 tokens on.
constexpr int kStSegKeys = 512, kS3SegKeys = 256;
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

// The same for 32 heads, with the mix on tcgen05: a pair's weights of all heads are a row of 32, so that 128 pairs are the wide operand, in tensor memory, and the
// talk matrix's pieces the narrow one: 12 products of 128 x 32 x 16 stand for the six products of pieces, where mma.sync took 1536 at a quarter of the rate.
//   split    a thread takes 16 heads of a pair: float32 weights from shared memory, three bfloat16 pieces into tensor memory
//   mix      D0 = a0 t0; D12 = a2 t0 + a1 t1 + a0 t2 + a1 t0 + a0 t1 (the smallest first), added in float32 and rounded into shared memory
//   weights  of the next tile, and values of the last one, while the mix runs; one barrier of the CTA a tile of 16 keys
// Queries lie in tensor memory, the sums in registers; keys are copied two tiles ahead, values one.
// Bound: latencies.  A tile takes 5500 cycles: weights 2400 (2050 of the special-function unit), values 1000, the split 700, mixed weights 600, the rest waits; 42 % of
// the issue slots.  2048 tokens, 32 heads of 64 on 8: 283 us with the mix on mma.sync in tiles of 32 keys, 240 so.  Tried: an exponential of each weight as a polynomial 258;
// sums in tensor memory and queries in registers 248; queries in shared memory and three barriers a tile 275.
constexpr int kS3Keys = 16, kS3Tries = 1 << 18;
struct S3Layout {
    static constexpr int kPair = 4 * 32 + 16, kRow = kS3Keys * kPair + 16, kW = kStRows * kRow;      // bytes: a pair's weights, a query row's, a tile's
    static constexpr int kMixRow = 2 * kS3Keys + 16, kMixHead = kStRows * kMixRow + 16, kMix = 32 * kMixHead;
    static constexpr int t_off = 0, kv_off = 8192;   // t, and keys and values: rows of 128 swizzled bytes
    __host__ __device__ static constexpr int tile(int G) { return G * kS3Keys * 64; }   // elements: eight keys of every head, then the other eight
    __host__ __device__ static constexpr int total(int G) { return 1024 + kv_off + 2 * kW + 2 * kMix + 4 * 2 * tile(G); }
};
constexpr int kS3Groups = 8, kS3Smem = S3Layout::total(kS3Groups);   // key heads at most; the next number that divides 32 does not fit
static_assert(kS3Smem <= 226 * 1024, "shared memory of a CTA");
constexpr int kS3Block = 112, kS3D = 48, kS3D12 = 80, kS3Q = 224;   // tensor-memory columns of 128 pairs: pieces, D0, D12; behind both blocks': the queries

__device__ __forceinline__ void s3_st8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]),
                 "r"(r[6]), "r"(r[7])
                 : "memory");
}

__device__ __forceinline__ void s3_load(void *dst, const CUtensorMap *map, uint64_t *bar, int row) {   // 8 or 16 rows (the map's box) of all heads, from a multiple of 8 on
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %3, %3, %4}], [%2];" ::"r"(smem_u32(dst)),
                 "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(0), "r"(row >> 3)
                 : "memory");
}

// For heads of 64 whose pages are whole runs of eight keys: a tile goes by one TMA copy each of keys and values, by two where its halves may lie in different pages.  With
// cp.async pieces instead (1100 to 1700 cycles of issue a tile) this kernel loses on long prompts to the one above: 4000 tokens of 32 heads of 64 on 8 in pages of 8 or 4 keys 975 us
// there, 1107 here by pieces, 835 (pages of 8) here by TMA; of 48 and 32 on 8 912 and 975; of 32 and 48 on 16 1015 and 1143.
// Segments add in pairs, the pairs in order: (s0 + s1) + (s2 + s3) + ..  per: segments a CTA takes, 1 (each has a place of its own in `partial`), 2 (a place a pair), or 0: all of its
// rows', with a place for the first of a pair behind one for the running sum.  All give the same bits.  places: of a token.  No scratch: one chain over all keys.
__global__ void __launch_bounds__(512, 1) sigmoid_talk32_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const atoma_sigmoid_attn_args a, int lo, int hi, int per, int places, float *__restrict__ partial, unsigned int *late_out) {
    using L = S3Layout;
    constexpr int H = 32, NT = 512;
    extern __shared__ unsigned char sm_raw[];
    unsigned char *sm = sm_raw + ((1024u - (smem_u32(sm_raw) & 1023u)) & 1023u);
    pdl_launch_dependents();
    pdl_wait();
    constexpr int D = 64, DV = 64;
    const int G = static_cast<int>(a.G), bs = static_cast<int>(a.block_size);
    const int b = blockIdx.y;
    int seg = blockIdx.z * per;   // the segment in hand
    const int t_begin = a.query_start[b], n_q = a.query_start[b + 1] - t_begin;
    const int first = max(0, lo - t_begin + kStRows - 1) / kStRows, last = (min(n_q, hi - t_begin) + kStRows - 1) / kStRows - 1;   // this run's row blocks
    const int blk = last - static_cast<int>(blockIdx.x);   // the rows with the most keys first
    if (n_q <= 0 || blk < first) return;
    const int r0 = blk * kStRows, rows = min(kStRows, n_q - r0), tok0 = t_begin + r0;
    const int ctx = static_cast<int>(a.positions[t_begin]), p0 = ctx + r0, total = ctx + n_q;
    const int all_end = p0 + rows, j_begin = seg * kS3SegKeys, j_end = blockIdx.z + 1 == gridDim.z ? all_end : min(all_end, j_begin + per * kS3SegKeys);
    if (j_begin >= all_end) return;
    const int32_t *bt = a.block_tables + static_cast<int64_t>(b) * a.max_blocks;
    unsigned char *talk = sm + L::t_off;
    const int tile = L::tile(G);
    __nv_bfloat16 *Ks = reinterpret_cast<__nv_bfloat16 *>(sm + L::kv_off), *Vs = Ks + 2 * tile;
    unsigned char *weights = reinterpret_cast<unsigned char *>(Vs + 2 * tile), *mix = weights + 2 * L::kW;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, t4 = lane & 3, rq = lane >> 2;
    __shared__ int32_t slot_s[4][2];   // cache rows of a tile's first and ninth key (-1: behind the sequence's end), looked up three tiles ahead
    __shared__ __align__(8) uint64_t split[2], mixed[2], k_full[2], v_full[2];   // split, mixed: of 128 pairs each
    __shared__ uint32_t tmem_base_s;
    __shared__ int late_s;
    volatile int *late = &late_s;
    const int bs_shift = (bs & (bs - 1)) == 0 ? __ffs(bs) - 1 : -1;
    auto look_up = [&](int j) {
        const int pg = bs_shift >= 0 ? j >> bs_shift : j / bs;
        return j < total ? bt[pg] * bs + (j - pg * bs) : -1;
    };
    if (tid < 6) slot_s[tid / 2][tid % 2] = look_up(j_begin + tid * 8);
    if (tid == 0) {
        late_s = 0;
        for (int i = 0; i < 2; ++i) {
            mbar_init(&split[i], 8);
            mbar_init(&mixed[i], 1);
            mbar_init(&k_full[i], 1);
            mbar_init(&v_full[i], 1);
        }
        fence_mbar_init();
    }
    if (warp == 0) tmem_alloc(&tmem_base_s, 512);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = tmem_base_s;
    // Keys or values of tile j, from one thread.  The map and the barrier come with the call: one cache may serve as both.
    const bool whole = bs % kS3Keys == 0;   // a tile lies in one page
    auto stage = [&](const CUtensorMap *map, uint64_t *full, __nv_bfloat16 *buffers, int j) {
        __nv_bfloat16 *dst = buffers + (j & 1) * tile;
        mbar_arrive_expect_tx(&full[j & 1], G * kS3Keys * 128);
        s3_load(dst, map, &full[j & 1], max(slot_s[j & 3][0], 0));
        if (!whole) s3_load(dst + tile / 2, map, &full[j & 1], max(slot_s[j & 3][1], 0));
    };
    const int tiles = (j_end - j_begin + kS3Keys - 1) / kS3Keys;
    if (tid == 0) {
        stage(&map_k, k_full, Ks, 0);
        if (tiles > 1) stage(&map_k, k_full, Ks, 1);
    }
    // ---- the talk matrix in three pieces, rows of heads h: [t0 | t1], then [t2 | -] ----
    for (int i = tid; i < H * H; i += NT) {
        const int h = i / H, g = i % H;
        float piece[kStPieces];
        st_split(a.talk[i], piece);
#pragma unroll
        for (int k = 0; k < kStPieces; ++k) {
            const int col = (k & 1) * 64 + g * 2;
            *reinterpret_cast<__nv_bfloat16 *>(talk + (k >> 1) * 4096 + h * 128 + (((col >> 4) ^ (h & 7)) << 4) + (col & 15)) = __float2bfloat16_rn(piece[k]);
        }
    }
    fence_proxy_async();   // generic-proxy writes -> visible to the tensor core's asynchronous reads
    const int h0 = 2 * warp, kv_head[2] = {h0 / (H / G), (h0 + 1) / (H / G)};
    float slope[2], hb[2];
#pragma unroll
    for (int x = 0; x < 2; ++x) {
        slope[x] = a.slopes ? a.slopes[h0 + x] : 0.f;
        hb[x] = a.head_bias[h0 + x];
    }
    // ---- this warp's queries as the products take them, in tensor memory: [head][16 of its entries][fragment] ----
    const uint32_t tmem_q = tmem_base + kS3Q + (warp >> 2) * 32 + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    {
        uint32_t qf[32];
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            const __nv_bfloat16 *q = static_cast<const __nv_bfloat16 *>(a.q) + static_cast<int64_t>(tok0) * H * D + (h0 + x) * D;
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int row = rq + (e & 1) * 8, col = kk * 16 + 2 * t4 + (e >> 1) * 8;
                    qf[x * 16 + kk * 4 + e] = kk * 16 < D && row < rows ? *reinterpret_cast<const uint32_t *>(q + static_cast<int64_t>(row) * H * D + col) : 0u;
                }
        }
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
    const float in = a.softcap > 0.f ? a.scale * 2.8853900817779268f / a.softcap : 0.f;   // e^(2 s / cap) = 2^(in dot)
    // the sums of a segment, out of the accumulators: onto the first of its pair, onto the running sum, and into a place or, where no other segment follows or precedes, out
    auto put = [&](bool end) {
        const bool second = per != 1 && (seg & 1), onto = per == 0 && seg >= 2 && (end || second), out = end && (per == 0 || all_end <= per * kS3SegKeys);
        const int64_t row_len = static_cast<int64_t>(places) * H * DV;
        float *mine = partial + (tok0 - lo) * row_len + (per == 0 ? (second ? 0 : H * DV) : (per == 2 ? seg >> 1 : seg) * H * DV);
        auto each = [&](auto f) {
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int nt = 0; nt < 8; ++nt)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int row = rq + 8 * e;
                        if (row < rows) f(o[x][nt][2 * e], o[x][nt][2 * e + 1], row, (h0 + x) * DV + nt * 8 + 2 * t4);
                    }
        };
        auto add = [&](const float *from) {   // all loads before the first store
            each([&](float &u, float &v, int row, int col) {
                const float2 f = *reinterpret_cast<const float2 *>(from + row * row_len + col);
                u = f.x + u, v = f.y + v;
            });
        };
        if (second) add(per == 0 ? mine + H * DV : mine);
        if (onto) add(second ? mine : mine - H * DV);
        if (out)
            each([&](float u, float v, int row, int col) {
                *reinterpret_cast<uint32_t *>(static_cast<__nv_bfloat16 *>(a.out) + static_cast<int64_t>(tok0 + row) * H * DV + col) = pack2<__nv_bfloat16>(u, v);
            });
        else
            each([&](float u, float v, int row, int col) { *reinterpret_cast<float2 *>(mine + row * row_len + col) = make_float2(u, v); });
    };
    auto wait = [&](uint64_t *bar, uint32_t parity) {   // bounded, for a whole warp
#pragma unroll 1
        for (int i = 0; !mbar_try_wait(bar, parity);) {
            if (*late) break;
            if (++i == kS3Tries) {
                *late = 1;
                break;
            }
        }
        __syncwarp();
    };
    // ---- scores and weights of this warp's two heads for tile j ----
    auto form_weights_as = [&](auto all_seen, int j) {
        const int j0 = j_begin + j * kS3Keys;
        const __nv_bfloat16 *kt = Ks + (j & 1) * tile;
        unsigned char *wt = weights + (j & 1) * L::kW;
        const float base = static_cast<float>(p0 + rq - j0 - 2 * t4);
        float w0[2][4];
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            float s[2][4];
#pragma unroll
            for (int i = 0; i < 2; ++i) s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.f;
            const int key = ((lane >> 4) * G + kv_head[x]) * 8 + (lane & 7), odd = (lane >> 3) & 1;
            const uint32_t kb = smem_u32(kt + key * 64);
            uint32_t qf[16];
            tmem_ld_32x32b_x16(tmem_q + x * 16, qf);
            tmem_ld_wait();
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                uint32_t r[4];
                const uint32_t(&qk)[4] = *reinterpret_cast<const uint32_t(*)[4]>(qf + kk * 4);
                ldmatrix_x4(r, kb + (((2 * kk + odd) ^ (lane & 7)) << 4));
                Mma16816<__nv_bfloat16>::run(s[0], qk, r[0], r[1]);
                Mma16816<__nv_bfloat16>::run(s[1], qk, r[2], r[3]);
            }
            // weights of hidden pairs are formed too and dropped: without a branch per weight their chains of exponentials and quotients overlap
            auto weigh = [&](auto with_cap) {
#pragma unroll
                for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        s[nt][e] = st_weight<decltype(with_cap)::value>(s[nt][e], a.scale, in, a.softcap, slope[x], base - static_cast<float>(nt * 8 + (e & 1) - (e >> 1) * 8), hb[x]);
            };
            if (a.softcap > 0.f) weigh(std::true_type{});
            else weigh(std::false_type{});
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int row = rq + (e >> 1) * 8, key = nt * 8 + 2 * t4 + (e & 1);
                    const float w = decltype(all_seen)::value || (row < rows && p0 + row >= j0 + key) ? s[nt][e] : 0.f;
                    if (x == 0) w0[nt][e] = w;
                    else *reinterpret_cast<float2 *>(wt + row * L::kRow + key * L::kPair + h0 * 4) = make_float2(w0[nt][e], w);
                }
        }
    };
    auto form_weights = [&](int j) {
        wait(&k_full[j & 1], (j >> 1) & 1);
        if (rows == kStRows && j_begin + (j + 1) * kS3Keys - 1 <= p0) form_weights_as(std::true_type{}, j);
        else form_weights_as(std::false_type{}, j);
    };
    // this thread's pair: block of 128 pairs (8 query rows x 16 keys), and which 16 of its heads
    const int block = warp >> 3, half = (warp >> 2) & 1, pair = (warp & 3) * 32 + lane, prow = 8 * block + pair / kS3Keys, pkey = pair % kS3Keys;
    const uint32_t tmem_block = tmem_base + block * kS3Block, tmem_lane = tmem_block + (static_cast<uint32_t>((warp & 3) * 32) << 16);
    __syncthreads();
    form_weights(0);
    // The sequence ends inside tile j (its last one): what follows in the page (or, in a second copy, of another) is not multiplied in.  Every warp zeroes what it reads.
    auto hide_rows = [&](int j) {
        for (int x = 0; x < 2; ++x)
            for (int i = lane; i < kS3Keys * 8; i += 32)
                if (j_begin + j * kS3Keys + i / 8 >= total) *reinterpret_cast<uint4 *>(Vs + (j & 1) * tile + ((i / 64 * G + kv_head[x]) * 8 + i / 8 % 8) * 64 + i % 8 * 8) = make_uint4(0, 0, 0, 0);
        __syncwarp();
    };
    // ---- values of tile j: what the mix of all heads has given this warp's two ----
    auto add_values = [&](int j) {
        wait(&v_full[j & 1], (j >> 1) & 1);
        if (j_begin + (j + 1) * kS3Keys > total) hide_rows(j);
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            const uint32_t vb = smem_u32(Vs + (j & 1) * tile + ((((lane >> 3) & 1) * G + kv_head[x]) * 8 + (lane & 7)) * 64);
            uint32_t af[4];
            ldmatrix_x4(af, smem_u32(mix + (j & 1) * L::kMix + (h0 + x) * L::kMixHead + (lane & 15) * L::kMixRow + (lane >> 4) * 16));
#pragma unroll
            for (int n2 = 0; n2 < 4; ++n2) {
                uint32_t r[4];
                ldmatrix_x4_trans(r, vb + (((2 * n2 + (lane >> 4)) ^ (lane & 7)) << 4));
                Mma16816<__nv_bfloat16>::run(o[x][2 * n2], af, r[0], r[1]);
                Mma16816<__nv_bfloat16>::run(o[x][2 * n2 + 1], af, r[2], r[3]);
            }
        }
        if (partial && j + 1 < tiles && (j_begin + (j + 1) * kS3Keys) % kS3SegKeys == 0 && (per == 0 || (per == 2 && !(seg & 1)))) {   // a segment ends here
            put(false);
            ++seg;
            clear();
        }
    };
    for (int j = 0; j < tiles; ++j) {
        // The one barrier of a tile: its weights, the mixed weights of the tile before, its values and the next tile's keys are there.  What follows, a warp does at
        // its own pace, so that one's exponentials run beside another's products.
        __syncthreads();
        if (tid == 0) {
            stage(&map_v, v_full, Vs, j);
            if (j + 2 < tiles) stage(&map_k, k_full, Ks, j + 2);
        }
        int next_slot = 0;
        if (tid < 2) next_slot = look_up(j_begin + (j + 3) * kS3Keys + tid * 8);
        // ---- split ----
        {
            const float4 *w = reinterpret_cast<const float4 *>(weights + (j & 1) * L::kW + prow * L::kRow + pkey * L::kPair + half * 64);
            uint32_t piece[kStPieces][8];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float4 v = w[i];
                float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int e = 0; e < 2; ++e)
#pragma unroll
                    for (int k = 0; k < kStPieces; ++k) {
                        const uint32_t two = pack2<__nv_bfloat16>(x[2 * e], x[2 * e + 1]);
                        piece[k][2 * i + e] = two;
                        x[2 * e] -= __uint_as_float(two << 16);
                        x[2 * e + 1] -= __uint_as_float(two & 0xffff0000u);
                    }
            }
#pragma unroll
            for (int k = 0; k < kStPieces; ++k) s3_st8(tmem_lane + k * 16 + half * 8, piece[k]);
            tmem_st_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&split[block]);
        }
        // ---- mix: issued by the block's first warp ----
        if ((warp & 7) == 0) {
            wait(&split[block], j & 1);
            tc_fence_after_sync();
            const uint32_t id = umma_idesc_f16(128, H, true);
            const uint64_t t01 = umma_desc_k_sw128(smem_u32(talk)), t2 = umma_desc_k_sw128(smem_u32(talk) + 4096);
            if (elect_one_sync()) {
                auto product = [&](int pa, uint64_t t, uint32_t d, bool fresh) {   // both steps of 16 heads
                    umma_f16_ts(tmem_block + d, tmem_block + pa * 16, t, id, fresh ? 0u : 1u);
                    umma_f16_ts(tmem_block + d, tmem_block + pa * 16 + 8, t + 2, id, 1u);
                };
                product(2, t01, kS3D12, true);
                product(1, t01 + 4, kS3D12, false);
                product(0, t2, kS3D12, false);
                product(1, t01, kS3D12, false);
                product(0, t01 + 4, kS3D12, false);
                product(0, t01, kS3D, true);
                umma_commit(&mixed[block]);
            }
            __syncwarp();
        }
        // Half of every scheduler's warps form weights (special functions) while the others apply the last tile's (tensor pipe, shared memory): 255 us without, 242 so.
#pragma unroll 1
        for (int step = 0; step < 2; ++step) {
            if (step == ((warp >> 2) & 1)) {
                if (j > 0) add_values(j - 1);
            } else {
                if (j + 1 < tiles) form_weights(j + 1);
            }
        }
        // ---- the mixed weights of this thread's pair, rounded, to where the values' warps read them ----
        wait(&mixed[block], j & 1);
        tc_fence_after_sync();
        {
            uint32_t d0[16], d1[16];
            tmem_ld_32x32b_x16(tmem_lane + kS3D + half * 16, d0);
            tmem_ld_32x32b_x16(tmem_lane + kS3D12 + half * 16, d1);
            tmem_ld_wait();
            unsigned char *m = mix + (j & 1) * L::kMix + half * 16 * L::kMixHead + prow * L::kMixRow + pkey * 2;
#pragma unroll
            for (int i = 0; i < 16; i += 2) {
                const uint32_t two = pack2<__nv_bfloat16>(__uint_as_float(d0[i]) + __uint_as_float(d1[i]), __uint_as_float(d0[i + 1]) + __uint_as_float(d1[i + 1]));
                *reinterpret_cast<uint16_t *>(m + i * L::kMixHead) = static_cast<uint16_t>(two);
                *reinterpret_cast<uint16_t *>(m + (i + 1) * L::kMixHead) = static_cast<uint16_t>(two >> 16);
            }
        }
        tc_fence_before_sync();
        if (tid < 2) slot_s[(j + 3) & 3][tid] = next_slot;
    }
    __syncthreads();
    add_values(tiles - 1);
    put(true);
    if (tid == 0) {   // whatever happened to the waits, the copies have landed before the CTA leaves
        auto landed = [&](uint64_t *bar, int uses) {
            for (int i = 0; uses > 0 && i < kS3Tries && !mbar_try_wait(bar, (uses - 1) & 1); ++i) {
            }
        };
        for (int i = 0; i < 2; ++i) {
            landed(&k_full[i], (tiles + 1 - i) / 2);
            landed(&v_full[i], (tiles + 1 - i) / 2);
        }
    }
    __syncthreads();
    tc_fence_after_sync();
    if (warp == 0) tmem_dealloc(tmem_base, 512);
    if (tid == 0 && *late && late_out) *reinterpret_cast<volatile unsigned int *>(late_out) = 1;
}

// A token's places of seg_keys keys each, in order, or in pairs (sigmoid_talk32_kernel); tokens of one place are out already.  AHEAD: places that a thread asks for at a time.
// Steps of many tokens hide the latency by their CTAs; few tokens of many places are bound by it (33 tokens behind 30000 keys, 118 places of 32 heads of 64, four / sixteen at a
// time: 51 / 16 us; 2048 tokens of eight places, the whole call 239 / 268).
template <int AHEAD>
__global__ void __launch_bounds__(256) sigmoid_talk_sum_kernel(const atoma_sigmoid_attn_args a, const float *__restrict__ partial, int lo, int hi, int segs, int seg_keys, int pairs) {
    pdl_launch_dependents();
    pdl_wait();
    const int64_t t = lo + static_cast<int64_t>(blockIdx.x);
    const int b = a.token_seq[t], t_begin = a.query_start[b], n_q = a.query_start[b + 1] - t_begin;
    const int r0 = static_cast<int>(t - t_begin) / kStRows * kStRows, end = static_cast<int>(a.positions[t_begin]) + min(r0 + kStRows, n_q);
    const int n = min(segs, (end + seg_keys - 1) / seg_keys), row = static_cast<int>(a.H * a.vdim);
    if (n < 2 || t_begin + r0 < lo || t_begin + r0 >= hi) return;
    const float *p = partial + (t - lo) * segs * row;
    auto plus = [](float4 u, float4 v) { return make_float4(u.x + v.x, u.y + v.y, u.z + v.z, u.w + v.w); };
    for (int i = (blockIdx.y * 256 + threadIdx.x) * 4; i < row; i += gridDim.y * 1024) {
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int k0 = 0; k0 < n; k0 += AHEAD) {
            float4 v[AHEAD];
#pragma unroll
            for (int j = 0; j < AHEAD; ++j)
                if (k0 + j < n) v[j] = *reinterpret_cast<const float4 *>(p + static_cast<int64_t>(k0 + j) * row + i);
#pragma unroll
            for (int j = 0; j < AHEAD; j += 2) {
                if (k0 + j >= n) break;
                const bool two = k0 + j + 1 < n;
                if (pairs && two) v[j] = plus(v[j], v[j + 1]);
                s = k0 + j > 0 ? plus(s, v[j]) : v[j];
                if (!pairs && two) s = plus(s, v[j + 1]);
            }
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

namespace {
// A cache of rows of G heads of 64 as runs of eight: one or two runs a copy, in each all heads' keys, head by head.
bool s3_map(CUtensorMap *out, const void *cache, int G, int runs) {
    EncodeTiledFn enc = get_encode_tiled();
    if (!enc) return false;
    const cuuint64_t g = static_cast<cuuint64_t>(G), dims[4] = {64, 8, g, 1ull << 28}, strides[3] = {g * 128, 128, g * 1024};
    const cuuint32_t box[4] = {64, 8, static_cast<cuuint32_t>(G), static_cast<cuuint32_t>(runs)}, estr[4] = {1, 1, 1, 1};
    const CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void *>(cache), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r == CUDA_SUCCESS) return true;
    set_status(kErrDriver, "sigmoid_talk: cuTensorMapEncodeTiled failed (CUresult %d)", static_cast<int>(r));
    return false;
}
}  // namespace

bool hyb_sigmoid_talk(const atoma_sigmoid_attn_args &a, cudaStream_t stream) {
    const int64_t longest = a.max_seq_len > 0 ? a.max_seq_len : a.max_blocks * a.block_size;
    const int G = static_cast<int>(a.G), D = static_cast<int>(a.dim), DV = static_cast<int>(a.vdim);
    // by the sizes of the model and its pages alone: a position's bits do not follow the step
    const bool on_tcgen05 = a.H == 32 && D == 64 && DV == 64 && G <= kS3Groups && a.block_size % 8 == 0;
    const int64_t seg_keys = on_tcgen05 ? kS3SegKeys : kStSegKeys, segs = std::min<int64_t>(65535, (longest + seg_keys - 1) / seg_keys), blocks = (a.T + kStRows - 1) / kStRows;
    const int64_t place = a.H * a.vdim * 4;   // bytes of a token's sums
    int64_t slots = 1, run = a.T;   // places a token; tokens a launch
    int per = on_tcgen05 ? 0 : 1;   // sigmoid_talk32_kernel: segments a CTA
    float *partial = nullptr;
    if (segs > 1) {
        // a segment per CTA unless the row blocks are four per SM and more, or two and the segments' sums do not fit at once
        auto fits = [&](int64_t n) { return std::max<int64_t>(kStRows, kStScratch / (n * place) / kStRows * kStRows); };
        const int64_t sms = current_device_info().sm_count, pairs = (segs + 1) / 2, most = on_tcgen05 ? pairs : segs;
        const bool chains = blocks >= 4 * sms || (blocks >= 2 * sms && fits(most) < a.T);
        if (on_tcgen05) {
            // Two of the shorter segments a CTA, and one place for both, where the row blocks have many (a CTA's start and end cost some four tiles), or where single ones do not
            // fit at once: a bound of 16384 keys (one that the caller does not know, in a wide table), 600 and 2048 tokens, us, on single places 234 and 478, on
            // pairs 122 and 357; of 131072 keys 801 and 3368, 435 and 1742.
            per = chains ? 0 : (fits(segs) < a.T || blocks * segs >= 4 * sms ? 2 : 1);
            slots = chains ? 2 : (per == 2 ? pairs : segs);
        } else {
            slots = chains ? 1 : segs;
        }
        run = std::min(a.T, fits(slots));
        if (on_tcgen05 && run < a.T) {   // runs of one length
            const int64_t n = (a.T + run - 1) / run;
            run = ((a.T + n - 1) / n + kStRows - 1) / kStRows * kStRows;
        }
        partial = static_cast<float *>(try_workspace(stream, static_cast<size_t>((run + kStRows) * slots * place), kWorkspaceHybridAttn));   // a run's last row block may end behind it
        if (!partial) slots = 1, run = a.T, per = on_tcgen05 ? 0 : 1;   // no scratch: one chain needs none
    }
    const int64_t shares = on_tcgen05 ? (per == 0 ? 1 : (segs + per - 1) / per) : slots;   // CTAs of a row block
    const int runs = a.block_size % kS3Keys == 0 ? 2 : 1;
    CUtensorMap map_k{}, map_v{};
    if (on_tcgen05 && (!s3_map(&map_k, a.k_cache, G, runs) || !s3_map(&map_v, a.v_cache, G, runs))) return false;
    auto kernel = a.H == 16 ? sigmoid_talk_kernel<1> : sigmoid_talk_kernel<2>;
    const size_t smem = a.H == 16 ? StLayout<1>::total(G, D, DV) : on_tcgen05 ? S3Layout::total(G) : StLayout<2>::total(G, D, DV);
    const cudaError_t attr = on_tcgen05 ? cudaFuncSetAttribute(sigmoid_talk32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kS3Smem)
                                        : cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 225 * 1024);
    if (attr != cudaSuccess) return hybrid::launched(attr, "sigmoid_talk_kernel");
    for (int64_t lo = 0; lo < a.T; lo += run) {
        const int64_t hi = std::min(a.T, lo + run), rows = (std::min<int64_t>(hi - lo, a.max_query_len) + kStRows - 1) / kStRows + 1;
        const dim3 grid(static_cast<unsigned>(rows), static_cast<unsigned>(a.B), static_cast<unsigned>(shares));
        const dim3 block(16 * static_cast<unsigned>(a.H));
        const int from = static_cast<int>(lo), to = static_cast<int>(hi), places = static_cast<int>(slots);
        if (!hybrid::launched(on_tcgen05 ? launch_ex(sigmoid_talk32_kernel, grid, block, smem, stream, map_k, map_v, a, from, to, per, places, partial, late_word())
                                         : launch_ex(kernel, grid, block, smem, stream, a, from, to, places, partial),
                              "sigmoid_talk_kernel"))
            return false;
        if (shares > 1) {
            const unsigned tokens = static_cast<unsigned>(std::min(a.T, hi + kStRows) - lo);
            const bool few = slots >= 24 && static_cast<int>(tokens) <= 2 * current_device_info().sm_count;
            const dim3 sums(tokens, few ? static_cast<unsigned>((place + 4095) / 4096) : 1);
            if (!hybrid::launched(launch_ex(few ? sigmoid_talk_sum_kernel<16> : sigmoid_talk_sum_kernel<4>, sums, dim3(256), 0, stream, a, static_cast<const float *>(partial), from, to,
                                            places, static_cast<int>(per == 2 ? 2 * seg_keys : seg_keys), on_tcgen05 && per == 1 ? 1 : 0),
                                  "sigmoid_talk_sum_kernel"))
                return false;
        }
    }
    return true;
}

}  // namespace atoma
