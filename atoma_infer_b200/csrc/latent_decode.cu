// Latent attention of DECODED tokens (one query token per sequence, up to 32 heads) on tcgen05 — include/atoma_hybrid.h,
// atoma_latent_attention_paged; bfloat16 caches whose rows are 128 to 576 entries in steps of 64,
// in pages of whole groups of eight rows.
//
// Bound: the cache stream (a row of 576 entries is read once for all heads, as keys and as values).  The heads of a token are far too few rows
// for a 128-row product, so the products are turned around: the CACHED ROWS are the wide operand and the heads the narrow one,
//   S^T [64 keys x heads]    = C [64 keys x R] . Q^T           (M = 64, N = heads, K = R; C as stored)
//   O^T [columns x heads]   += C^T [128 columns x 64 keys] . P^T  (M = 128 per 128 columns, N = heads, K = 64; the SAME tile, read transposed)
// with S^T (two buffers) and O^T in tensor memory; nothing is padded but heads to 16 or 32.  Per 64-key tile of 73 KB: about 3500 cycles of
// products and softmax in a row, half of them under the next tile's copy, where the bytes alone take 3200 at the HBM rate per SM.
//
// Work: all sequences' 64-key tiles in a row, cut into equal runs, one per CTA (a CTA fills an SM's shared memory), so ragged contexts keep
// every SM reading to the end; a sequence that several CTAs share is merged in CTA order by latent_decode_merge_kernel.
// Warps 0-3: softmax and results (a thread owns a head and an eighth or a quarter of a tile's keys; scores change hands through shared memory),
// warp 4: loads (TMA, eight rows a copy, rows through the block table; one tile lands while the other is used), warp 5: products.
// O^T is rescaled whenever a head's maximum grows, so that the largest weight is 1, which bfloat16 holds (error against 64 bits at batch 32, contexts of 2048 to
// 4096: 3.015e-3; rescaled from 2^8 on 3.061e-3 and 2 us less of 80).
//
// Every wait is bounded: one that runs out raises a flag, the other roles stop waiting, the loads land, tensor memory is freed and a
// counter is raised (atoma_latent_decode_timeouts, atoma_kernel_timeouts).
#include "common.cuh"
#include "hybrid_common.cuh"

#include "atoma_hybrid.h"

#include <algorithm>

namespace atoma {
namespace {

using namespace hybrid;

constexpr int kLdKeys = 64, kLdStages = 2, kLdGroup = 8;   // keys per tile; keys per copy: one group of the 128-byte swizzle
constexpr int kLdThreads = 192;                             // softmax 0-3, loads 4, products 5
constexpr int kLdMaxSeqs = 512;
constexpr int kLdTries = 1 << 18;
constexpr int kLdPlain = 9;                    // 16-byte loads in flight per lane where a group goes by plain loads
constexpr int kLdOCol = 64, kLdTmem = 256;     // S^T: columns 0.. and 32..; O^T: 32 columns per 128 latent columns from 64 on

__device__ unsigned int g_latent_late;

__device__ __forceinline__ void ld_wait(uint64_t *bar, uint32_t parity, volatile int *late) {
#pragma unroll 1
    for (int i = 0; !mbar_try_wait(bar, parity);) {
        if (*late) break;
        if (++i == kLdTries) {
            *late = 1;
            break;
        }
    }
}
__host__ __device__ __forceinline__ long long ld_start(long long units, int c, int n) { return units * c / n; }
__host__ __device__ __forceinline__ int ld_owner(long long units, long long u, int n) { return static_cast<int>(((u + 1) * n + units - 1) / units - 1); }

// umma_desc_k_sw128 / umma_desc_mn_sw128 (common.cuh) with the distances of this layout: groups of eight rows `sbo` bytes apart, 64-entry blocks `lbo`.
__device__ __forceinline__ uint64_t ld_desc(uint32_t smem_addr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = static_cast<uint64_t>((smem_addr & 0x3FFFFu) >> 4);
    d |= static_cast<uint64_t>(lbo > 16 ? lbo >> 4 : lbo) << 16;
    d |= static_cast<uint64_t>(sbo >> 4) << 32;
    d |= static_cast<uint64_t>(1) << 46;
    d |= static_cast<uint64_t>(2) << 61;
    return d;
}
__device__ __forceinline__ void tma_load_3d(void *smem_dst, const CUtensorMap *map, uint64_t *bar, int c0, int c1, int c2) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%3, %4, %5}], [%2], %6;" ::"r"(smem_u32(smem_dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "l"(kL2EvictFirst)
        : "memory");
}

// A sequence's first tile starts on a whole group of rows (inside the page of lo: pages are whole groups).
__device__ __forceinline__ int ld_first(int lo) { return lo & ~(kLdGroup - 1); }

// Keys [lo, hi) that row b's token sees, and the tiles they take; no tokens or a portion served elsewhere: none.
__device__ __forceinline__ int ld_span(const atoma_latent_attn_args &a, int b, int &lo, int &hi) {
    const int q0 = a.query_start[b], nq = a.query_start[b + 1] - q0;
    lo = hi = 0;
    if (nq <= 0 || (a.skip_min_q > 0 && nq >= a.skip_min_q)) return 0;
    hi = static_cast<int>(a.positions[q0]) + 1;
    lo = a.window > 0 ? max(0, hi - static_cast<int>(a.window)) : 0;
    return (hi - ld_first(lo) + kLdKeys - 1) / kLdKeys;
}

template <int NH>   // heads, padded: 16 or 32
__global__ void __launch_bounds__(kLdThreads, 1)
latent_decode_kernel(const __grid_constant__ CUtensorMap map, const atoma_latent_attn_args a, float *__restrict__ partial, float *__restrict__ partial_ml, int *__restrict__ prefix_out,
                     unsigned int *late_out) {
    constexpr int kParts = 128 / NH, kPart = kLdKeys / kParts;   // keys of a tile per softmax thread: 8 or 16
    constexpr int kSLd = NH + 1;
    extern __shared__ unsigned char smem_dyn[];
    const int R = static_cast<int>(a.R), H = static_cast<int>(a.H), B = static_cast<int>(a.B), kbs = R / 64, pieces = R / 8;
    const int Rv = a.out_cols > 0 ? static_cast<int>(a.out_cols) : R;
    const int stage_bytes = kLdKeys * R * 2;
    unsigned char *ring = smem_dyn + ((1024u - (smem_u32(smem_dyn) & 1023u)) & 1023u);
    unsigned char *qs = ring + kLdStages * stage_bytes;             // [64-entry block][NH rows][128 bytes]
    unsigned char *ps = qs + kbs * NH * 128;                        // [2][NH rows][128 bytes]: 64 keys
    float *ss = reinterpret_cast<float *>(ps + 2 * NH * 128);       // [64 keys][NH + 1]
    int *prefix = reinterpret_cast<int *>(ss + kLdKeys * kSLd);     // [B + 1] tiles before every sequence
    __shared__ __align__(8) uint64_t full[kLdStages], empty[kLdStages], s_full[2], p_full, pv_done, q_full;
    __shared__ uint32_t tmem_base_smem;
    __shared__ int late_s;
    __shared__ float merge_s[kParts][NH], alpha_s[NH];
    volatile int *late = &late_s;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        late_s = 0;
        for (int i = 0; i < kLdStages; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        mbar_init(&s_full[0], 1);
        mbar_init(&s_full[1], 1);
        mbar_init(&p_full, 4);         // the softmax warps
        mbar_init(&pv_done, 1);
        mbar_init(&q_full, 4);
        fence_mbar_init();
        tma_prefetch_desc(&map);
    }
    if (warp == 5) tmem_alloc(&tmem_base_smem, kLdTmem);
    pdl_launch_dependents();
    pdl_wait();
    if (warp == 0) {   // tiles before every sequence
        int base = 0;
        for (int b0 = 0; b0 < B; b0 += 32) {
            int lo, hi;
            const int n = b0 + lane < B ? ld_span(a, b0 + lane, lo, hi) : 0;
            int x = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            if (b0 + lane < B) prefix[b0 + lane] = base + x - n;
            base += __shfl_sync(0xffffffffu, x, 31);
        }
        if (lane == 0) prefix[B] = base;
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = tmem_base_smem;
    const int units = prefix[B];
    const int cta = blockIdx.x, ncta = min(static_cast<int>(gridDim.x), units);
    if (cta == 0)
        for (int i = tid; i <= B; i += kLdThreads) prefix_out[i] = prefix[i];
    const int u0 = cta < ncta ? static_cast<int>(ld_start(units, cta, ncta)) : 0, u1 = cta < ncta ? static_cast<int>(ld_start(units, cta + 1, ncta)) : 0;
    int b_first = 0;
    if (u0 < u1) {   // the last sequence that starts at or before u0 and is not empty
        int lo = 0, hi = B - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) / 2;
            if (prefix[mid] <= u0) lo = mid;
            else hi = mid - 1;
        }
        b_first = lo;
    }

    if (warp < 4) {
        // ============================ softmax, results ============================
        const int h = tid % NH, part = tid / NH;
        const float sc = a.scale * 1.4426950408889634f;
        const uint32_t taddr = tmem_base + (static_cast<uint32_t>(warp * 32) << 16);
        int it = 0;
        for (int u = u0, b = b_first; u < u1; ++b) {
            const int e = min(prefix[b + 1], u1);
            if (e <= u) continue;
            int k_lo, k_hi;
            ld_span(a, b, k_lo, k_hi);
            const int64_t token = a.query_start[b];
            // ---- queries -> bfloat16 rows in the products' layout (the products of the sequence before are complete) ----
            const float *q = a.q_lat + token * H * R;
            constexpr int kBatch = 9;   // 32 heads of 576 in two rounds of eighteen loads; three rounds of twelve 55.3 us for 54.1 (32 sequences), one load at a time 8 us a sequence
            for (int i0 = tid; i0 < NH * pieces; i0 += kBatch * 128) {
                float4 v[kBatch][2];
#pragma unroll
                for (int k = 0; k < kBatch; ++k) {
                    const int i = min(i0 + k * 128, NH * pieces - 1), r = i / pieces, c = i - r * pieces;
                    const float4 *src = reinterpret_cast<const float4 *>(q + static_cast<int64_t>(min(r, H - 1)) * R + c * 8);
                    v[k][0] = src[0];
                    v[k][1] = src[1];
                }
#pragma unroll
                for (int k = 0; k < kBatch; ++k) {
                    const int i = i0 + k * 128, r = i / pieces, c = i - r * pieces;
                    uint4 w = make_uint4(0, 0, 0, 0);
                    if (r < H)
                        w = make_uint4(pack2<__nv_bfloat16>(v[k][0].x, v[k][0].y), pack2<__nv_bfloat16>(v[k][0].z, v[k][0].w), pack2<__nv_bfloat16>(v[k][1].x, v[k][1].y),
                                       pack2<__nv_bfloat16>(v[k][1].z, v[k][1].w));
                    if (i < NH * pieces) *reinterpret_cast<uint4 *>(qs + (c >> 3) * (NH * 128) + r * 128 + (((c & 7) ^ (r & 7)) << 4)) = w;
                }
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(&q_full);
            float m_ref = -INFINITY, l_run = 0.f;
            if (a.sink && u == prefix[b] && h < H) {   // one more term of the denominator, on the sequence's first CTA
                m_ref = a.sink[h] * 1.4426950408889634f;
                l_run = part == 0 ? 1.f : 0.f;
            }
            const int first = it;
            for (int j0 = ld_first(k_lo) + (u - prefix[b]) * kLdKeys; u < e; ++u, ++it, j0 += kLdKeys) {
                ld_wait(&s_full[it & 1], (it >> 1) & 1, late);
                tc_fence_after_sync();
                uint32_t sv[NH];
                if constexpr (NH == 32) tmem_ld_32x32b_x32(taddr + (it & 1) * 32, sv);
                else tmem_ld_32x32b_x16(taddr + (it & 1) * 32, sv);
                tmem_ld_wait();
                if (lane < 16) {   // M = 64: rows 16 w .. 16 w + 15 in the first lanes of warp w's quarter
                    float *row = ss + (warp * 16 + lane) * kSLd;
                    const int key = j0 + warp * 16 + lane;
                    const bool seen = key < k_hi && key >= k_lo;
#pragma unroll
                    for (int i = 0; i < NH; ++i) row[i] = seen ? __uint_as_float(sv[i]) * sc : -INFINITY;
                }
                named_bar_sync(1, 128);
                float x[kPart], mx = -INFINITY;
#pragma unroll
                for (int i = 0; i < kPart; ++i) {
                    x[i] = ss[(part * kPart + i) * kSLd + h];
                    mx = fmaxf(mx, x[i]);
                }
                uint32_t any;
                {
                    const uint32_t need = mx > m_ref ? 1u : 0u;   // also a first finite score
                    asm volatile(
                        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbarrier.cta.red.or.pred q, 2, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                        : "=r"(any)
                        : "r"(need)
                        : "memory");
                }
                if (any) {
                    merge_s[part][h] = mx;
                    named_bar_sync(1, 128);
                    float mt = merge_s[0][h];
#pragma unroll
                    for (int i = 1; i < kParts; ++i) mt = fmaxf(mt, merge_s[i][h]);
                    const bool move = mt > m_ref;
                    const float alpha = move ? (m_ref == -INFINITY ? 0.f : fast_exp2(m_ref - mt)) : 1.f;
                    if (move) m_ref = mt;
                    l_run *= alpha;
                    if (part == 0) alpha_s[h] = alpha;
                    named_bar_sync(1, 128);
                    if (it > first) {
                        ld_wait(&pv_done, (it - 1) & 1, late);
                        tc_fence_after_sync();
                        for (int c = 0; c < Rv / 128; ++c) {
                            uint32_t o[NH];
                            const uint32_t at = taddr + kLdOCol + c * 32;
                            if constexpr (NH == 32) tmem_ld_32x32b_x32(at, o);
                            else tmem_ld_32x32b_x16(at, o);
                            tmem_ld_wait();
#pragma unroll
                            for (int i = 0; i < NH; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha_s[i]);
                            if constexpr (NH == 32) tmem_st_32x32b_x32(at, o);
                            else tmem_st_32x32b_x16(at, o);
                        }
                        tmem_st_wait();
                    }
                }
                const float m_use = m_ref == -INFINITY ? 0.f : m_ref;
                uint32_t pk[kPart / 2];
#pragma unroll
                for (int i = 0; i < kPart / 2; ++i) {
                    const float p0 = fast_exp2(x[2 * i] - m_use), p1 = fast_exp2(x[2 * i + 1] - m_use);
                    l_run += p0 + p1;
                    pk[i] = pack2<__nv_bfloat16>(p0, p1);
                }
                unsigned char *prow = ps + (it & 1) * (NH * 128) + h * 128;
#pragma unroll
                for (int i = 0; i < kPart / 8; ++i)
                    *reinterpret_cast<uint4 *>(prow + (((part * (kPart / 8) + i) ^ (h & 7)) << 4)) = make_uint4(pk[4 * i], pk[4 * i + 1], pk[4 * i + 2], pk[4 * i + 3]);
                fence_proxy_async();
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(&p_full);
            }
            // ---- the run's sums: out when the whole sequence was this CTA's, else for the merge ----
            merge_s[part][h] = l_run;
            named_bar_sync(1, 128);
            float l = merge_s[0][h];
#pragma unroll
            for (int i = 1; i < kParts; ++i) l += merge_s[i][h];
            const bool whole = first == it - (prefix[b + 1] - prefix[b]);
            const int slot = b + cta;   // CTAs and sequences both ascend: no two runs share a slot
            if (part == 0) {
                alpha_s[h] = l == 0.f ? 0.f : 1.f / l;
                if (!whole && h < H) {
                    partial_ml[(static_cast<int64_t>(slot) * NH + h) * 2] = m_ref;
                    partial_ml[(static_cast<int64_t>(slot) * NH + h) * 2 + 1] = l;
                }
            }
            named_bar_sync(1, 128);
            ld_wait(&pv_done, (it - 1) & 1, late);
            tc_fence_after_sync();
            // a run for the merge is laid out [column][heads], as the accumulator gives it: 16-byte stores
            float *out = a.out + token * H * R + warp * 32 + lane, *part_out = partial + (static_cast<int64_t>(slot) * Rv + warp * 32 + lane) * NH;
            for (int c = 0; c < Rv / 128; ++c) {
                uint32_t o[NH];
                if constexpr (NH == 32) tmem_ld_32x32b_x32(taddr + kLdOCol + c * 32, o);
                else tmem_ld_32x32b_x16(taddr + kLdOCol + c * 32, o);
                tmem_ld_wait();
                if (whole) {
#pragma unroll
                    for (int i = 0; i < NH; ++i)
                        if (i < H) out[i * R + c * 128] = __uint_as_float(o[i]) * alpha_s[i];
                } else {
#pragma unroll
                    for (int i = 0; i < NH; i += 4) *reinterpret_cast<uint4 *>(part_out + c * 128 * NH + i) = make_uint4(o[i], o[i + 1], o[i + 2], o[i + 3]);
                }
            }
            tc_fence_before_sync();
            named_bar_sync(1, 128);   // alpha_s, merge_s and the query rows are free for the next sequence
        }
    } else if (warp == 4) {
        // ============================ loads ============================
        // A copy moves eight neighbouring rows: one run of bytes in memory, R / 64 swizzled groups of 1 KiB in shared memory (cp.async, a 16-byte
        // piece each, kept only some 30 KB of an SM's loads in flight: 2.9 us a tile).  What lies before a window or behind a sequence's end is zero: the
        // groups that hold them go by plain loads.
        const __nv_bfloat16 *cache = static_cast<const __nv_bfloat16 *>(a.latent_cache);
        const int bs = static_cast<int>(a.block_size), group_bytes = kLdGroup * R * 2;
        int it = 0;
        bool go = true;
        for (int u = u0, b = b_first; u < u1 && go; ++b) {
            const int e = min(prefix[b + 1], u1);
            if (e <= u) continue;
            int k_lo, k_hi;
            ld_span(a, b, k_lo, k_hi);
            const int32_t *table = a.block_tables + static_cast<int64_t>(b) * a.max_blocks;
            int j0 = ld_first(k_lo) + (u - prefix[b]) * kLdKeys;
            auto group_row = [&](int j) {   // cache row of group lane % 8's first key
                const int key = j + (lane & 7) * kLdGroup;
                return key < k_hi ? table[key / bs] * bs + key % bs : 0;
            };
            int row = group_row(j0);
            for (; u < e; ++u, ++it, j0 += kLdKeys) {
                const int st = it & 1;
                ld_wait(&empty[st], ((it >> 1) & 1) ^ 1, late);
                if (__any_sync(0xffffffffu, *late != 0)) {
                    go = false;
                    break;
                }
                unsigned char *dst = ring + st * stage_bytes;
                // Groups [cut, whole) lie inside the keys that are seen.  The first one of a window and the one that holds the end go by plain loads, with
                // zeros for what is not seen (a hidden row's weight is 0, which does not make a sum of a row that holds an infinity or NaN), and what
                // follows the end is zeros.
                const int cut = j0 < k_lo ? 1 : 0, whole = max(cut, min(kLdKeys, k_hi - j0) / kLdGroup);
                const int ends = (k_hi - j0 + kLdGroup - 1) / kLdGroup;   // groups from here on hold nothing
                auto plain = [&](int g) {
                    const int r = lane >> 2, key = j0 + g * kLdGroup + r;
                    const bool seen = key >= k_lo && key < k_hi;
                    const __nv_bfloat16 *src = cache + (static_cast<int64_t>(__shfl_sync(0xffffffffu, row, g)) + r) * R + (lane & 3) * 8;
                    unsigned char *to = dst + g * group_bytes + r * 128;
                    for (int k0 = 0; k0 < pieces / 4; k0 += kLdPlain) {
                        uint4 v[kLdPlain];
#pragma unroll
                        for (int k = 0; k < kLdPlain; ++k) {
                            v[k] = make_uint4(0, 0, 0, 0);
                            if (seen && k0 + k < pieces / 4) v[k] = *reinterpret_cast<const uint4 *>(src + (k0 + k) * 32);
                        }
#pragma unroll
                        for (int k = 0; k < kLdPlain; ++k) {
                            const int c = 4 * (k0 + k) + (lane & 3);
                            if (k0 + k < pieces / 4) *reinterpret_cast<uint4 *>(to + (c >> 3) * 1024 + (((c & 7) ^ r) << 4)) = v[k];
                        }
                    }
                };
                if (cut) plain(0);
                if (whole < min(ends, kLdKeys / kLdGroup)) plain(whole);
                if (ends < kLdKeys / kLdGroup)
                    for (int i = max(cut, ends) * group_bytes / 16 + lane; i < stage_bytes / 16; i += 32) reinterpret_cast<uint4 *>(dst)[i] = make_uint4(0, 0, 0, 0);
                fence_proxy_async();   // generic-proxy writes -> visible to the tensor core's async reads
                __syncwarp();
                if (elect_one_sync()) mbar_arrive_expect_tx(&full[st], (whole - cut) * group_bytes);
                for (int g = cut; g < whole; ++g) {
                    const int first = __shfl_sync(0xffffffffu, row, g);
                    if (elect_one_sync()) tma_load_3d(dst + g * group_bytes, &map, &full[st], 0, first, 0);
                    __syncwarp();
                }
                if (u + 1 < e) row = group_row(j0 + kLdKeys);
            }
        }
        // whatever happened to the other roles, the copies have landed before this warp leaves
        for (int i = max(0, it - kLdStages); i < it; ++i)
            for (int k = 0; k < kLdTries && !mbar_try_wait(&full[i & 1], (i >> 1) & 1); ++k) {
            }
    } else {
        // ============================ products ============================
        const uint32_t idesc_s = umma_idesc_f16(64, NH, true), idesc_o = umma_idesc_f16(128, NH, true) | (1u << 15);   // A of the second: columns contiguous
        const uint32_t group_bytes = kLdGroup * R * 2, ring_a = smem_u32(ring), q_a = smem_u32(qs), p_a = smem_u32(ps);
        int it = 0, seg = 0;
        auto scores = [&](int i) {
            tc_fence_after_sync();
            if (elect_one_sync()) {
                for (int kb = 0; kb < kbs; ++kb) {
                    const uint64_t da = ld_desc(ring_a + (i & 1) * stage_bytes + kb * 1024, 1, group_bytes), db = umma_desc_k_sw128(q_a + kb * (NH * 128));
#pragma unroll
                    for (int k = 0; k < 4; ++k) umma_f16_ss(tmem_base + (i & 1) * 32, da + 2 * k, db + 2 * k, idesc_s, (kb | k) != 0 ? 1u : 0u);
                }
                umma_commit(&s_full[i & 1]);
            }
            __syncwarp();
        };
        for (int u = u0, b = b_first; u < u1; ++b) {
            const int e = min(prefix[b + 1], u1);
            if (e <= u) continue;
            const int n = e - u;
            ld_wait(&q_full, seg & 1, late);   // this sequence's queries are there, the last one's sums are out of tensor memory
            tc_fence_after_sync();
            ld_wait(&full[it & 1], (it >> 1) & 1, late);
            scores(it);
            for (int i = 0; i < n; ++i, ++it) {
                // The next tile's scores under the softmax of this one if that tile has landed by then; else this tile's sums first, which give
                // its stage back to the loads.
                bool ahead = false;
                for (int k = 0; !__all_sync(0xffffffffu, mbar_try_wait(&p_full, it & 1)); ++k) {
                    if (!ahead && i + 1 < n && __all_sync(0xffffffffu, mbar_try_wait(&full[(it + 1) & 1], ((it + 1) >> 1) & 1))) {
                        scores(it + 1);
                        ahead = true;
                    }
                    if (k == kLdTries) *late = 1;
                    if (__any_sync(0xffffffffu, *late != 0)) break;
                }
                tc_fence_after_sync();
                if (elect_one_sync()) {
                    const uint32_t tile = ring_a + (it & 1) * stage_bytes;
                    for (int c = 0; c < Rv / 128; ++c) {
#pragma unroll
                        for (int k = 0; k < kLdKeys / 16; ++k)
                            umma_f16_ss(tmem_base + kLdOCol + c * 32, ld_desc(tile + c * 2 * 1024 + k * 2 * group_bytes, 1024, group_bytes),
                                        umma_desc_k_sw128(p_a + (it & 1) * (NH * 128) + k * 32), idesc_o, (i | k) != 0 ? 1u : 0u);
                    }
                    umma_commit(&empty[it & 1]);
                    umma_commit(&pv_done);
                }
                __syncwarp();
                if (!ahead && i + 1 < n) {
                    ld_wait(&full[(it + 1) & 1], ((it + 1) >> 1) & 1, late);
                    scores(it + 1);
                }
            }
            u = e;
            ++seg;
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 5) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, kLdTmem);
    }
    if (tid == 0 && *late) {
        atomicAdd(&g_latent_late, 1u);
        if (late_out) *reinterpret_cast<volatile unsigned int *>(late_out) = 1;
    }
}

// The runs of a sequence that several CTAs shared, in CTA order: M = max m, out = sum acc 2^(m - M) / sum l 2^(m - M).  A CTA takes 32 columns of
// one sequence, a warp four of its heads at a time (16 bytes of a run's [column][heads] row), a lane a column.
// Bound: latency.  Many runs: their maxima and denominators come a lane each, beside the first eight runs' sums (one after the other: one sequence of 1024 keys, attention and
// merge, 24.6 us for 20.5, eight of 4096 40 for 34).  Few, as where sequences outnumber the SMs: every lane reads all of it at once, without shuffles (32 heads, 128 sequences of
// 200 keys, attention and merge, one after the other / a lane each / so 44.9 / 52.8 / 44.2 us, 96 of 4000 122 / 128 / 120).
template <int NH>
__global__ void __launch_bounds__(NH * 8) latent_decode_merge_kernel(const atoma_latent_attn_args a, const float *__restrict__ partial,
                                                                     const float *__restrict__ partial_ml, const int *__restrict__ prefix, int grid) {
    pdl_launch_dependents();
    pdl_wait();
    const int H = static_cast<int>(a.H), R = static_cast<int>(a.R), Rv = a.out_cols > 0 ? static_cast<int>(a.out_cols) : R, B = static_cast<int>(a.B);
    const int b = blockIdx.y, col = blockIdx.x * 32 + (threadIdx.x & 31), h0 = (threadIdx.x >> 5) * 4;
    const int units = prefix[B], ncta = min(grid, units), first = prefix[b], last = prefix[b + 1] - 1;
    if (last < first) return;
    const int c0 = ld_owner(units, first, ncta), c1 = ld_owner(units, last, ncta);
    if (c0 == c1 || h0 >= H) return;   // whole warps
    const int lane = threadIdx.x & 31, runs = c1 - c0 + 1;
    const float *sums = partial + (static_cast<int64_t>(b + c0) * Rv + col) * NH + h0;
    const int64_t pitch = static_cast<int64_t>(Rv) * NH;
    auto of_run = [&](int r) -> const float * { return partial_ml + (static_cast<int64_t>(b + c0 + min(r, runs - 1)) * NH + h0) * 2; };
    float M[4], den[4], num[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) M[i] = -INFINITY, den[i] = num[i] = 0.f;
    auto highest = [&](const float4 &x, const float4 &y) { M[0] = fmaxf(M[0], x.x), M[1] = fmaxf(M[1], x.z), M[2] = fmaxf(M[2], y.x), M[3] = fmaxf(M[3], y.z); };
    auto factors = [&](const float4 &x, const float4 &y, float (&f)[4], float (&l)[4]) {
        const float m[4] = {x.x, x.z, y.x, y.z};
        l[0] = x.y, l[1] = x.w, l[2] = y.y, l[3] = y.w;
#pragma unroll
        for (int i = 0; i < 4; ++i) f[i] = exp2f(m[i] - (M[i] == -INFINITY ? 0.f : M[i]));
    };
    constexpr int kFew = 4, kAhead = 8;
    if (runs <= kFew) {   // every lane reads all of it at once
        float4 v[kFew], x[kFew], y[kFew];
#pragma unroll
        for (int k = 0; k < kFew; ++k)
            if (k < runs) {
                x[k] = *reinterpret_cast<const float4 *>(of_run(k)), y[k] = *reinterpret_cast<const float4 *>(of_run(k) + 4);
                v[k] = *reinterpret_cast<const float4 *>(sums + k * pitch);
            }
#pragma unroll
        for (int k = 0; k < kFew; ++k)
            if (k < runs) highest(x[k], y[k]);
#pragma unroll
        for (int k = 0; k < kFew; ++k)
            if (k < runs) {
                const float xs[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
                float f[4], l[4];
                factors(x[k], y[k], f, l);
#pragma unroll
                for (int i = 0; i < 4; ++i) den[i] = fmaf(l[i], f[i], den[i]), num[i] = fmaf(xs[i], f[i], num[i]);
            }
    } else {
        // Lane j holds run c + j's maxima and denominators of the warp's four heads; the sums' first pieces are under way meanwhile.
        float4 v[kAhead];
#pragma unroll
        for (int k = 0; k < kAhead; ++k)
            if (k < runs) v[k] = *reinterpret_cast<const float4 *>(sums + k * pitch);
        for (int r = lane; r - lane < runs; r += 32) highest(*reinterpret_cast<const float4 *>(of_run(r)), *reinterpret_cast<const float4 *>(of_run(r) + 4));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int i = 0; i < 4; ++i) M[i] = fmaxf(M[i], __shfl_xor_sync(0xffffffffu, M[i], o));
        for (int r0 = 0; r0 < runs; r0 += 32) {
            float f[4], l[4];
            factors(*reinterpret_cast<const float4 *>(of_run(r0 + lane)), *reinterpret_cast<const float4 *>(of_run(r0 + lane) + 4), f, l);
            for (int k0 = 0; k0 < 32 && r0 + k0 < runs; k0 += kAhead) {
                float4 next[kAhead];
#pragma unroll
                for (int k = 0; k < kAhead; ++k)
                    if (r0 + k0 + kAhead + k < runs) next[k] = *reinterpret_cast<const float4 *>(sums + (r0 + k0 + kAhead + k) * pitch);
#pragma unroll
                for (int k = 0; k < kAhead; ++k) {
                    const float xs[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float fr = __shfl_sync(0xffffffffu, f[i], k0 + k), lr = __shfl_sync(0xffffffffu, l[i], k0 + k);
                        if (r0 + k0 + k < runs) {
                            den[i] = fmaf(lr, fr, den[i]);
                            num[i] = fmaf(xs[i], fr, num[i]);
                        }
                    }
                    v[k] = next[k];
                }
            }
        }
    }
    float *out = a.out + (static_cast<int64_t>(a.query_start[b]) * H + h0) * R + col;
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (h0 + i < H) out[i * R] = den[i] == 0.f ? 0.f : num[i] / den[i];   // a NaN sum stays one
}

size_t ld_smem(int nh, int64_t R, int64_t B) {
    return 1024 + static_cast<size_t>(kLdStages) * kLdKeys * R * 2 + (R / 64) * nh * 128 + 2 * nh * 128 + kLdKeys * (nh + 1) * 4 + (B + 1) * 4;
}

}  // namespace

// Decoded tokens only (one token per sequence, or none), up to 32 heads, rows of 64 ... 576 bfloat16 entries of which a multiple of 128 are summed.
bool hyb_latent_decode_ok(const atoma_latent_attn_args &a) {
    const int64_t rv = a.out_cols > 0 ? a.out_cols : a.R;
    auto al = [](const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    return a.dtype == ATOMA_DTYPE_BF16 && a.max_query_len == 1 && a.query_start && a.H <= 32 && a.B <= kLdMaxSeqs && a.R % 64 == 0 && a.R >= 128 && a.R <= 576 &&
           rv % 128 == 0 && rv <= 512 && al(a.latent_cache) && al(a.q_lat) && al(a.out) && a.max_blocks * a.block_size < (1ll << 30) && a.block_size % kLdGroup == 0 &&
           current_device_info().cc_major == 10;
}

// Where this kernel is the faster one, by the longest sequence's tiles.  A CTA pays some 8 us for a sequence's queries and sums whatever it reads, and holds one
// sequence at a time, so many sequences want several tiles each; and few sequences of narrow rows are cut into so many runs that their merge
// takes longer than the tiles.  Warp-level kernels / this one, us, 32 heads of 576: 96 sequences of 64, 128, 192 keys 17 / 19, 26 / 31, 35 / 33; 32 of 384
// and 4096 33 / 28 and 196 / 52; one of 128, 1024, 8192 keys 26 / 15, 35 / 21, 82 / 80.  8 heads of 128: 256 of 192 and 384 keys 19 / 22 and 34 / 27; one of 1024, 2048
// and 8192 keys 16 / 14, 18 / 20, 29 / 56, four of 8192 32 / 25.
bool hyb_latent_decode_better(const atoma_latent_attn_args &a) {
    int64_t span = a.max_seq_len > 0 ? a.max_seq_len : a.max_blocks * a.block_size;
    if (a.window > 0) span = std::min<int64_t>(span, a.window);
    const int64_t tiles = (span + kLdKeys - 1) / kLdKeys;
    return tiles >= 2 + a.B / 96 && (tiles <= a.R / 8 || 2 * a.B * tiles >= 5 * current_device_info().sm_count);
}

// `taken`: false where there is no workspace for the runs' sums (the caller's other kernels may need none).
bool hyb_latent_decode(const atoma_latent_attn_args &a, cudaStream_t stream, bool &taken) {
    taken = true;
    const int nh = a.H <= 16 ? 16 : 32;
    const int64_t span = a.max_seq_len > 0 ? a.max_seq_len : a.max_blocks * a.block_size;
    const int grid = static_cast<int>(std::min<int64_t>(current_device_info().sm_count, a.B * ((span + kLdKeys - 1) / kLdKeys)));
    const int64_t rv = a.out_cols > 0 ? a.out_cols : a.R, slots = a.B + grid;
    const size_t n_acc = static_cast<size_t>(slots) * nh * rv, n_ml = static_cast<size_t>(slots) * nh * 2;
    float *ws = static_cast<float *>(try_workspace(stream, (n_acc + n_ml + a.B + 1) * 4, kWorkspaceHybridAttn));
    if (!ws) return taken = false;
    float *ml = ws + n_acc;
    int *prefix = reinterpret_cast<int *>(ml + n_ml);
    const size_t smem = ld_smem(nh, a.R, a.B);
    CUtensorMap map;
    EncodeTiledFn enc = get_encode_tiled();
    if (!enc) return false;
    const cuuint64_t dims[3] = {64, 1ull << 30, static_cast<cuuint64_t>(a.R / 64)};   // how many rows the cache has is not known here: slots are the caller's
    const cuuint64_t strides[2] = {static_cast<cuuint64_t>(a.R) * 2, 128};
    const cuuint32_t box[3] = {64, kLdGroup, static_cast<cuuint32_t>(a.R / 64)}, estr[3] = {1, 1, 1};
    const CUresult r = enc(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void *>(a.latent_cache), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_status(kErrDriver, "latent_decode_kernel: cuTensorMapEncodeTiled failed (CUresult %d)", static_cast<int>(r));
        return false;
    }
    auto kernel = nh == 16 ? latent_decode_kernel<16> : latent_decode_kernel<32>;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 225 * 1024);
    if (e != cudaSuccess) {
        set_status(static_cast<int>(e), "latent_decode_kernel: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
        return false;
    }
    if (!hybrid::launched(launch_ex(kernel, dim3(std::max(grid, 1)), dim3(kLdThreads), smem, stream, map, a, ws, ml, prefix, late_word()), "latent_decode_kernel")) return false;
    const dim3 mgrid(static_cast<unsigned>(rv / 32), static_cast<unsigned>(a.B));
    return hybrid::launched(launch_ex(nh == 16 ? latent_decode_merge_kernel<16> : latent_decode_merge_kernel<32>, mgrid, dim3(nh * 8), 0, stream, a,
                                      static_cast<const float *>(ws), static_cast<const float *>(ml), static_cast<const int *>(prefix), std::max(grid, 1)),
                            "latent_decode_merge_kernel");
}

}  // namespace atoma

extern "C" int atoma_latent_decode_timeouts(void) {
    unsigned int n = 0;
    if (cudaMemcpyFromSymbol(&n, atoma::g_latent_late, sizeof(n)) != cudaSuccess) return -1;
    return static_cast<int>(n);
}
