// Prompt-sized products on CTA pairs (tcgen05 cta_group::2):  y[t, n] = sum_k x[t, k] w[n, k]  for many rows t, plain or with a
// gated activation of two products (gate row n, up row n) in the epilogue; dense, or grouped by expert.
//
// What bounds it: the tensor pipe, behind it the shared-memory and L2 bandwidth that feed it.  One SM multiplies 128 x N x 16 in N / 2
// cycles and reads its operands from shared memory at 128 bytes a cycle, so a lone CTA's 128 x 256 tile (4 + 8 KiB a product) starves the
// pipe; a pair shares one 256 x N product, each CTA holding 128 weight rows (M) and HALF of the N token rows, 4 + 4 KiB a product, and
// L2 hands out 2/3 of the bytes.  The weights are the M operand because tokens come ragged: N may be any multiple of 32, so a chunk of
// tokens is cut to what there is (an expert's 375 rows are two chunks of 192, not three tiles of 128 or two of 256).
//
// Work: persistent pairs (grid = SMs), tile = (256 weight rows or 128 gate / up pairs) x (a chunk of up to 256 tokens), whole K.
// Per CTA: warp 0 loads (TMA, 128-byte swizzle, three to nine stages in 192 KiB; completion is counted on the pair's first CTA) the weights and the last warp the
// tokens, warp 1 of the
// pair's first CTA issues the products, warps 2-9 empty the accumulator: two of 256 columns fill tensor memory, so a tile's
// epilogue runs under the next tile's products.  An epilogue thread owns a weight row (TMEM lane) and sees tokens in columns; four lanes
// turn 4 x 4 blocks with shuffles and store 8 bytes per token.  With the activation, gate and up rows alternate in the operand
// (a 3-D TMA box writes them so), and a lane pair trades them with one shuffle.
//
// Measured on a B200 (us, L2 flushed; one-CTA stream-K kernel / this one): 2999 x 4096 x 14336: 394 / 249 (1415 TFLOP/s, 0.85 of the measured
// peak), 8192 x 4096 x 4096: 257 / 173 (1590), 1024 x 4096 x 4096: 62 / 38, 256 x 2048 x 8192: 71 / 32; gate_up with silu, 2999 tokens of
// 4096 to 2 x 14336: 24 launches of 128 tokens 1400 / 480.
//
// Every wait is bounded: one that runs out raises a flag, the CTA's other roles stop waiting, the loads' warp waits (again with a bound)
// for its copies, tensor memory is freed, a counter is raised (atoma_gemm_pair_timeouts) and the host is told (atoma_kernel_timeouts).
#include "common.cuh"
#include "gemm_pair.h"
#include "hybrid_common.cuh"

#include <algorithm>
#include <cstring>
#include <vector>

namespace atoma {
namespace {

constexpr int kGpEpiWarps = 8;
constexpr int kGpThreads = 32 * (3 + kGpEpiWarps);   // weights' loads, products, epilogue, tokens' loads
constexpr int kGpRows = 128;                 // weight rows per CTA
constexpr int kGpK = 64;                     // a k block: 128 bytes, one swizzle row
constexpr int kGpMaxStages = 10;
constexpr int kGpMaxN = 256;
constexpr int kGpABytes = kGpRows * 128, kGpRing = 12 * kGpABytes;   // B: half a chunk, at most 128 rows; six stages of full chunks
constexpr int kGpWidths = kGpMaxN / 32;
constexpr int kGpTries = 1 << 18;            // milliseconds at least (a try may also suspend the thread for a hardware-chosen time)
constexpr int kGpChunkGroup = 16;            // dense raster: token chunks that share the weight tiles of a wave

__device__ unsigned int g_pair_late;

struct XMaps {
    CUtensorMap m[kGpWidths];                // box rows 16, 32, ... 128: half a chunk of 32, 64, ... 256 tokens
};

__device__ __forceinline__ void gp_wait(uint64_t *bar, uint32_t parity, volatile int *late) {
#pragma unroll 1
    for (int i = 0; !mbar_try_wait(bar, parity);) {
        if (*late) break;
        if (++i == kGpTries) {
            *late = 1;
            break;
        }
    }
}
__device__ __forceinline__ void gp_tma_5d(uint32_t dst, const CUtensorMap *map, uint32_t cluster_bar, int c0, int c1, int c2, int c3, int c4, uint64_t policy) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2.L2::cache_hint"
        " [%0], [%1, {%3, %4, %5, %6, %7}], [%2], %8;" ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(cluster_bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3),
        "r"(c4), "l"(policy)
        : "memory");
}
__device__ __forceinline__ void gp_tma_3d(uint32_t dst, const CUtensorMap *map, uint32_t cluster_bar, int c0, int c1, int c2, uint64_t policy) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2.L2::cache_hint"
        " [%0], [%1, {%3, %4, %5}], [%2], %6;" ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(cluster_bar), "r"(c0), "r"(c1), "r"(c2), "l"(policy)
        : "memory");
}
__device__ __forceinline__ void gp_mma(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// arrives at the same barrier of both CTAs of the pair once all products issued so far have completed
__device__ __forceinline__ void gp_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
                 "h"(static_cast<unsigned short>(3))
                 : "memory");
}
__device__ __forceinline__ void gp_arrive_cluster(uint32_t cluster_bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}

struct GpTile {
    int w_row;       // first weight row (output column) of the pair's tile within its expert
    int expert;
    int t0, t_end;   // token rows: first, one past the last that counts
    int width;       // tokens of the product, a multiple of 32
};

template <bool GLU>
__device__ __forceinline__ GpTile gp_tile(const GemmPairArgs &a, int tile) {
    constexpr int kOut = GLU ? kGpRows : 2 * kGpRows;   // output columns of a tile
    GpTile r;
    if (a.plan) {
        const int c = tile / a.w_tiles;
        const int4 pc = reinterpret_cast<const int4 *>(a.plan)[1 + c];   // expert, first row, rows, width
        r.w_row = (tile - c * a.w_tiles) * kOut;
        r.expert = pc.x;
        r.t0 = pc.y;
        r.t_end = pc.y + pc.z;
        r.width = pc.w;
    } else {
        const int per_group = kGpChunkGroup * a.w_tiles;
        const int g = tile / per_group, in = tile - g * per_group;
        const int gc = min(kGpChunkGroup, a.chunks - g * kGpChunkGroup);
        const int w = in / gc, c = g * kGpChunkGroup + in - w * gc;
        r.w_row = w * kOut;
        r.expert = 0;
        r.t0 = c * a.width;
        r.t_end = min(a.T, r.t0 + a.width);
        r.width = a.width;
    }
    return r;
}

// Four lanes that differ in two lane bits (M, 2 M) hold 4 values each: lane q of the four gets value q of all four, in lane order.
template <int M>
__device__ __forceinline__ void gp_turn4(float (&v)[4], int lane) {
    const bool hi = lane & M;
    float s0 = hi ? v[0] : v[1], s1 = hi ? v[2] : v[3];
    s0 = __shfl_xor_sync(0xffffffffu, s0, M);
    s1 = __shfl_xor_sync(0xffffffffu, s1, M);
    float a0 = hi ? s0 : v[0], a1 = hi ? v[1] : s0, b0 = hi ? s1 : v[2], b1 = hi ? v[3] : s1;   // (a0, a1): value hi of the lane pair; (b0, b1): value 2 + hi
    const bool up = lane & (2 * M);
    float t0 = up ? a0 : b0, t1 = up ? a1 : b1;
    t0 = __shfl_xor_sync(0xffffffffu, t0, 2 * M);
    t1 = __shfl_xor_sync(0xffffffffu, t1, 2 * M);
    v[0] = up ? t0 : a0;
    v[1] = up ? t1 : a1;
    v[2] = up ? b0 : t0;
    v[3] = up ? b1 : t1;
}

// The gated activation, each operation within 2 ulp.
__device__ __forceinline__ float gp_act(const GemmPairArgs &a, float g, float u, float bias_g, float bias_u) {
    if (a.act == 1) return fmaxf(g, 0.f) * u;
    if (a.act == 2) return hybrid::glu_act(g, 2) * u;
    float alpha = 1.f;
    if (a.act == kPairClamped) {
        g += bias_g;
        u += bias_u;
        if (a.limit > 0.f) {
            g = fminf(g, a.limit);
            u = fminf(fmaxf(u, -a.limit), a.limit);
        }
        u += a.shift;
        alpha = a.alpha;
    }
    return over_one_plus(g, expf(-alpha * g)) * u;
}

template <typename T, bool GLU>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kGpThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ XMaps map_x, const GemmPairArgs a) {
    extern __shared__ unsigned char smem_dyn[];
    unsigned char *tiles = smem_dyn + ((1024u - (smem_u32(smem_dyn) & 1023u)) & 1023u);
    __shared__ __align__(8) uint64_t full[kGpMaxStages], empty[kGpMaxStages], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_base_smem;
    __shared__ int late_s;
    volatile int *late = &late_s;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_ctarank();
    const int stages = a.stages, stage_bytes = a.stage_bytes;
    if (tid == 0) {
        late_s = 0;
        for (int i = 0; i < stages; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&acc_full[i], 1);
            mbar_init(&acc_empty[i], 2 * kGpEpiWarps);   // both CTAs' epilogue warps
        }
        fence_mbar_init();
        tma_prefetch_desc(&map_w);
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_smem)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before_sync();
    __syncthreads();
    cluster_arrive_release();
    cluster_wait_acquire();
    tc_fence_after_sync();
    const uint32_t tmem_base = tmem_base_smem;
    pdl_launch_dependents();
    pdl_wait();

    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const int n_tiles = a.plan ? a.plan[0] * a.w_tiles : a.tiles;
    const int nkb = (a.K + kGpK - 1) / kGpK, kbs = a.kbs;
    if (warp == 0 || warp == 2 + kGpEpiWarps) {
        // ============================ loads: weights (warp 0), tokens (last warp) ============================
        int it = 0, s = 0;
        uint32_t phase = 0;
        const uint64_t w_policy = a.w_once ? kL2EvictFirst : kL2EvictNormal;
        for (int tile = pair; tile < n_tiles; tile += pairs) {
            const GpTile t = gp_tile<GLU>(a, tile);
            const int half = t.width / 2;
            const CUtensorMap *mx = &map_x.m[t.width / 32 - 1];
            const int w_row = t.w_row + static_cast<int>(rank) * (GLU ? kGpRows / 2 : kGpRows);
            const int x_row = t.t0 + static_cast<int>(rank) * half;
            const uint32_t bytes = 2u * kbs * (kGpABytes + half * 128);
            for (int kb = 0; kb < nkb; kb += kbs, ++it) {
                gp_wait(&empty[s], phase ^ 1, late);
                if (__any_sync(0xffffffffu, *late != 0)) break;
                if (elect_one_sync()) {
                    const uint32_t st = smem_u32(tiles + s * stage_bytes), bar = mapa_shared(smem_u32(&full[s]), 0);
                    // a map of whole 64-wide k blocks counts blocks, a map of single columns (kbs 1, K not a multiple of 64) counts columns
                    const int k0 = a.k_blocked ? 0 : kb * kGpK, k1 = a.k_blocked ? kb : 0;
                    if (warp == 0) {
                        if (rank == 0) mbar_arrive_expect_tx(&full[s], bytes);
                        gp_tma_5d(st, &map_w, bar, k0, 0, w_row, k1, t.expert, w_policy);
                    } else {
                        gp_tma_3d(st + kbs * kGpABytes, mx, bar, k0, x_row, k1, kL2EvictNormal);
                    }
                }
                __syncwarp();
                if (++s == stages) s = 0, phase ^= 1;
            }
            if (__any_sync(0xffffffffu, *late != 0)) break;
        }
        // whatever happened to the other roles, the pair's copies have landed before the pair leaves
        if (rank == 0)
            for (int i = max(0, it - stages); i < it; ++i)
                for (int k = 0; k < kGpTries && !mbar_try_wait(&full[i % stages], (i / stages) & 1); ++k) {
                }
    } else if (warp == 1 && rank == 0) {
        // ============================ products ============================
        int n = 0, s = 0;
        uint32_t phase = 0;
        for (int tile = pair; tile < n_tiles; tile += pairs, ++n) {
            const GpTile t = gp_tile<GLU>(a, tile);
            const uint32_t idesc = umma_idesc_f16(256, t.width, a.is_bf16 != 0);
            const uint32_t tmem_d = tmem_base + (n & 1) * kGpMaxN;
            gp_wait(&acc_empty[n & 1], ((n >> 1) & 1) ^ 1, late);
            tc_fence_after_sync();
            for (int kb = 0; kb < nkb; kb += kbs) {
                gp_wait(&full[s], phase, late);
                tc_fence_after_sync();
                if (elect_one_sync()) {
                    uint32_t wa = smem_u32(tiles + s * stage_bytes), xa = wa + kbs * kGpABytes;
                    for (int b = 0; b < kbs && kb + b < nkb; ++b, wa += kGpABytes, xa += t.width * 64) {
                        const uint64_t da = umma_desc_k_sw128(wa), db = umma_desc_k_sw128(xa);
#pragma unroll
                        for (int k = 0; k < kGpK / 16; ++k) gp_mma(tmem_d, da + 2 * k, db + 2 * k, idesc, (kb | b | k) != 0 ? 1u : 0u);
                    }
                    gp_commit(&empty[s]);
                    if (kb + kbs >= nkb) gp_commit(&acc_full[n & 1]);
                }
                __syncwarp();
                if (++s == stages) s = 0, phase ^= 1;
            }
        }
    } else if (warp >= 2) {
        // ============================ epilogue ============================
        const int quad = warp & 3;                         // TMEM lanes this warp may read
        const int side = (warp - 2) >> 2;                  // two warps per quarter take the 32-token columns in turn
        const uint32_t taddr0 = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
        T *y = static_cast<T *>(a.y);
        const bool vec = a.ldy % 4 == 0 && (reinterpret_cast<uintptr_t>(a.y) & 7) == 0 && a.N % 4 == 0;
        const int row = quad * 32 + lane;   // accumulator row of this thread
        int n = 0;
        for (int tile = pair; tile < n_tiles; tile += pairs, ++n) {
            const GpTile t = gp_tile<GLU>(a, tile);
            float weight[GLU ? 1 : kGpWidths / 2];   // of token c + lane: fetched while the products run
            if constexpr (!GLU) {
#pragma unroll
                for (int i = 0; i < kGpWidths / 2; ++i) {
                    weight[i] = 1.f;
                    const int tok = t.t0 + 64 * i + 32 * side + lane;
                    if (a.out_weight && tok < t.t_end) {
                        const int pr = a.row_pair[tok];
                        weight[i] = pr >= 0 ? a.out_weight[pr] : 0.f;
                    }
                }
            }
            gp_wait(&acc_full[n & 1], (n >> 1) & 1, late);
            tc_fence_after_sync();
            const uint32_t taddr = taddr0 + (n & 1) * kGpMaxN;
            // the four output columns this thread stores (after the turn), and whether it is gate (even) or up (odd)
            const int col = GLU ? t.w_row + static_cast<int>(rank) * 64 + (quad * 32 + (lane & 24)) / 2 : t.w_row + static_cast<int>(rank) * kGpRows + (row & ~3);
            float bias_g = 0.f, bias_u = 0.f;
            if constexpr (GLU) {
                const int j = t.w_row + static_cast<int>(rank) * 64 + row / 2;
                if (a.bias && j < a.N) {
                    bias_g = a.bias[j];
                    bias_u = a.bias[a.N + j];
                }
            }
#pragma unroll (GLU ? 1 : kGpWidths / 2)
            for (int ci = 0; ci < kGpWidths / 2; ++ci) {
                const int c = 64 * ci + 32 * side;
                if (c >= t.width || t.t0 + c >= t.t_end) break;
                uint32_t v[32];
                tmem_ld_32x32b_x32(taddr + c, v);
                tmem_ld_wait();
                if constexpr (GLU) {
#pragma unroll
                    for (int g = 0; g < 4; ++g) {   // 8 tokens
                        float o[4];
                        const bool up = lane & 1;
#pragma unroll
                        for (int m = 0; m < 4; ++m) {
                            const float v0 = __uint_as_float(v[8 * g + 2 * m]), v1 = __uint_as_float(v[8 * g + 2 * m + 1]);
                            const float got = __shfl_xor_sync(0xffffffffu, up ? v0 : v1, 1);
                            float gate = up ? got : v0, upv = up ? v1 : got;   // of token 2 m + (lane & 1)
                            if (a.round_products) {
                                gate = hybrid::to_f(hybrid::from_f<T>(gate));
                                upv = hybrid::to_f(hybrid::from_f<T>(upv));
                            }
                            o[m] = gp_act(a, gate, upv, bias_g, bias_u);
                        }
                        gp_turn4<2>(o, lane);   // this thread: columns col .. col + 3 of token 2 ((lane >> 1) & 3) + (lane & 1)
                        const int tok = t.t0 + c + 8 * g + 2 * ((lane >> 1) & 3) + (lane & 1);
                        if (tok < t.t_end && col < a.N) {
                            T *yp = y + static_cast<int64_t>(tok) * a.ldy + col;
                            if (vec) {
                                *reinterpret_cast<uint2 *>(yp) = make_uint2(pack2<T>(o[0], o[1]), pack2<T>(o[2], o[3]));
                            } else {
                                for (int i = 0; i < 4 && col + i < a.N; ++i) yp[i] = hybrid::from_f<T>(o[i]);
                            }
                        }
                    }
                } else {
#pragma unroll
                    for (int g = 0; g < 8; ++g) {   // 4 tokens
                        float o[4];
#pragma unroll
                        for (int m = 0; m < 4; ++m) o[m] = __uint_as_float(v[4 * g + m]);
                        gp_turn4<1>(o, lane);
                        const int tok = t.t0 + c + 4 * g + (lane & 3);
                        if (a.out_weight) {
                            const float ow = __shfl_sync(0xffffffffu, weight[ci], 4 * g + (lane & 3));
#pragma unroll
                            for (int m = 0; m < 4; ++m) o[m] *= ow;
                        }
                        if (tok < t.t_end && col < a.N) {
                            T *yp = y + static_cast<int64_t>(tok) * a.ldy + col;
                            if (vec) {
                                *reinterpret_cast<uint2 *>(yp) = make_uint2(pack2<T>(o[0], o[1]), pack2<T>(o[2], o[3]));
                            } else {
                                for (int i = 0; i < 4 && col + i < a.N; ++i) yp[i] = hybrid::from_f<T>(o[i]);
                            }
                        }
                    }
                }
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) gp_arrive_cluster(mapa_shared(smem_u32(&acc_empty[n & 1]), 0));
        }
    }
    // both CTAs stay until the pair's products, copies and remote arrivals are done
    tc_fence_before_sync();
    __syncthreads();
    cluster_arrive_release();
    cluster_wait_acquire();
    if (warp == 1) {
        tc_fence_after_sync();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
    }
    if (tid == 0 && *late) {
        atomicAdd(&g_pair_late, 1u);
        if (a.late) *reinterpret_cast<volatile unsigned int *>(a.late) = 1;
    }
}

// ---------------------------------------------------------------------------------------------
struct GpMapKey {
    const void *ptr;
    uint64_t dims[5], strides[4];
    uint32_t box[5], rank, bf16;
    bool operator==(const GpMapKey &o) const { return std::memcmp(this, &o, sizeof(GpMapKey)) == 0; }
};
struct GpMapEntry {
    GpMapKey key;
    CUtensorMap map;
};

bool gp_map(CUtensorMap *out, const GpMapKey &key) {
    static thread_local std::vector<GpMapEntry> cache;
    for (const GpMapEntry &e : cache)
        if (e.key == key) {
            *out = e.map;
            return true;
        }
    EncodeTiledFn enc = get_encode_tiled();
    if (!enc) return false;
    cuuint64_t dims[5], strides[4];
    cuuint32_t box[5], estr[5] = {1, 1, 1, 1, 1};
    for (int i = 0; i < 5; ++i) dims[i] = key.dims[i], box[i] = key.box[i];
    for (int i = 0; i < 4; ++i) strides[i] = key.strides[i];
    const CUresult r = enc(out, key.bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, key.rank, const_cast<void *>(key.ptr), dims,
                           strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_status(kErrDriver, "gemm_pair: cuTensorMapEncodeTiled failed (CUresult %d)", static_cast<int>(r));
        return false;
    }
    if (cache.size() >= 256) cache.clear();
    cache.push_back(GpMapEntry{key, *out});
    return true;
}

template <typename T, bool GLU>
bool gp_launch(const CUtensorMap &mw, const XMaps &mx, const GemmPairArgs &a, cudaStream_t stream) {
    constexpr int smem = kGpRing + 1024;
    static thread_local int attr_dev = -1;
    const DeviceInfo &di = current_device_info();
    if (attr_dev != di.ordinal) {
        const cudaError_t e = cudaFuncSetAttribute(gemm_pair_kernel<T, GLU>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) {
            set_status(static_cast<int>(e), "gemm_pair: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
            return false;
        }
        attr_dev = di.ordinal;
    }
    const int grid = 2 * std::min(di.sm_count / 2, std::max(1, a.tiles));
    return hybrid::launched(launch_ex(gemm_pair_kernel<T, GLU>, dim3(grid), dim3(kGpThreads), smem, stream, mw, mx, a), "gemm_pair_kernel");
}

}  // namespace

int gemm_pair_w_tiles(int64_t N, bool glu) {
    const int out = glu ? kGpRows : 2 * kGpRows;
    return static_cast<int>((N + out - 1) / out);
}

// The width whose waves of tiles take the least time.  A k block took (us, K = 2048 ... 14336, all pairs busy) 0.245 at 64 tokens, 0.25 at 96,
// 0.27 at 128, 0.33 at 160, 0.35 at 192, 0.40 at 224 and 0.43 at 256: wide chunks are the cheaper ones per token, narrow ones fill the
// pairs when there are few tiles; the last tile's epilogue costs about 0.01 us a token.  Over 6 weight shapes and 132 to 8192 tokens the choice is within 8 % of
// the best width but for one shape (10 %).
int gemm_pair_width(int64_t T, int64_t N, int64_t K, bool glu) {
    const int pairs = current_device_info().sm_count / 2;
    const int64_t w_tiles = gemm_pair_w_tiles(N, glu), kb = (K + kGpK - 1) / kGpK;
    int best = 0;
    double best_cost = 0;
    for (int width = kGpMaxN; width >= 32; width -= 32) {
        const int64_t tiles = w_tiles * ((T + width - 1) / width), waves = (tiles + pairs - 1) / pairs;
        const double block = width <= 128 ? 0.22 + 0.0004 * width : 0.19 + 0.00095 * width;
        const double cost = static_cast<double>(waves) * kb * block + 0.01 * width;
        if (best == 0 || cost < best_cost) best = width, best_cost = cost;
    }
    return best;
}

// w: `experts` x (glu: N gate rows, then N up rows; else N rows) of K, row stride ldw; x [rows, K], row stride ldx.  `a` arrives with the
// output, the activation and, when grouped, plan / tiles (an upper bound) filled in.
bool launch_gemm_pair(GemmPairArgs a, const void *x, const void *w, int64_t rows, int64_t N, int64_t K, int64_t ldx, int64_t ldw, int64_t experts, bool glu,
                      bool is_bf16, cudaStream_t stream) {
    a.late = late_word();
    a.N = static_cast<int>(N);
    a.K = static_cast<int>(K);
    a.is_bf16 = is_bf16 ? 1 : 0;
    a.w_tiles = gemm_pair_w_tiles(N, glu);
    // Narrow chunks take stages of two k blocks: a warp starts only about 6 copies a microsecond whatever their size, and a product of 64
    // or 128 tokens needs its next block after 0.07 or 0.14 us (measured per block at width 64, one loading warp and single blocks 0.30 us,
    // two warps and double blocks 0.18).  Wide chunks keep six single blocks in flight (K = 14336, 1024 tokens: 87 us, double blocks 92).
    // A map that counts whole blocks would read the next row behind a K that is not a multiple of 64, so such a K takes single blocks
    // and the map's zero fill.
    a.k_blocked = K % kGpK == 0 ? 1 : 0;
    const int widest = a.plan ? a.max_width : a.width;
    a.kbs = a.k_blocked && K >= 2 * kGpK && widest <= 128 ? 2 : 1;
    if (!a.plan) {
        a.T = static_cast<int>(rows);
        a.tiles = a.w_tiles * a.chunks;
    }
    a.stage_bytes = a.kbs * (kGpABytes + widest * 64);   // narrow chunks: more stages (operands stay 1024-byte aligned)
    a.stages = std::min(kGpMaxStages, kGpRing / a.stage_bytes);
    const uint64_t es = 2, row = static_cast<uint64_t>(ldw) * es, kblocks = static_cast<uint64_t>((K + kGpK - 1) / kGpK);
    GpMapKey kw;
    std::memset(&kw, 0, sizeof(kw));
    kw.ptr = w, kw.rank = 5, kw.bf16 = a.is_bf16;
    kw.dims[0] = a.k_blocked ? kGpK : K, kw.dims[1] = glu ? 2 : 1, kw.dims[2] = N, kw.dims[3] = a.k_blocked ? kblocks : 1, kw.dims[4] = experts;
    kw.strides[0] = row * N, kw.strides[1] = row, kw.strides[2] = kGpK * es, kw.strides[3] = row * N * (glu ? 2 : 1);
    kw.box[0] = kGpK, kw.box[1] = glu ? 2 : 1, kw.box[2] = glu ? kGpRows / 2 : kGpRows, kw.box[3] = a.kbs, kw.box[4] = 1;
    CUtensorMap mw;
    if (!gp_map(&mw, kw)) return false;
    XMaps mx;
    std::memset(&mx, 0, sizeof(mx));
    for (int i = 0; i < kGpWidths; ++i) {
        if (a.plan ? 32 * (i + 1) > a.max_width : 32 * (i + 1) != a.width) continue;
        GpMapKey kx;
        std::memset(&kx, 0, sizeof(kx));
        kx.ptr = x, kx.rank = 3, kx.bf16 = a.is_bf16;
        kx.dims[0] = a.k_blocked ? kGpK : K, kx.dims[1] = rows, kx.dims[2] = a.k_blocked ? kblocks : 1, kx.dims[3] = kx.dims[4] = 1;
        kx.strides[0] = static_cast<uint64_t>(ldx) * es, kx.strides[1] = kGpK * es;
        kx.box[0] = kGpK, kx.box[1] = 16 * (i + 1), kx.box[2] = a.kbs, kx.box[3] = kx.box[4] = 1;
        if (!gp_map(&mx.m[i], kx)) return false;
    }
    if (is_bf16) return glu ? gp_launch<__nv_bfloat16, true>(mw, mx, a, stream) : gp_launch<__nv_bfloat16, false>(mw, mx, a, stream);
    if (glu) return gp_launch<__half, true>(mw, mx, a, stream);
    set_status(kErrUnsupported, "gemm_pair: float16 with the gated activation only");
    return false;
}

// Operands this path takes (strides in elements).
bool gemm_pair_ok(const void *x, const void *w, int64_t N, int64_t K, int64_t ldx, int64_t ldw) {
    auto al = [](const void *p) { return p && (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    return al(x) && al(w) && ldx % 8 == 0 && ldw % 8 == 0 && ldx >= K && ldw >= K && K >= kGpK && K < (1ll << 30) && N > 0 && N < (1ll << 30) &&
           current_device_info().cc_major == 10 && current_device_info().sm_count >= 2;
}

}  // namespace atoma

extern "C" int atoma_gemm_pair_timeouts(void) {
    unsigned int n = 0;
    if (cudaMemcpyFromSymbol(&n, atoma::g_pair_late, sizeof(n)) != cudaSuccess) return -1;
    return static_cast<int>(n);
}
