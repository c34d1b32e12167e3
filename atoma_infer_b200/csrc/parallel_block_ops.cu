// Operators of PARALLEL decoder blocks and their mixers — include/atoma_hybrid.h.
//
// A parallel block norms the residual stream once; the mixer and the feed-forward both read that row, each through a
// causal tap filter over time, and both results join the stream in one update (fused here with whatever precedes the next
// layer and with its input norm).  The mixers that need more than attention kernels:
//   - tap filters whose inputs before a portion come from a per-sequence history (the portion's last inputs replace it),
//   - matrix-state recurrences: state_scan.cu,
//   - rotary positions on queries, keys and values with the cache write, the turn-back of a head's sum, and the
//     latent-attention variants that keep one rotated key part beside the latent.
// Statistics, angles, decays, gates of the recurrences and the state are float32 whatever the activation format; every
// result is reduced in an order that depends on the token alone, never on the batch around it.
#include "common.cuh"
#include "hybrid_common.cuh"

#include "atoma_hybrid.h"

#include <algorithm>

namespace atoma {

extern int g_hybrid_debug;   // bit 1: general kernels only
bool hyb_head_project_ld(const void *, int64_t, int64_t, const void *, void *, int64_t, int64_t, int64_t, int64_t, int64_t, int64_t, int32_t,
                         uint32_t, cudaStream_t, const void * = nullptr, int64_t = 0);   // latent_attention.cu

namespace {

using namespace hybrid;

constexpr int kMaxTaps = 16;

// ---------------------------------------------------------------------------------------------
// residual update of a parallel block + what precedes the next layer + its input norm
// ---------------------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(kRowThreads) parallel_residual_norm_kernel(const atoma_parallel_residual_args a) {
    extern __shared__ float row[];
    __shared__ float red[32];
    pdl_launch_dependents();
    pdl_wait();
    const int64_t t = blockIdx.x;
    const int W = static_cast<int>(a.width);
    const T *ya = a.y_a ? static_cast<const T *>(a.y_a) + t * W : nullptr;
    const T *yb = a.y_b ? static_cast<const T *>(a.y_b) + t * W : nullptr;
    const T *yf = a.y_ff ? static_cast<const T *>(a.y_ff) + t * W : nullptr;
    float inv_a = 1.f, inv_b = 1.f;
    if (ya && a.norm_a) {
        float ss = 0.f;
        for (int c = threadIdx.x; c < W; c += blockDim.x) {
            const float v = to_f(ya[c]);
            ss = fmaf(v, v, ss);
        }
        inv_a = 1.0f / sqrtf(block_sum(ss, red) / static_cast<float>(W) + a.eps);
    }
    if (yb && a.norm_b) {
        float ss = 0.f;
        for (int c = threadIdx.x; c < W; c += blockDim.x) {
            const float v = to_f(yb[c]);
            ss = fmaf(v, v, ss);
        }
        inv_b = 1.0f / sqrtf(block_sum(ss, red) / static_cast<float>(W) + a.eps);
    }
    float *x = a.x + t * W;
    float ss = 0.f;
    for (int c = threadIdx.x; c < W; c += blockDim.x) {
        float m = 0.f;
        if (ya) m += a.norm_a ? to_f(ya[c]) * inv_a * a.norm_a[c] : to_f(ya[c]);
        if (yb) m += a.norm_b ? to_f(yb[c]) * inv_b * a.norm_b[c] : to_f(yb[c]);
        float v = x[c] + a.mix_scale * m;
        if (yf) v += to_f(yf[c]);
        if (a.trace) a.trace[t * W + c] = v;
        if (a.add_rows) v += a.add_rows[t * W + c];
        if (a.add_vec) v += a.add_vec[c];
        x[c] = v;
        row[c] = v;
        ss = fmaf(v, v, ss);
    }
    if (!a.w_next) return;
    const float inv = 1.0f / sqrtf(block_sum(ss, red) / static_cast<float>(W) + a.eps);
    T *h = static_cast<T *>(a.h) + t * W;
    for (int c = threadIdx.x; c < W; c += blockDim.x) h[c] = from_f<T>(row[c] * inv * (a.weight_offset + a.w_next[c]));
}

// ---------------------------------------------------------------------------------------------
// tap filters with carried inputs
// ---------------------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) tap_filter_kernel(const atoma_tap_filter_args a) {
    pdl_launch_dependents();
    pdl_wait();
    const int64_t t = blockIdx.y;
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int C = static_cast<int>(a.channels), taps = static_cast<int>(a.taps);
    if (c >= C) return;
    const int b = a.token_seq[t];
    const int i = static_cast<int>(t) - a.query_start[b];     // index inside the portion
    const int ctx = a.context_lens[b];
    const T *in = static_cast<const T *>(a.in);
    const float *hist = a.history ? a.history + static_cast<int64_t>(a.state_slots[b]) * a.history_stride : nullptr;
    const float ib = a.in_bias ? a.in_bias[c] : 0.f;
    const float cur = to_f(in[t * a.ld_in + c]) + ib;
    float f1 = a.bias1 ? a.bias1[c] : 0.f, f2 = 0.f;
    for (int j = 0; j + 1 < taps; ++j) {
        const int back = taps - 1 - j;
        float v = 0.f;
        if (i - back >= 0) v = to_f(in[(t - back) * a.ld_in + c]) + ib;
        else if (ctx + i - back >= 0 && hist) v = hist[static_cast<int64_t>(taps - 1 + i - back) * C + c];
        f1 = fmaf(a.w1[c * taps + j], v, f1);
        if (a.w2) f2 = fmaf(a.w2[c * taps + j], v, f2);
    }
    f1 = fmaf(a.w1[c * taps + taps - 1], cur, f1);
    if (a.residual) f1 += cur;
    if (a.act == 1) f1 = silu(f1);
    static_cast<T *>(a.out1)[t * a.ld_out + c] = from_f<T>(f1);
    if (a.w2) {
        f2 = fmaf(a.w2[c * taps + taps - 1], cur, f2);
        if (a.residual) f2 += cur;
        if (a.act == 1) f2 = silu(f2);
        static_cast<T *>(a.out2)[t * a.ld_out + c] = from_f<T>(f2);
    }
}

// The same filter for bfloat16 rows of 16-byte pieces: a thread owns 8 neighbouring channels and `run` consecutive tokens, keeps
// the filters' weights and the last TAPS - 1 inputs in registers, and slides that window from token to token; it is filled anew
// at the run's first token and wherever a portion starts (from the rows before, the sequence's carried inputs, or zeros).
// Per element the products are added in the order of the kernel above, so both give the same bits.
template <int TAPS>
__global__ void __launch_bounds__(128) tap_filter_vec_kernel(const atoma_tap_filter_args a, int run) {
    pdl_launch_dependents();
    pdl_wait();
    const int C = static_cast<int>(a.channels), T = static_cast<int>(a.T);
    const int c0 = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
    if (c0 >= C) return;
    const int t_first = blockIdx.y * run, t_end = min(T, t_first + run);
    const __nv_bfloat16 *in = static_cast<const __nv_bfloat16 *>(a.in);
    float w1[8][TAPS], w2[8][TAPS];
    {
        const float4 *p1 = reinterpret_cast<const float4 *>(a.w1 + static_cast<int64_t>(c0) * TAPS);
        const float4 *p2 = a.w2 ? reinterpret_cast<const float4 *>(a.w2 + static_cast<int64_t>(c0) * TAPS) : p1;
#pragma unroll
        for (int i = 0; i < 2 * TAPS; ++i) {
            const float4 x = p1[i], y = p2[i];
            const float xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                w1[(4 * i + e) / TAPS][(4 * i + e) % TAPS] = xs[e];
                w2[(4 * i + e) / TAPS][(4 * i + e) % TAPS] = ys[e];
            }
        }
    }
    float ib[8], ob[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        ib[e] = a.in_bias ? a.in_bias[c0 + e] : 0.f;
        ob[e] = a.bias1 ? a.bias1[c0 + e] : 0.f;
    }
    auto row8 = [&](int64_t t, float *v) {
        const uint4 r = *reinterpret_cast<const uint4 *>(in + t * a.ld_in + c0);
        const uint32_t u[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            v[2 * e] = __uint_as_float(u[e] << 16) + ib[2 * e];
            v[2 * e + 1] = __uint_as_float(u[e] & 0xffff0000u) + ib[2 * e + 1];
        }
    };
    float win[TAPS > 1 ? TAPS - 1 : 1][8];                     // win[k]: the input TAPS - 1 - k tokens back
    for (int t = t_first; t < t_end; ++t) {
        const int b = a.token_seq[t];
        const int i = t - a.query_start[b];
        if (TAPS > 1 && (t == t_first || i == 0)) {
            const int ctx = a.context_lens[b];
            const float *hist = a.history ? a.history + static_cast<int64_t>(a.state_slots[b]) * a.history_stride : nullptr;
#pragma unroll
            for (int k = 0; k < TAPS - 1; ++k) {
                const int back = TAPS - 1 - k;
                if (i - back >= 0) {
                    row8(t - back, win[k]);
                } else if (ctx + i - back >= 0 && hist) {
#pragma unroll
                    for (int e = 0; e < 8; ++e) win[k][e] = hist[static_cast<int64_t>(TAPS - 1 + i - back) * C + c0 + e];
                } else {
#pragma unroll
                    for (int e = 0; e < 8; ++e) win[k][e] = 0.f;
                }
            }
        }
        float cur[8], f1[8], f2[8];
        row8(t, cur);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            float x = ob[e], y = 0.f;
#pragma unroll
            for (int k = 0; k < TAPS - 1; ++k) {
                x = fmaf(w1[e][k], win[k][e], x);
                y = fmaf(w2[e][k], win[k][e], y);
            }
            x = fmaf(w1[e][TAPS - 1], cur[e], x);
            y = fmaf(w2[e][TAPS - 1], cur[e], y);
            if (a.residual) {
                x += cur[e];
                y += cur[e];
            }
            if (a.act == 1) {
                x = silu(x);
                y = silu(y);
            }
            f1[e] = x;
            f2[e] = y;
        }
        uint4 o;
        o.x = pack2<__nv_bfloat16>(f1[0], f1[1]);
        o.y = pack2<__nv_bfloat16>(f1[2], f1[3]);
        o.z = pack2<__nv_bfloat16>(f1[4], f1[5]);
        o.w = pack2<__nv_bfloat16>(f1[6], f1[7]);
        *reinterpret_cast<uint4 *>(static_cast<__nv_bfloat16 *>(a.out1) + static_cast<int64_t>(t) * a.ld_out + c0) = o;
        if (a.w2) {
            o.x = pack2<__nv_bfloat16>(f2[0], f2[1]);
            o.y = pack2<__nv_bfloat16>(f2[2], f2[3]);
            o.z = pack2<__nv_bfloat16>(f2[4], f2[5]);
            o.w = pack2<__nv_bfloat16>(f2[6], f2[7]);
            *reinterpret_cast<uint4 *>(static_cast<__nv_bfloat16 *>(a.out2) + static_cast<int64_t>(t) * a.ld_out + c0) = o;
        }
#pragma unroll
        for (int k = 0; k + 1 < TAPS - 1; ++k)
#pragma unroll
            for (int e = 0; e < 8; ++e) win[k][e] = win[k + 1][e];
        if (TAPS > 1) {
#pragma unroll
            for (int e = 0; e < 8; ++e) win[TAPS - 2][e] = cur[e];
        }
    }
}

// history[k] <- the sequence's input at position (context + n) - (taps - 1) + k, from the portion or from the old history
template <typename T>
__global__ void __launch_bounds__(256) tap_history_kernel(const atoma_tap_filter_args a) {
    pdl_launch_dependents();
    pdl_wait();
    const int b = blockIdx.y;
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int C = static_cast<int>(a.channels), keep = static_cast<int>(a.taps) - 1;
    if (c >= C) return;
    const int q0 = a.query_start[b], n = a.query_start[b + 1] - q0, ctx = a.context_lens[b];
    if (n <= 0) return;
    float *hist = a.history + static_cast<int64_t>(a.state_slots[b]) * a.history_stride;
    const T *in = static_cast<const T *>(a.in);
    const float ib = a.in_bias ? a.in_bias[c] : 0.f;
    float old[kMaxTaps];
#pragma unroll
    for (int k = 0; k < kMaxTaps; ++k) old[k] = (k < keep && k + n < keep && ctx - keep + k + n >= 0) ? hist[static_cast<int64_t>(k + n) * C + c] : 0.f;
#pragma unroll
    for (int k = 0; k < kMaxTaps; ++k) {
        if (k >= keep) break;
        const int rel = n - keep + k;
        hist[static_cast<int64_t>(k) * C + c] = rel >= 0 ? to_f(in[static_cast<int64_t>(q0 + rel) * a.ld_in + c]) + ib : old[k];
    }
}

// ---------------------------------------------------------------------------------------------
// per-head RMS norm of a float32 read-out, times a gate
// ---------------------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) headnorm_gate_kernel(const float *__restrict__ o, const float *__restrict__ weight,
                                                            const T *__restrict__ gate, int64_t ld_gate, T *__restrict__ out, int H, int V,
                                                            float eps) {
    pdl_launch_dependents();
    pdl_wait();
    const int64_t t = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    for (int h = warp; h < H; h += nwarp) {
        const float *r = o + (t * H + h) * V;
        float ss = 0.f;
        for (int c = lane; c < V; c += 32) ss = fmaf(r[c], r[c], ss);
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, s);
        const float inv = 1.0f / sqrtf(ss / static_cast<float>(V) + eps);
        for (int c = lane; c < V; c += 32) {
            float v = r[c] * inv * weight[c];
            if (gate) v *= silu(to_f(gate[t * ld_gate + h * V + c]));
            out[(t * H + h) * V + c] = from_f<T>(v);
        }
    }
}

// ---------------------------------------------------------------------------------------------
// rotary positions
// ---------------------------------------------------------------------------------------------
// sin and cos of pos * (freq + freq_lo), times amplitude.  The product is kept to twice float32's precision (its rounding error and the
// part of the frequency that float32 drops turn the pair by a correction): at position 10^5 a plain float32 angle is off by 4e-3.
__device__ __forceinline__ void turn(float pos, float freq, float freq_lo, float amplitude, float &sn, float &cs) {
    const float ang = pos * freq;
    const float rest = fmaf(pos, freq, -ang) + pos * freq_lo;
    float s, c;
    sincosf(ang, &s, &c);
    const float near_one = fmaf(-0.5f * rest, rest, 1.f);     // cos of the correction; its sine is the correction itself
    sn = amplitude * fmaf(rest, c, s * near_one);
    cs = amplitude * fmaf(-rest, s, c * near_one);
}

// buf [n] float32 (one warp's): the first 2 pairs entries turned by the token's angles (sin and cos of pair i at turns[2 i]), written to dst.
template <typename T>
__device__ __forceinline__ void rotate_store(const float *buf, int n, const float *turns, int pairs, int interleaved, T *__restrict__ dst, int lane) {
    for (int i = lane; i < pairs; i += 32) {
        const int ia = interleaved ? 2 * i : i, ib = interleaved ? 2 * i + 1 : i + pairs;
        const float sn = turns[2 * i], cs = turns[2 * i + 1], u = buf[ia], v = buf[ib];
        dst[ia] = from_f<T>(u * cs - v * sn);
        dst[ib] = from_f<T>(v * cs + u * sn);
    }
    for (int i = 2 * pairs + lane; i < n; i += 32) dst[i] = from_f<T>(buf[i]);
}

template <typename T>
__global__ void __launch_bounds__(256) qkv_headnorm_rope_cache_kernel(const atoma_qkv_rope_args a) {
    extern __shared__ float sm[];
    pdl_launch_dependents();
    pdl_wait();
    const int64_t t = blockIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    const int H = static_cast<int>(a.H), G = static_cast<int>(a.G), D = static_cast<int>(a.dim), V = static_cast<int>(a.vdim);
    const int Gv = a.v_heads > 0 ? static_cast<int>(a.v_heads) : G;
    const int units = a.slot_mapping ? H + G + Gv : H;
    const float amplitude = a.qk_amplitude != 0.f ? a.qk_amplitude : 1.f;
    const int wide = max(D, V);
    const int qk_pairs = a.qk_freq ? static_cast<int>(a.rot_pairs) : 0, v_pairs = a.v_freq ? static_cast<int>(a.v_pairs) : 0;
    float *turns = sm + nwarp * wide, *v_turns = turns + 2 * qk_pairs;   // all heads of the token turn by the same angles
    float *buf = sm + warp * wide;
    const T *row = static_cast<const T *>(a.proj) + t * a.ld;
    const float pos = static_cast<float>(a.positions[t]);
    for (int i = threadIdx.x; i < qk_pairs; i += blockDim.x)
        turn(pos, a.qk_freq[i], a.qk_freq_lo ? a.qk_freq_lo[i] : 0.f, amplitude, turns[2 * i], turns[2 * i + 1]);
    for (int i = threadIdx.x; i < v_pairs; i += blockDim.x) turn(pos, a.v_freq[i], 0.f, 1.f, v_turns[2 * i], v_turns[2 * i + 1]);
    __syncthreads();
    const int64_t slot = a.slot_mapping ? a.slot_mapping[t] : -1;
    for (int u = warp; u < units; u += nwarp) {
        const bool is_q = u < H, is_k = !is_q && u < H + G;
        const int hd = is_q ? u : (is_k ? u - H : u - H - G);
        if (!is_q && slot < 0) continue;
        const int n = (is_q || is_k) ? D : V;
        const int64_t col = is_q ? a.q_off + hd * D : (is_k ? a.k_off + hd * D : a.v_off + hd * V);
        const T *src = row + col;
        const float *bias = a.bias ? a.bias + col : nullptr;
        const float *w = is_q ? a.q_weight : (is_k ? a.k_weight : nullptr);
        float ss = 0.f;
        for (int c = lane; c < n; c += 32) {
            const float v = to_f(src[c]) + (bias ? bias[c] : 0.f);
            buf[c] = v;
            ss = fmaf(v, v, ss);
        }
        if (w || (a.unit_norm && (is_q || is_k))) {
#pragma unroll
            for (int s = 16; s > 0; s >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, s);
            float inv = 1.0f / sqrtf(ss / static_cast<float>(n) + a.eps);
            if (is_q && a.q_head_scale) inv *= a.q_head_scale[hd];
            for (int c = lane; c < n; c += 32) buf[c] = w ? buf[c] * inv * w[c] : buf[c] * inv;
        }
        __syncwarp();
        T *dst = is_q ? static_cast<T *>(a.q_out) + (t * H + hd) * D
                      : (is_k ? static_cast<T *>(a.k_cache) + (slot * G + hd) * D : static_cast<T *>(a.v_cache) + (slot * Gv + hd) * V);
        const bool vpart = !is_q && !is_k;
        rotate_store<T>(buf, n, vpart ? v_turns : turns, vpart ? v_pairs : qk_pairs, a.interleaved, dst, lane);
        __syncwarp();
    }
}

// The same for bfloat16 heads of whole 16-byte pieces: L lanes own a head, each two runs of four entries that stay in registers from the load
// to the store.  A lane's runs are the two halves of its four pairs (or, pairs of neighbours, eight entries in a row), so it turns
// them without asking another lane, and its sines and cosines serve every head of the token; entries behind the turned ones go to the lanes that
// are left, eight in a row.  A warp takes one of `parts` equal shares of a token's heads, 32 / L at a time, forms the token's angles itself (each group of
// L lanes some of them, the others by shuffles) and issues the loads of up to four rounds before it uses the first; no shared memory, no barrier.
// Values that only move are one run of bytes.
// Bound: HBM.  8192 tokens of 32 + 16 heads of 128, 201 MB: a warp per head, element by element through shared memory 147 us; a CTA per token
// 61.5 (0.73 of the issue slots: 47 M instructions, weights read and addresses formed per head, angles behind a barrier); this 41.0 (20 M); 3000 tokens of
// 32 + 16 heads of 64 24.6 and 17.0.  At 32 warps an SM a lane's 64 registers spill 8 to 88 bytes; 24 warps without spills took 51.2 us where this took 46.1 (at
// lower clocks), 40 with loads of three heads 71.8.
constexpr int kQkvHeads = 4;
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t unpack2(uint32_t w) { return pk2(__uint_as_float(__byte_perm(w, 0u, 0x1044)), __uint_as_float(w & 0xffff0000u)); }
__device__ __forceinline__ uint32_t repack2(uint64_t v) {
    float lo, hi;
    upk2(v, lo, hi);
    return pack2<__nv_bfloat16>(lo, hi);
}
struct HeadRuns {   // a lane's two runs of four entries in a head of n with `pairs` turned pairs (-1: none)
    int a, b;
    bool turned;
};
__device__ __forceinline__ HeadRuns head_runs(int l, int n, int pairs, bool interleaved) {
    HeadRuns r;
    r.turned = 4 * l < pairs;
    const bool halves = r.turned && !interleaved;
    r.a = halves ? 4 * l : 8 * l;   // 2 pairs + 8 (l - pairs / 4) = 8 l behind the turned ones
    r.b = halves ? pairs + 4 * l : 8 * l + 4;
    if (8 * l >= n) r.a = r.b = -1;
    return r;
}
// What turns a lane's pairs: halves (0, 1), (2, 3): cosines, sines and their negatives of two pairs at a time; neighbours: (cos, cos) and (-sin, sin) of each.
struct HeadTurns {
    uint64_t c[4], s[4];
};
// The angles of a lane's four pairs (4 l .. 4 l + 3 of `pairs`): the groups of L lanes take turns, and every lane asks for what it needs.
template <int L, bool IL>
__device__ __forceinline__ HeadTurns head_turns(float pos, const float *freq, const float *freq_lo, float amplitude, int pairs) {
    constexpr int NG = 32 / L, OWN = NG >= 4 ? 1 : 4 / NG;
    const int lane = threadIdx.x & 31, l = lane % L, g = lane / L;
    float sn[OWN], cs[OWN];
#pragma unroll
    for (int k = 0; k < OWN; ++k) {
        const int i = 4 * l + k * NG + g;
        sn[k] = 0.f, cs[k] = 1.f;
        if (i < pairs && k * NG + g < 4) turn(pos, freq[i], freq_lo ? freq_lo[i] : 0.f, amplitude, sn[k], cs[k]);
    }
    float s4[4], c4[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        s4[j] = __shfl_sync(0xffffffffu, sn[j / NG], j % NG * L + l);
        c4[j] = __shfl_sync(0xffffffffu, cs[j / NG], j % NG * L + l);
    }
    HeadTurns t;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (IL) {
            t.c[j] = pk2(c4[j], c4[j]);
            t.s[j] = pk2(-s4[j], s4[j]);
        } else if (j < 2) {
            t.c[j] = pk2(c4[2 * j], c4[2 * j + 1]);
            t.s[j] = pk2(s4[2 * j], s4[2 * j + 1]);
            t.c[j + 2] = 0;
            t.s[j + 2] = pk2(-s4[2 * j], -s4[2 * j + 1]);
        }
    }
    return t;
}
// Rounds of 32 / L heads from head u0 on, to n, of a token: src, dst and bias point to head 0; norm over the head's L lanes (mul = 1 / size; 0: none),
// weight w, scale per head, turn, back to bfloat16.  Every lane of a warp makes the same rounds, since a head's sum is asked for by shuffles.
// WHOLE: heads of 8 L entries, all of them turned, so that every lane has its eight and all distances are constants.
template <int L, bool IL, bool WHOLE>
__device__ __forceinline__ void heads_finish(const __nv_bfloat16 *src, __nv_bfloat16 *dst, int u0, int n, int size, const HeadRuns &r, const float *bias, float mul, float eps,
                                             const float *head_scale, const float *w, const HeadTurns &turns) {
    constexpr int NG = 32 / L;
    const int lane = threadIdx.x & 31, g = lane / L, l = lane % L;
    const bool mine = WHOLE || r.a >= 0, turned = WHOLE || r.turned;
    const int at = WHOLE ? (IL ? 8 : 4) * l : max(r.a, 0), gap = WHOLE ? (IL ? 4 : 4 * L) : r.b - r.a, stride = WHOLE ? 256 : NG * size;
    const int64_t begin = static_cast<int64_t>(u0 + g) * (WHOLE ? 8 * L : size) + at;
    src += begin, dst += begin;
    if (bias) bias += begin;
    ulonglong2 w0 = make_ulonglong2(0, 0), w1 = w0;
    if (w && mine) {
        w0 = *reinterpret_cast<const ulonglong2 *>(w + at);
        w1 = *reinterpret_cast<const ulonglong2 *>(w + at + gap);
    }
    for (; u0 < n; u0 += kQkvHeads * NG) {
        const int left = n - u0 - g;             // heads from this lane's on
        uint2 ra[kQkvHeads], rb[kQkvHeads];
#pragma unroll
        for (int i = 0; i < kQkvHeads; ++i) {
            ra[i] = rb[i] = make_uint2(0, 0);
            if (left > i * NG && mine) {
                ra[i] = *reinterpret_cast<const uint2 *>(src + i * stride);
                rb[i] = *reinterpret_cast<const uint2 *>(src + i * stride + gap);
            }
        }
#pragma unroll
        for (int i = 0; i < kQkvHeads; ++i) {
            if (u0 + i * NG >= n) break;
            uint64_t v[4] = {unpack2(ra[i].x), unpack2(ra[i].y), unpack2(rb[i].x), unpack2(rb[i].y)};
            const bool live = left > i * NG && mine;
            if (bias && live) {
                const ulonglong2 b0 = *reinterpret_cast<const ulonglong2 *>(bias + i * stride), b1 = *reinterpret_cast<const ulonglong2 *>(bias + i * stride + gap);
                v[0] = add2(v[0], b0.x), v[1] = add2(v[1], b0.y), v[2] = add2(v[2], b1.x), v[3] = add2(v[3], b1.y);
            }
            if (mul > 0.f) {
                float lo, hi;
                upk2(fma2(v[0], v[0], fma2(v[1], v[1], fma2(v[2], v[2], mul2(v[3], v[3])))), lo, hi);
                float ss = lo + hi;
#pragma unroll
                for (int o = L / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
                float inv = rsqrtf(fmaf(ss, mul, eps));
                if (head_scale && left > i * NG) inv *= head_scale[u0 + g + i * NG];
                const uint64_t inv2 = pk2(inv, inv);
#pragma unroll
                for (int j = 0; j < 4; ++j) v[j] = mul2(v[j], inv2);
                if (w) v[0] = mul2(v[0], w0.x), v[1] = mul2(v[1], w0.y), v[2] = mul2(v[2], w1.x), v[3] = mul2(v[3], w1.y);
            }
            if (turned) {
                if (IL) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        float lo, hi;
                        upk2(v[j], lo, hi);
                        v[j] = fma2(v[j], turns.c[j], mul2(pk2(hi, lo), turns.s[j]));
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const uint64_t u = v[j];
                        v[j] = fma2(u, turns.c[j], mul2(v[2 + j], turns.s[2 + j]));
                        v[2 + j] = fma2(v[2 + j], turns.c[j], mul2(u, turns.s[j]));
                    }
                }
            }
            if (live) {
                *reinterpret_cast<uint2 *>(dst + i * stride) = make_uint2(repack2(v[0]), repack2(v[1]));
                *reinterpret_cast<uint2 *>(dst + i * stride + gap) = make_uint2(repack2(v[2]), repack2(v[3]));
            }
        }
        src += kQkvHeads * stride;
        dst += kQkvHeads * stride;
        if (bias) bias += kQkvHeads * stride;
    }
}
constexpr int kQkvWarps = 4, kQkvResident = 32;   // warps of a CTA, of an SM
template <int L, bool IL, bool WHOLE>
__global__ void __launch_bounds__(32 * kQkvWarps, kQkvResident / kQkvWarps) qkv_headnorm_rope_cache_vec_kernel(const atoma_qkv_rope_args a, int parts) {
    using bf16 = __nv_bfloat16;
    constexpr int NG = 32 / L;
    pdl_launch_dependents();
    pdl_wait();
    const unsigned job = blockIdx.x * kQkvWarps + threadIdx.x / 32;
    const int t = static_cast<int>(job / static_cast<unsigned>(parts)), part = static_cast<int>(job % static_cast<unsigned>(parts));
    if (t >= a.T) return;
    const int H = static_cast<int>(a.H), G = static_cast<int>(a.G), D = static_cast<int>(a.dim), V = static_cast<int>(a.vdim);
    const int Gv = a.v_heads > 0 ? static_cast<int>(a.v_heads) : G;
    const int lane = threadIdx.x & 31, l = lane % L;
    const int64_t slot = a.slot_mapping ? a.slot_mapping[t] : -1;
    const int qk_pairs = a.qk_freq ? static_cast<int>(a.rot_pairs) : 0, v_pairs = a.v_freq ? static_cast<int>(a.v_pairs) : 0;
    const HeadRuns qk = head_runs(l, D, qk_pairs, IL);
    const bf16 *row = static_cast<const bf16 *>(a.proj) + t * a.ld;
    const bool v_plain = v_pairs == 0 && !a.bias;
    if (slot >= 0 && v_plain) {   // values as projected: one run of bytes
        const uint4 *src = reinterpret_cast<const uint4 *>(row + a.v_off);
        uint4 *dst = reinterpret_cast<uint4 *>(static_cast<bf16 *>(a.v_cache) + slot * Gv * V);
#pragma unroll 2
        for (int i = part * 32 + lane; i < Gv * V / 8; i += parts * 32) dst[i] = src[i];
    }
    // this warp's share of the token's rounds: query heads, key heads, values
    const int rq = (H + NG - 1) / NG, rk = a.slot_mapping ? (G + NG - 1) / NG : 0, rv = a.slot_mapping && !v_plain ? (Gv + NG - 1) / NG : 0;
    const int each = (rq + rk + rv + parts - 1) / parts, from = part * each, to = from + each;
    const float amplitude = a.qk_amplitude != 0.f ? a.qk_amplitude : 1.f, pos = static_cast<float>(a.positions[t]), mul = 1.f / static_cast<float>(D);
    HeadTurns tr;
    if (from < rq + rk) tr = head_turns<L, IL>(pos, a.qk_freq, a.qk_freq_lo, amplitude, qk_pairs);
    if (from < rq)
        heads_finish<L, IL, WHOLE>(row + a.q_off, static_cast<bf16 *>(a.q_out) + static_cast<int64_t>(t) * H * D, from * NG, min(H, to * NG), D, qk, a.bias ? a.bias + a.q_off : nullptr,
                                   a.q_weight || a.unit_norm ? mul : 0.f, a.eps, a.q_head_scale, a.q_weight, tr);
    if (slot < 0) return;
    if (from < rq + rk && to > rq)
        heads_finish<L, IL, WHOLE>(row + a.k_off, static_cast<bf16 *>(a.k_cache) + slot * G * D, max(0, from - rq) * NG, min(G, (to - rq) * NG), D, qk, a.bias ? a.bias + a.k_off : nullptr,
                                   a.k_weight || a.unit_norm ? mul : 0.f, a.eps, nullptr, a.k_weight, tr);
    if (v_plain || to <= rq + rk) return;
    const HeadRuns vr = head_runs(l, V, v_pairs, IL);
    tr = head_turns<L, IL>(pos, a.v_freq, nullptr, 1.f, v_pairs);
    heads_finish<L, IL, false>(row + a.v_off, static_cast<bf16 *>(a.v_cache) + slot * Gv * V, max(0, from - rq - rk) * NG, min(Gv, (to - rq - rk) * NG), V, vr, a.bias ? a.bias + a.v_off : nullptr,
                               0.f, 0.f, nullptr, nullptr, tr);
}

template <typename T>
__global__ void __launch_bounds__(256) rotate_heads_kernel(T *__restrict__ x, const int64_t *__restrict__ positions,
                                                           const float *__restrict__ freq, const float *__restrict__ freq_lo, float amplitude,
                                                           int H, int n, int pairs, int interleaved, float sign) {
    pdl_launch_dependents();
    pdl_wait();
    const int64_t t = blockIdx.x;
    const float pos = static_cast<float>(positions[t]);
    T *row = x + t * H * n;
    for (int idx = threadIdx.x; idx < H * pairs; idx += blockDim.x) {
        const int h = idx / pairs, i = idx % pairs;
        const int ia = h * n + (interleaved ? 2 * i : i), ib = h * n + (interleaved ? 2 * i + 1 : i + pairs);
        float sn, cs;
        turn(pos, freq[i], freq_lo ? freq_lo[i] : 0.f, amplitude, sn, cs);
        sn *= sign;
        const float u = to_f(row[ia]), v = to_f(row[ib]);
        row[ia] = from_f<T>(u * cs - v * sn);
        row[ib] = from_f<T>(v * cs + u * sn);
    }
}

template <typename T>
__global__ void __launch_bounds__(kRowThreads) latent_norm_rope_cache_kernel(const T *__restrict__ proj, int64_t ld,
                                                                             const float *__restrict__ q_w, const float *__restrict__ kv_w,
                                                                             const float *__restrict__ freq, const float *__restrict__ freq_lo,
                                                                             float amplitude, int pairs, int interleaved,
                                                                             const int64_t *__restrict__ positions,
                                                                             const int64_t *__restrict__ slots, T *__restrict__ cq_out,
                                                                             T *__restrict__ cache, int q_rank, int kv_rank, int rot_dim,
                                                                             float eps) {
    __shared__ float red[32];
    pdl_launch_dependents();
    pdl_wait();
    const int64_t t = blockIdx.x;
    const T *r = proj + t * ld;
    if (q_rank > 0) {
        float ss = 0.f;
        for (int c = threadIdx.x; c < q_rank; c += blockDim.x) {
            const float v = to_f(r[c]);
            ss = fmaf(v, v, ss);
        }
        const float inv = 1.0f / sqrtf(block_sum(ss, red) / static_cast<float>(q_rank) + eps);
        for (int c = threadIdx.x; c < q_rank; c += blockDim.x) cq_out[t * q_rank + c] = from_f<T>(to_f(r[c]) * inv * q_w[c]);
    }
    const int64_t slot = slots ? slots[t] : -1;
    if (slot < 0) return;
    float ss = 0.f;
    for (int c = threadIdx.x; c < kv_rank; c += blockDim.x) {
        const float v = to_f(r[q_rank + c]);
        ss = fmaf(v, v, ss);
    }
    const float inv = 1.0f / sqrtf(block_sum(ss, red) / static_cast<float>(kv_rank) + eps);
    T *dst = cache + slot * (kv_rank + rot_dim);
    for (int c = threadIdx.x; c < kv_rank; c += blockDim.x) dst[c] = from_f<T>(to_f(r[q_rank + c]) * inv * kv_w[c]);
    const T *kr = r + q_rank + kv_rank;
    const float pos = static_cast<float>(positions[t]);
    for (int i = threadIdx.x; i < pairs; i += blockDim.x) {
        const int ia = interleaved ? 2 * i : i, ib = interleaved ? 2 * i + 1 : i + pairs;
        float sn, cs;
        turn(pos, freq[i], freq_lo ? freq_lo[i] : 0.f, amplitude, sn, cs);
        const float u = to_f(kr[ia]), v = to_f(kr[ib]);
        dst[kv_rank + ia] = from_f<T>(u * cs - v * sn);
        dst[kv_rank + ib] = from_f<T>(v * cs + u * sn);
    }
    for (int c = 2 * pairs + threadIdx.x; c < rot_dim; c += blockDim.x) dst[kv_rank + c] = kr[c];
}

// q_lat[t, h, kv_rank + c] = the rotated part of query head h, float32
template <typename T>
__global__ void __launch_bounds__(256) latent_query_rope_kernel(const T *__restrict__ q, const float *__restrict__ freq,
                                                                const float *__restrict__ freq_lo, float amplitude, int pairs, int interleaved, const int64_t *__restrict__ positions,
                                                                float *__restrict__ q_lat, int H, int dim, int rot_dim, int kv_rank) {
    pdl_launch_dependents();
    pdl_wait();
    const int64_t t = blockIdx.x;
    const float pos = static_cast<float>(positions[t]);
    const int hs = dim + rot_dim, row = kv_rank + rot_dim;
    for (int idx = threadIdx.x; idx < H * pairs; idx += blockDim.x) {
        const int h = idx / pairs, i = idx % pairs;
        const int ia = interleaved ? 2 * i : i, ib = interleaved ? 2 * i + 1 : i + pairs;
        const T *src = q + (t * H + h) * hs + dim;
        float sn, cs;
        turn(pos, freq[i], freq_lo ? freq_lo[i] : 0.f, amplitude, sn, cs);
        const float u = to_f(src[ia]), v = to_f(src[ib]);
        float *dst = q_lat + (t * H + h) * row + kv_rank;
        dst[ia] = u * cs - v * sn;
        dst[ib] = v * cs + u * sn;
    }
    const int rest = rot_dim - 2 * pairs;
    for (int idx = threadIdx.x; idx < H * rest; idx += blockDim.x) {
        const int h = idx / rest, c = 2 * pairs + idx % rest;
        q_lat[(t * H + h) * row + kv_rank + c] = to_f(q[(t * H + h) * hs + dim + c]);
    }
}

// Queries of a few tokens into the latent space, their rotated part beside them: q_lat[t, h, :kv_rank] = q[t, h, :dim] . w_uk[h] and the rotation of what follows, by one
// launch.  Bound: latency (32 tokens of 32 heads move 9 MB).  A CTA takes 32 tokens x 64 columns of one head with all of its operands in flight at once, or, the last
// of a head, that head's rotations.  32 tokens of 32 heads of 128 + 64 on 512: a product in 64-token tiles and a rotation behind it 16.3 us a call, this 12.9; with the L2 cache
// flushed, 1, 33 and 64 tokens 19.5 / 10.3, 19.6 / 14.4, 19.5 / 14.4, of 128 heads 37.9 / 13.3, 42.0 / 20.6, 43.8 / 22.5.  4 to 128 heads of 128 or 192 + 64 and of 128 alone on 512, of 64 +
// 32 on 256: 1 to 64 tokens take 0.3 to 0.95 of the time.
constexpr int kAbsorbTokens = 32, kAbsorbCols = 64;
__global__ void __launch_bounds__(128) latent_absorb_few_kernel(const __nv_bfloat16 *__restrict__ q, const __nv_bfloat16 *__restrict__ w, const float *__restrict__ freq,
                                                                const float *__restrict__ freq_lo, float amplitude, int pairs, int interleaved,
                                                                const int64_t *__restrict__ positions, float *__restrict__ q_lat, int T, int H, int dim, int rot_dim, int kv_rank) {
    extern __shared__ __align__(16) unsigned char absorb_sm[];
    pdl_launch_dependents();
    pdl_wait();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h = blockIdx.z, t0 = blockIdx.y * kAbsorbTokens, n = min(kAbsorbTokens, T - t0);
    const int hs = dim + rot_dim, row = kv_rank + rot_dim;
    const __nv_bfloat16 *qh = q + (static_cast<int64_t>(t0) * H + h) * hs;
    float *oh = q_lat + (static_cast<int64_t>(t0) * H + h) * row;
    if (blockIdx.x == gridDim.x - 1 && rot_dim > 0) {
        for (int i = tid; i < n * pairs; i += 128) {
            const int t = i / pairs, c = i - t * pairs, ia = interleaved ? 2 * c : c, ib = interleaved ? 2 * c + 1 : c + pairs;
            const __nv_bfloat16 *src = qh + static_cast<int64_t>(t) * H * hs + dim;
            float sn, cs;
            turn(static_cast<float>(positions[t0 + t]), freq[c], freq_lo ? freq_lo[c] : 0.f, amplitude, sn, cs);
            const float u = to_f(src[ia]), v = to_f(src[ib]);
            float *dst = oh + static_cast<int64_t>(t) * H * row + kv_rank;
            dst[ia] = u * cs - v * sn;
            dst[ib] = v * cs + u * sn;
        }
        const int rest = rot_dim - 2 * pairs;
        for (int i = tid; i < n * rest; i += 128) {
            const int t = i / rest, c = 2 * pairs + i - t * rest;
            oh[static_cast<int64_t>(t) * H * row + kv_rank + c] = to_f(qh[static_cast<int64_t>(t) * H * hs + dim + c]);
        }
        return;
    }
    const int n0 = blockIdx.x * kAbsorbCols, q_row = dim * 2 + 16, pieces = dim / 8;
    constexpr int kWRow = kAbsorbCols * 2 + 16;   // 16 bytes more than whole lines: eight rows hit distinct banks
    unsigned char *ws = absorb_sm, *qs = absorb_sm + dim * kWRow;
    const __nv_bfloat16 *wh = w + static_cast<int64_t>(h) * dim * kv_rank + n0;
    for (int i = tid; i < dim * 8; i += 128) cp_async_16(smem_u32(ws + (i >> 3) * kWRow + (i & 7) * 16), wh + static_cast<int64_t>(i >> 3) * kv_rank + (i & 7) * 8, 16);
    for (int i = tid; i < kAbsorbTokens * pieces; i += 128) {
        const int t = i / pieces, c = i - t * pieces;
        cp_async_16(smem_u32(qs + t * q_row + c * 16), qh + static_cast<int64_t>(min(t, n - 1)) * H * hs + c * 8, 16);
    }
    cp_async_commit();
    cp_async_wait_all();
    __syncthreads();
    float acc[2][2][4] = {};
    for (int k = 0; k < dim; k += 16) {
        uint32_t b[4];
        ldmatrix_x4_trans(b, smem_u32(ws + (k + (lane & 7) + ((lane >> 3) & 1) * 8) * kWRow + (warp * 16 + (lane >> 4) * 8) * 2));
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
            uint32_t a[4];
            ldmatrix_x4(a, smem_u32(qs + (mt * 16 + (lane & 15)) * q_row + (k + (lane >> 4) * 8) * 2));
            Mma16816<__nv_bfloat16>::run(acc[mt][0], a, b[0], b[1]);
            Mma16816<__nv_bfloat16>::run(acc[mt][1], a, b[2], b[3]);
        }
    }
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int t = mt * 16 + (lane >> 2) + 8 * e;
            if (t >= n) continue;
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
                *reinterpret_cast<float2 *>(oh + static_cast<int64_t>(t) * H * row + n0 + warp * 16 + nt * 8 + 2 * (lane & 3)) = make_float2(acc[mt][nt][2 * e], acc[mt][nt][2 * e + 1]);
        }
}

}  // namespace

#define HYB_DISPATCH(dtype, CALL) ((dtype) == ATOMA_DTYPE_BF16 ? CALL(__nv_bfloat16) : CALL(float))

bool hyb_parallel_residual_norm(const atoma_parallel_residual_args &a, cudaStream_t stream) {
    if (a.T <= 0) return true;
    if (!hybrid::known_dtype(a.dtype, "atoma_parallel_residual_norm")) return false;
    if (!a.x || a.width <= 0 || (a.w_next && !a.h) || (a.norm_a && !a.y_a) || (a.norm_b && !a.y_b)) {
        set_status(kErrInvalidArg, "atoma_parallel_residual_norm: null argument");
        return false;
    }
    const size_t smem = static_cast<size_t>(a.width) * 4;
    if (smem > 200 * 1024) {
        set_status(kErrUnsupported, "atoma_parallel_residual_norm: a width of %lld exceeds shared memory", static_cast<long long>(a.width));
        return false;
    }
    if (smem > 48 * 1024) {
        cudaFuncSetAttribute(parallel_residual_norm_kernel<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
        cudaFuncSetAttribute(parallel_residual_norm_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    }
#define CALL(TT) launch_ex(parallel_residual_norm_kernel<TT>, dim3(static_cast<unsigned>(a.T)), dim3(kRowThreads), smem, stream, a)
    return hybrid::launched(HYB_DISPATCH(a.dtype, CALL), "parallel_residual_norm_kernel");
#undef CALL
}

bool hyb_tap_filter(const atoma_tap_filter_args &a, cudaStream_t stream) {
    if (a.T <= 0 || a.channels <= 0) return true;
    if (!hybrid::known_dtype(a.dtype, "atoma_tap_filter")) return false;
    if (!a.in || !a.w1 || !a.out1 || (a.w2 && !a.out2) || a.taps < 1 || a.taps > kMaxTaps || a.ld_in < a.channels || a.ld_out < a.channels ||
        !a.token_seq || !a.query_start || !a.context_lens || a.B <= 0 ||
        (a.taps > 1 && (!a.history || !a.state_slots || a.history_stride < (a.taps - 1) * a.channels))) {
        set_status(kErrInvalidArg, "atoma_tap_filter: null argument, more than %d taps, or a history row shorter than (taps - 1) channels", kMaxTaps);
        return false;
    }
    const unsigned cb = static_cast<unsigned>((a.channels + 255) / 256);
    auto piece16 = [](const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    const bool vec = a.dtype == ATOMA_DTYPE_BF16 && a.taps >= 2 && a.taps <= 4 && a.channels % 8 == 0 && a.ld_in % 8 == 0 && a.ld_out % 8 == 0 &&
                     piece16(a.in) && piece16(a.out1) && piece16(a.out2) && piece16(a.w1) && piece16(a.w2) && !(g_hybrid_debug & 2);
    if (vec) {
        // tokens per thread: long steps amortise the window's refill, short ones keep the device filled
        const int run = a.T >= 4096 ? 16 : (a.T >= 1024 ? 8 : (a.T >= 256 ? 4 : 1));
        const dim3 grid(static_cast<unsigned>((a.channels / 8 + 127) / 128), static_cast<unsigned>((a.T + run - 1) / run));
        cudaError_t e;
        if (a.taps == 2) e = launch_ex(tap_filter_vec_kernel<2>, grid, dim3(128), 0, stream, a, run);
        else if (a.taps == 3) e = launch_ex(tap_filter_vec_kernel<3>, grid, dim3(128), 0, stream, a, run);
        else e = launch_ex(tap_filter_vec_kernel<4>, grid, dim3(128), 0, stream, a, run);
        if (!hybrid::launched(e, "tap_filter_vec_kernel")) return false;
    } else {
#define CALL(TT) launch_ex(tap_filter_kernel<TT>, dim3(cb, static_cast<unsigned>(a.T)), dim3(256), 0, stream, a)
        if (!hybrid::launched(HYB_DISPATCH(a.dtype, CALL), "tap_filter_kernel")) return false;
#undef CALL
    }
    if (a.taps == 1) return true;
#define CALL(TT) launch_ex(tap_history_kernel<TT>, dim3(cb, static_cast<unsigned>(a.B)), dim3(256), 0, stream, a)
    return hybrid::launched(HYB_DISPATCH(a.dtype, CALL), "tap_history_kernel");
#undef CALL
}

bool hyb_headnorm_gate(const float *o, const float *weight, const void *gate, int64_t ld_gate, void *out, int64_t T, int64_t H, int64_t vdim,
                       float eps, uint32_t dtype, cudaStream_t stream) {
    if (T <= 0) return true;
    if (!hybrid::known_dtype(dtype, "atoma_headnorm_gate")) return false;
    if (!o || !weight || !out || H <= 0 || vdim <= 0 || (gate && ld_gate < H * vdim)) {
        set_status(kErrInvalidArg, "atoma_headnorm_gate: null argument or a gate row shorter than heads * vdim");
        return false;
    }
    const unsigned threads = static_cast<unsigned>(std::min<int64_t>(8, H) * 32);
#define CALL(TT) launch_ex(headnorm_gate_kernel<TT>, dim3(static_cast<unsigned>(T)), dim3(threads), 0, stream, o, weight, \
                           static_cast<const TT *>(gate), ld_gate, static_cast<TT *>(out), static_cast<int>(H), static_cast<int>(vdim), eps)
    return hybrid::launched(HYB_DISPATCH(dtype, CALL), "headnorm_gate_kernel");
#undef CALL
}

bool hyb_qkv_headnorm_rope_cache(const atoma_qkv_rope_args &a, cudaStream_t stream) {
    if (a.T <= 0) return true;
    if (!hybrid::known_dtype(a.dtype, "atoma_qkv_headnorm_rope_cache")) return false;
    if (!a.proj || !a.q_out || !a.positions || a.H <= 0 || a.G <= 0 || a.H % a.G || a.dim <= 0 || a.vdim <= 0 ||
        (a.slot_mapping && (!a.k_cache || !a.v_cache)) || a.q_off < 0 || (a.slot_mapping && (a.k_off < 0 || a.v_off < 0)) || a.q_off + a.H * a.dim > a.ld ||
        (a.slot_mapping && (a.k_off + a.G * a.dim > a.ld || a.v_off + (a.v_heads > 0 ? a.v_heads : a.G) * a.vdim > a.ld)) || a.v_heads < 0 || a.rot_pairs < 0 || 2 * a.rot_pairs > a.dim || a.v_pairs < 0 ||
        2 * a.v_pairs > a.vdim || (a.rot_pairs > 0 && !a.qk_freq) || (a.q_head_scale && !a.q_weight && !a.unit_norm)) {
        set_status(kErrInvalidArg, "atoma_qkv_headnorm_rope_cache: null argument, columns outside the row, or more rotated entries than a head has");
        return false;
    }
    const unsigned warps = static_cast<unsigned>(std::min<int64_t>(8, a.H + 2 * a.G));
    const size_t smem = (static_cast<size_t>(warps) * std::max(a.dim, a.vdim) + 2 * (a.rot_pairs + a.v_pairs)) * 4;
    if (smem > 48 * 1024) {
        set_status(kErrUnsupported, "atoma_qkv_headnorm_rope_cache: heads of %lld entries", static_cast<long long>(std::max(a.dim, a.vdim)));
        return false;
    }
    // 16-byte pieces everywhere and whole runs of four pairs; heads of up to 256 entries fit a warp
    auto al = [](const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    const bool pieces = a.dtype == ATOMA_DTYPE_BF16 && !(g_hybrid_debug & 2) && a.dim % 8 == 0 && a.vdim % 8 == 0 && std::max(a.dim, a.vdim) <= 256 && a.ld % 8 == 0 &&
                        a.q_off % 8 == 0 && (!a.slot_mapping || (a.k_off % 8 == 0 && a.v_off % 8 == 0)) && al(a.proj) && al(a.q_out) &&
                        (!a.slot_mapping || (al(a.k_cache) && al(a.v_cache))) && al(a.q_weight) && al(a.k_weight) && al(a.bias) &&
                        a.rot_pairs % 4 == 0 && a.v_pairs % 4 == 0 && a.T < (1ll << 24);
    if (pieces) {
        const int64_t n = std::max(a.dim, a.vdim), groups = n <= 64 ? 4 : n <= 128 ? 2 : 1;
        const int64_t heads = a.H + (a.slot_mapping ? a.G + (a.bias || (a.v_freq && a.v_pairs > 0) ? (a.v_heads > 0 ? a.v_heads : a.G) : 0) : 0), rounds = (heads + groups - 1) / groups;
        // shares of a token: so many that the warps stay within the SMs once, and no more than there are rounds (a share more, which starts a second wave / this, us:
        // 1000 tokens of 32 + 32 + 32 heads, values of 128 rotated, 17.5 / 14.5, a CTA per token 16.4; 1700 tokens of 32 + 16 of 128, half of them turned, 18.4 / 16.5, 16.4;
        // 2200 tokens of 32 + 16 of 128 17.8 / 14.5; twice as many shares, 8192 tokens, 47.3 where once took 46.1)
        const int64_t want = kQkvResident * current_device_info().sm_count / a.T;
        const int parts = static_cast<int>(std::max<int64_t>(1, std::min(rounds, want)));
        const dim3 grid(static_cast<unsigned>((a.T * parts + kQkvWarps - 1) / kQkvWarps)), block(32 * kQkvWarps);
        const bool whole = a.dim == 256 / groups && a.qk_freq && 2 * a.rot_pairs == a.dim;
#define PICK_L(IL, WHOLE) (n <= 64 ? qkv_headnorm_rope_cache_vec_kernel<8, IL, WHOLE> : n <= 128 ? qkv_headnorm_rope_cache_vec_kernel<16, IL, WHOLE> : qkv_headnorm_rope_cache_vec_kernel<32, IL, WHOLE>)
#define PICK(IL) (whole ? PICK_L(IL, true) : PICK_L(IL, false))
        const cudaError_t e = launch_ex(a.interleaved ? PICK(true) : PICK(false), grid, block, 0, stream, a, parts);
#undef PICK
#undef PICK_L
        return hybrid::launched(e, "qkv_headnorm_rope_cache_vec_kernel");
    }
#define CALL(TT) launch_ex(qkv_headnorm_rope_cache_kernel<TT>, dim3(static_cast<unsigned>(a.T)), dim3(warps * 32), smem, stream, a)
    return hybrid::launched(HYB_DISPATCH(a.dtype, CALL), "qkv_headnorm_rope_cache_kernel");
#undef CALL
}

bool hyb_rotate_heads(void *x, const int64_t *positions, const float *freq, const float *freq_lo, float amplitude, int64_t T, int64_t H, int64_t n,
                      int64_t pairs, int32_t interleaved, float sign, uint32_t dtype, cudaStream_t stream) {
    if (T <= 0 || pairs <= 0) return true;
    if (!hybrid::known_dtype(dtype, "atoma_rotate_heads")) return false;
    if (!x || !positions || !freq || H <= 0 || 2 * pairs > n) {
        set_status(kErrInvalidArg, "atoma_rotate_heads: null argument or more rotated entries than a head has");
        return false;
    }
#define CALL(TT) launch_ex(rotate_heads_kernel<TT>, dim3(static_cast<unsigned>(T)), dim3(256), 0, stream, static_cast<TT *>(x), positions, freq, \
                           freq_lo, amplitude, static_cast<int>(H), static_cast<int>(n), static_cast<int>(pairs), interleaved, sign)
    return hybrid::launched(HYB_DISPATCH(dtype, CALL), "rotate_heads_kernel");
#undef CALL
}

bool hyb_latent_norm_rope_cache(const void *proj, int64_t ld, const float *q_w, const float *kv_w, const float *freq, const float *freq_lo, float amplitude, int64_t pairs,
                                int32_t interleaved, const int64_t *positions, const int64_t *slots, void *cq_out, void *cache, int64_t T,
                                int64_t q_rank, int64_t kv_rank, int64_t rot_dim, float eps, uint32_t dtype, cudaStream_t stream) {
    if (T <= 0) return true;
    if (!hybrid::known_dtype(dtype, "atoma_latent_norm_rope_cache")) return false;
    if (!proj || kv_rank <= 0 || q_rank < 0 || rot_dim < 0 || ld < q_rank + kv_rank + rot_dim || !kv_w || (q_rank > 0 && (!q_w || !cq_out)) ||
        (slots && !cache) || !positions || pairs < 0 || 2 * pairs > rot_dim || (pairs > 0 && !freq)) {
        set_status(kErrInvalidArg, "atoma_latent_norm_rope_cache: null argument or a row shorter than q_rank + kv_rank + rot_dim");
        return false;
    }
#define CALL(TT) launch_ex(latent_norm_rope_cache_kernel<TT>, dim3(static_cast<unsigned>(T)), dim3(kRowThreads), 0, stream, \
                           static_cast<const TT *>(proj), ld, q_w, kv_w, freq, freq_lo, amplitude, static_cast<int>(pairs), interleaved, positions, slots, \
                           static_cast<TT *>(cq_out), static_cast<TT *>(cache), static_cast<int>(q_rank), static_cast<int>(kv_rank), \
                           static_cast<int>(rot_dim), eps)
    return hybrid::launched(HYB_DISPATCH(dtype, CALL), "latent_norm_rope_cache_kernel");
#undef CALL
}

bool hyb_latent_query_absorb_rope(const void *q, const void *w_uk, const float *freq, const float *freq_lo, float amplitude, int64_t pairs, int32_t interleaved,
                                  const int64_t *positions, float *q_lat, int64_t T, int64_t H, int64_t dim, int64_t rot_dim, int64_t kv_rank,
                                  uint32_t dtype, cudaStream_t stream) {
    if (T <= 0) return true;
    if (!hybrid::known_dtype(dtype, "atoma_latent_query_absorb_rope")) return false;
    if (!q || !w_uk || !q_lat || !positions || H <= 0 || dim <= 0 || rot_dim < 0 || kv_rank <= 0 || pairs < 0 || 2 * pairs > rot_dim ||
        (pairs > 0 && !freq)) {
        set_status(kErrInvalidArg, "atoma_latent_query_absorb_rope: null argument or more rotated entries than the rotated part has");
        return false;
    }
    const int64_t hs = dim + rot_dim, row = kv_rank + rot_dim;
    // decoded tokens, whose rows are whole pieces of 16 bytes (a result row: of 8): one launch; more tokens fill the SMs in tiles of 64
    auto al = [](const void *p, int bytes) { return (reinterpret_cast<uintptr_t>(p) & (bytes - 1)) == 0; };
    const size_t smem = static_cast<size_t>(dim) * (kAbsorbCols * 2 + 16) + kAbsorbTokens * (static_cast<size_t>(dim) * 2 + 16);
    if (dtype == ATOMA_DTYPE_BF16 && !(g_hybrid_debug & 1) && T <= 64 && dim % 16 == 0 && hs % 8 == 0 && row % 2 == 0 && kv_rank % kAbsorbCols == 0 && smem <= 48 * 1024 &&
        H <= 65535 && al(q, 16) && al(w_uk, 16) && al(q_lat, 8)) {
        const dim3 grid(static_cast<unsigned>(kv_rank / kAbsorbCols + (rot_dim > 0 ? 1 : 0)), static_cast<unsigned>((T + kAbsorbTokens - 1) / kAbsorbTokens), static_cast<unsigned>(H));
        return hybrid::launched(launch_ex(latent_absorb_few_kernel, grid, dim3(128), smem, stream, static_cast<const __nv_bfloat16 *>(q), static_cast<const __nv_bfloat16 *>(w_uk), freq,
                                          freq_lo, amplitude, static_cast<int>(pairs), interleaved, positions, q_lat, static_cast<int>(T), static_cast<int>(H), static_cast<int>(dim),
                                          static_cast<int>(rot_dim), static_cast<int>(kv_rank)),
                                "latent_absorb_few_kernel");
    }
    if (!hyb_head_project_ld(q, H * hs, hs, w_uk, q_lat, H * row, row, T, H, dim, kv_rank, 1, dtype, stream)) return false;
    if (rot_dim == 0) return true;
#define CALL(TT) launch_ex(latent_query_rope_kernel<TT>, dim3(static_cast<unsigned>(T)), dim3(256), 0, stream, static_cast<const TT *>(q), freq, freq_lo, amplitude, \
                           static_cast<int>(pairs), interleaved, positions, q_lat, static_cast<int>(H), static_cast<int>(dim), \
                           static_cast<int>(rot_dim), static_cast<int>(kv_rank))
    return hybrid::launched(HYB_DISPATCH(dtype, CALL), "latent_query_rope_kernel");
#undef CALL
}

bool hyb_latent_expand_values(const float *o_lat, const void *w_uv, const void *gate, int64_t ld_gate, void *out, int64_t T, int64_t H, int64_t vdim,
                              int64_t kv_rank, int64_t row, uint32_t dtype, cudaStream_t stream) {
    if (row < kv_rank || (gate && ld_gate < H * vdim)) {
        set_status(kErrInvalidArg, "atoma_latent_expand_values: rows of %lld entries for a latent of %lld, or a gate row shorter than the heads", static_cast<long long>(row),
                   static_cast<long long>(kv_rank));
        return false;
    }
    return hyb_head_project_ld(o_lat, H * row, row, w_uv, out, H * vdim, vdim, T, H, vdim, kv_rank, 0, dtype, stream, gate, ld_gate);
}

}  // namespace atoma

using namespace atoma;

extern "C" void atoma_parallel_residual_norm(const atoma_parallel_residual_args *args, atoma_stream_t stream) {
    clear_status();
    if (!args) {
        set_status(kErrInvalidArg, "atoma_parallel_residual_norm: args is NULL");
        return;
    }
    hyb_parallel_residual_norm(*args, static_cast<cudaStream_t>(stream));
}

extern "C" void atoma_tap_filter(const atoma_tap_filter_args *args, atoma_stream_t stream) {
    clear_status();
    if (!args) {
        set_status(kErrInvalidArg, "atoma_tap_filter: args is NULL");
        return;
    }
    hyb_tap_filter(*args, static_cast<cudaStream_t>(stream));
}

extern "C" void atoma_headnorm_gate(const float *o, const float *weight, const void *gate, int64_t ld_gate, void *out, int64_t T, int64_t H,
                                    int64_t vdim, float eps, uint32_t dtype, atoma_stream_t stream) {
    clear_status();
    hyb_headnorm_gate(o, weight, gate, ld_gate, out, T, H, vdim, eps, dtype, static_cast<cudaStream_t>(stream));
}

extern "C" void atoma_qkv_headnorm_rope_cache(const atoma_qkv_rope_args *args, atoma_stream_t stream) {
    clear_status();
    if (!args) {
        set_status(kErrInvalidArg, "atoma_qkv_headnorm_rope_cache: args is NULL");
        return;
    }
    hyb_qkv_headnorm_rope_cache(*args, static_cast<cudaStream_t>(stream));
}

extern "C" void atoma_rotate_heads(void *x, const int64_t *positions, const float *freq, const float *freq_lo, float amplitude, int64_t T, int64_t H,
                                   int64_t n, int64_t pairs, int32_t interleaved, float sign, uint32_t dtype, atoma_stream_t stream) {
    clear_status();
    hyb_rotate_heads(x, positions, freq, freq_lo, amplitude, T, H, n, pairs, interleaved, sign, dtype, static_cast<cudaStream_t>(stream));
}

extern "C" void atoma_latent_norm_rope_cache(const void *proj, int64_t ld, const float *q_weight, const float *kv_weight, const float *freq, const float *freq_lo, float amplitude,
                                             int64_t pairs, int32_t interleaved, const int64_t *positions, const int64_t *slot_mapping,
                                             void *cq_out, void *cache, int64_t T, int64_t q_rank, int64_t kv_rank, int64_t rot_dim, float eps,
                                             uint32_t dtype, atoma_stream_t stream) {
    clear_status();
    hyb_latent_norm_rope_cache(proj, ld, q_weight, kv_weight, freq, freq_lo, amplitude, pairs, interleaved, positions, slot_mapping, cq_out, cache, T, q_rank, kv_rank,
                               rot_dim, eps, dtype, static_cast<cudaStream_t>(stream));
}

extern "C" void atoma_latent_query_absorb_rope(const void *q, const void *w_uk, const float *freq, const float *freq_lo, float amplitude, int64_t pairs, int32_t interleaved,
                                               const int64_t *positions, float *q_lat, int64_t T, int64_t H, int64_t dim, int64_t rot_dim,
                                               int64_t kv_rank, uint32_t dtype, atoma_stream_t stream) {
    clear_status();
    hyb_latent_query_absorb_rope(q, w_uk, freq, freq_lo, amplitude, pairs, interleaved, positions, q_lat, T, H, dim, rot_dim, kv_rank, dtype,
                                 static_cast<cudaStream_t>(stream));
}

extern "C" void atoma_latent_expand_values(const float *o_lat, const void *w_uv, const void *gate, int64_t ld_gate, void *out, int64_t T, int64_t H,
                                           int64_t vdim, int64_t kv_rank, int64_t row, uint32_t dtype, atoma_stream_t stream) {
    clear_status();
    hyb_latent_expand_values(o_lat, w_uv, gate, ld_gate, out, T, H, vdim, kv_rank, row, dtype, static_cast<cudaStream_t>(stream));
}
