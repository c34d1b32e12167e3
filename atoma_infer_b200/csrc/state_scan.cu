// Matrix-state recurrences of the parallel and summed blocks (gated linear attention, gated delta rule, state space) — include/atoma_hybrid.h,
// atoma_state_scan.  Every head keeps S [dim, vdim] in float32; the columns of S are independent, and a token is visited after all before it:
// every sum's order depends on the sizes alone, so a sequence's bits do not depend on how it was cut into steps or what stands beside it.
#include "common.cuh"
#include "hybrid_common.cuh"

#include "atoma_hybrid.h"

#include <algorithm>
#include <type_traits>

namespace atoma {

extern int g_hybrid_debug;   // bit 4: scans with many rows per lane

namespace {

using namespace hybrid;

// log(sigmoid(z)) = min(z, 0) - log(1 + x) with x = exp(-|z|) in [0, 1], without a branch, so that a lane's tokens overlap:
// log(1 + x) = 2 artanh(s) = 2 s (1 + s^2 / 3 + s^4 / 5 + ...), s = x / (2 + x) <= 1/3; the terms from s^16 / 17 on are below 2^-29.  The decay that comes of it is
// off by 5.2e-7 at most (tau = 1, z in [-85, 85]; 1.3e-7 with tau = 16), as it is with log1pf.  With a rounded division 4000 tokens of 32 heads take 484 us for 418.
__device__ __forceinline__ float log_sigmoid(float z) {
    const float x = expf(-fabsf(z));
    float s = __fdividef(x, 2.f + x);
    const float y = s * s;
    float p = 1.f / 15.f;
    p = fmaf(p, y, 1.f / 13.f);
    p = fmaf(p, y, 1.f / 11.f);
    p = fmaf(p, y, 1.f / 9.f);
    p = fmaf(p, y, 1.f / 7.f);
    p = fmaf(p, y, 1.f / 5.f);
    p = fmaf(p, y, 1.f / 3.f);
    s += s;
    return fminf(z, 0.f) - fmaf(s * y, p, s);
}
__device__ __forceinline__ float softplusf_(float z) { return z > 20.f ? z : log1pf(expf(z)); }

constexpr int kStagers = 4;        // staging warps of a CTA; the compute warps are NW
constexpr int kScanBuffers = 3;    // chunks in shared memory: one is walked through, one gets its scalars, one is in flight

__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// R consecutive values of a staged row as packed float32 pairs
template <int R>
__device__ __forceinline__ void unpack(const uint4 *raw, uint64_t *out, __nv_bfloat16) {
#pragma unroll
    for (int i = 0; i < R / 8; ++i) {
        const uint32_t w[4] = {raw[i].x, raw[i].y, raw[i].z, raw[i].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) out[4 * i + e] = pk2(__uint_as_float(__byte_perm(w[e], 0u, 0x1044)), __uint_as_float(w[e] & 0xffff0000u));
    }
}
template <int R>
__device__ __forceinline__ void unpack(const uint4 *raw, uint64_t *out, float) {
#pragma unroll
    for (int i = 0; i < R / 4; ++i) {
        out[2 * i] = pk2(__uint_as_float(raw[i].x), __uint_as_float(raw[i].y));
        out[2 * i + 1] = pk2(__uint_as_float(raw[i].z), __uint_as_float(raw[i].w));
    }
}

__device__ __forceinline__ void fetch_pair(const __nv_bfloat16 *p, float &x, float &y) {
    const uint32_t w = *reinterpret_cast<const uint32_t *>(p);
    x = __uint_as_float(w << 16);
    y = __uint_as_float(w & 0xffff0000u);
}
__device__ __forceinline__ void fetch_pair(const float *p, float &x, float &y) {
    const float2 w = *reinterpret_cast<const float2 *>(p);
    x = w.x;
    y = w.y;
}

// Sum over a lane's R rows of S x: groups of 8 rows, each (rows 0 1 + 4 5) and (2 3 + 6 7) as pairs, then a binary tree over the groups,
// which the lanes of the column continue by xor-shuffles.  The order is the same for 8 and for 16 rows a lane.
template <int R>
__device__ __forceinline__ float row_sum(const uint64_t *S, const uint64_t *x) {
    float gs[R / 8];
#pragma unroll
    for (int g = 0; g < R / 8; ++g) {
        const uint64_t a = fma2(S[4 * g + 2], x[4 * g + 2], mul2(S[4 * g], x[4 * g]));
        const uint64_t b = fma2(S[4 * g + 3], x[4 * g + 3], mul2(S[4 * g + 1], x[4 * g + 1]));
        float lo, hi;
        upk2(add2(a, b), lo, hi);
        gs[g] = lo + hi;
    }
#pragma unroll
    for (int w = 1; w < R / 8; w <<= 1)
#pragma unroll
        for (int g = 0; g < R / 8; g += 2 * w) gs[g] += gs[g + w];
    return gs[0];
}

// A staged token: q, k, v (of the CTA's columns) as they stand in memory, for gated linear attention its pre-activations and then the decays
// in float32, and eight scalars.  An odd number of 16-byte pieces, so that lanes that read one piece of eight tokens hit distinct banks.
template <typename T, int KIND, int R, int PW, int NW>
struct Staged {
    static constexpr int kRow = R * PW, kCols = 64 * NW / PW;
    static constexpr int kRowBytes = kRow * static_cast<int>(sizeof(T)), kColBytes = (kCols * static_cast<int>(sizeof(T)) + 15) / 16 * 16;
    static constexpr int kK = kRowBytes, kV = 2 * kRowBytes, kZ = kV + kColBytes, kDecay = kZ + (KIND == 0 ? kRowBytes : 0);
    static constexpr int kScalars = kDecay + (KIND == 0 ? kRow * 4 : 0), kEnd = kScalars + 32;
    static constexpr int kBytes = kEnd / 16 % 2 ? kEnd : kEnd + 16;
};

// The state of a CTA's columns in shared memory, where it passes through on its way (SHORT): the rows of a lane apart by what lets a column's lanes hit distinct banks.
template <int R, int PW, int NW>
struct StateTile {
    static constexpr int kCols = 64 * NW / PW, kPad = 128 / PW > 4 ? 64 / PW : 4, kPart = R * kCols + kPad, kBytes = PW * kPart * 4;
    static __device__ __forceinline__ int at(int row, int col) { return row / R * kPart + row % R * kCols + col; }
};

// Whether the compute warps hand a token's sums over to the staging warps, which add the lanes' parts and write the outputs: nine instructions of a token's 178 fewer where
// one warp a scheduler is bound by what it issues.  Only where it was measured to be faster (us, shuffles in the compute warps / handed over): delta rule of 32 heads of
// 128 x 128, 4000 and 1000 tokens 715 / 681, 184 / 176, three portions 457 / 445; state space of 64 heads of 128 x 64, 4000 tokens 508 / 473.  Eight rows a lane lose
// (16 heads 568 / 573, state space of 32 heads 355 / 392), heads of 256 and 512 too (987 / 1161, 966 / 981), and gated linear attention, whose staging warps have the decays
// to form (420 / 643).  Float32 rows: the delta rule loses in CTAs of four warps (32 heads of 128 x 128, 4000 tokens 742 / 785, two portions of 500 199 / 209) and gains in
// those of eight (32 portions of 40 tokens 245 / 233); the state space gains in both (64 heads of 128 x 64, 4000 tokens 606 / 488).
template <typename T, int KIND, int R, int PW, int NW, bool SHORT>
constexpr bool kHandOver = !SHORT && (KIND == 2 || (KIND == 1 && (sizeof(T) == 2 || NW == 8))) && R == 16 && PW == 8;
// Read-outs of a token on their way to the staging warps: the lanes' sums, a part's columns together and the parts apart by what lets half a warp's stores hit
// distinct banks, then what is added to the scaled sum of each column.
template <int PW, int NW>
struct ReadOut {
    static constexpr int kCols = 64 * NW / PW, kPart = kCols + 64 / PW, kAdd = PW * kPart, kFloats = kAdd + kCols;
};

__device__ __forceinline__ void cp_async_4(uint32_t dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}

// One CTA: NW compute and 4 staging warps for 64 NW / PW columns of one head of one sequence.  A compute lane owns R rows of two neighbouring
// columns (so a staged value is read and converted once for both); the dim rows of a column lie over PW lanes.  The staging warps copy a chunk
// of tokens two chunks ahead (cp.async, as it stands in memory) and form the scalars of the chunk that comes next; one barrier per chunk.
// Per token the delta rule's lanes form S^T k and S^T q on the state as the token before left it, all lanes of a column learn the first sum
// by PW-lane shuffles, and the write is one product and one FMA per entry:
//   q, k as projected; lengths enter as scalars: S^T khat = fk (S^T k)
//   u = beta (v - g fk S^T k);  o = g fq S^T q + (qhat . khat) u;  S <- g S + k (fk u)
// What bounds it: what one warp a scheduler issues for a token, some 170 instructions, 64 of them packed FMAs of two cycles, in 330 cycles; the chain alone (row sum,
// PW-lane shuffles of 29 cycles each, write) is 215.  Delta rule, 4096 tokens of 32 heads of 128 x 128, 699 us; before sums were handed over 733, and of that without the
// shuffles 643, the sums of S^T q 666, the conversions 678; two warps of half the rows a scheduler 811.  Shared memory delivers 128 bytes a cycle to all warps of an SM.
// Rows kept as bfloat16 in shared memory and converted per warp beat float32 rows (718 us against 729, before sums were handed over, for 4096 tokens of 32 heads of 128 x 128),
// one column a lane loses to two (924 to 1330 us).  Against one column a lane, 32 rows, rows converted and normed by the staging warps: delta
// rule 1064 -> 729 us (that case, before sums were handed over), 504 -> 289 (16 heads, 2000 tokens); state space 794 -> 365 (32 heads of 128 x 64, 4000 tokens); gated linear
// attention 752 -> 421 (32 heads of 64 x 128, 4000 tokens).
// SHORT: steps of a few tokens a sequence are bound by the states, read and written once.  What counts there is bytes on their way: four CTAs an SM (no token ahead
// in registers), and the state through shared memory in pieces of 16 bytes, since the 8 to 32 bytes of a row that a warp's columns are touch as many
// lines.  One token of 32 sequences, one column a lane / wide CTAs without this / this, us: delta rule, 32 heads of 128 x 128 (134 MB), 78 / 113 / 60; state space,
// 128 x 64, 37 / 57 / 27; gated linear attention, 64 x 128, 49 / 56 / 29; 64 heads of 64 x 64 47 / 104 / 29; of 128 sequences, 32 heads of 64 x 32, 57 / 203 / 32.
template <typename T, int KIND, int R, int PW, int NW, int NB, bool SHORT>
__global__ void __launch_bounds__(32 * (NW + kStagers), NB) state_scan_kernel(const atoma_state_scan_args a, int chunk, int buffers, int piece, int v_piece) {
    using L = Staged<T, KIND, R, PW, NW>;
    extern __shared__ __align__(16) unsigned char sm[];
    constexpr int CW = 32 / PW, COLS = L::kCols, NP = R * static_cast<int>(sizeof(T)) / 16;
    pdl_launch_dependents();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int h = blockIdx.y, b = blockIdx.z;
    const int D = static_cast<int>(a.dim), V = static_cast<int>(a.vdim), H = static_cast<int>(a.H);
    const int q0 = a.query_start[b], n = a.query_start[b + 1] - q0;
    if (n <= 0) return;
    const int jb = blockIdx.x * COLS, chunk_bytes = chunk * L::kBytes;
    using RO = ReadOut<PW, NW>;
    constexpr bool HAND = kHandOver<T, KIND, R, PW, NW, SHORT>;
    [[maybe_unused]] float *read_outs = reinterpret_cast<float *>(sm + buffers * chunk_bytes);   // of two chunks
    __shared__ float2 out_scale[HAND ? 4 : 1][HAND ? 32 : 1];                          // a token's factors of its sum and of what was written: of the chunk before, in hand and next
    if (D < L::kRow || jb + COLS > V) {                          // what lies beyond dim and vdim stays zero
        for (int i = threadIdx.x * 16; i < buffers * chunk_bytes; i += blockDim.x * 16) *reinterpret_cast<uint4 *>(sm + i) = make_uint4(0, 0, 0, 0);
        __syncthreads();
    }
    if (warp >= NW) {
        // ---- staging: warp w copies tokens [w, w + 1) chunk / 4 of every chunk and forms their scalars, four lanes a token ----
        const int w = warp - NW, mine = chunk / kStagers, tok = lane >> 2, sub = lane & 3;
        const int kvh = KIND != 0 ? h / (H / static_cast<int>(a.G)) : h;
        const T *qp = static_cast<const T *>(a.q) + kvh * D, *kp = static_cast<const T *>(a.k) + kvh * D, *vp = static_cast<const T *>(a.v) + h * V + jb;
        const T *zp = KIND == 0 ? static_cast<const T *>(a.z) + h * D : nullptr;
        const int vn = min(COLS, V - jb);
        float neg_rate = 0.f, dtb = 0.f;
        if (KIND != 0) {
            neg_rate = -expf(a.a_log[h]);
            dtb = a.dt_bias[h];
        }
        T a_now{}, b_now{}, a_next{}, b_next{};                   // gate pre-activations of token `tok`: of the chunk that gets its scalars, of the one in flight
        // lanes 0 .. 15 carry a token's q, the others its k; then four lanes a token carry v
        constexpr int size = static_cast<int>(sizeof(T));
        const int half = lane & 15, row_end = D * size, v_end = vn * size;
        const T *qk = lane < 16 ? qp : kp;
        const int64_t qk_ld = lane < 16 ? a.ld_q : a.ld_k;
        const int qk_dst = lane < 16 ? 0 : L::kK;
        auto copy_row = [&](uint32_t dst, const void *from, int at, int end, int step, int unit) {       // bytes at, at + step, .. < end of a row
            const unsigned char *src = static_cast<const unsigned char *>(from);
            for (int i = at; i < end; i += step) {
                if (unit == 16) cp_async_16(dst + i, src + i, 16);
                else cp_async_4(dst + i, src + i);
            }
        };
        // rows of no alignment: values of NR tokens, four of a lane's each, in flight
        auto copy_batch = [&](auto nr, unsigned char *dst, const T *src, int64_t ld, int cnt, int at, int end, int step) {
            constexpr int NR = decltype(nr)::value;
            for (int r = 0; r < cnt; r += NR)
                for (int i = at; i < end; i += 4 * step) {
                    T x[NR][4];
#pragma unroll
                    for (int f = 0; f < NR; ++f)
#pragma unroll
                        for (int e = 0; e < 4; ++e) x[f][e] = src[min(r + f, cnt - 1) * ld + min(i + e * step, end - 1)];
#pragma unroll
                    for (int f = 0; f < NR; ++f)
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            if (i + e * step < end && r + f < cnt) reinterpret_cast<T *>(dst + (r + f) * L::kBytes)[i + e * step] = x[f][e];
                }
        };
        auto copy_values = [&](unsigned char *dst, const T *src, int64_t ld, int cnt, int at, int end, int step) {
            if (cnt == 1) copy_batch(std::integral_constant<int, 1>{}, dst, src, ld, cnt, at, end, step);
            else copy_batch(std::integral_constant<int, 4>{}, dst, src, ld, cnt, at, end, step);
        };
        auto issue = [&](int t0, unsigned char *buf) {
            const int left = min(mine, n - t0 - w * mine);
            if (left > 0) {
                const int64_t tt = q0 + t0 + w * mine;
                unsigned char *rows = buf + w * mine * L::kBytes;
                if (piece) {
                    const T *src = qk + tt * qk_ld;
                    uint32_t dst = smem_u32(rows) + qk_dst;
#pragma unroll 4
                    for (int i = 0; i < left; ++i, src += qk_ld, dst += L::kBytes) copy_row(dst, src, half * piece, row_end, 16 * piece, piece);
                    if (KIND == 0)
                        for (int i = 0; i < left; ++i) copy_row(smem_u32(rows + i * L::kBytes + L::kZ), zp + (tt + i) * a.ld_z, lane * piece, row_end, 32 * piece, piece);
                } else {
                    copy_values(rows + qk_dst, qk + tt * qk_ld, qk_ld, left, half, D, 16);
                    if (KIND == 0) copy_values(rows + L::kZ, zp + tt * a.ld_z, a.ld_z, left, lane, D, 32);
                }
                if (v_piece) {
                    if (tok < left) copy_row(smem_u32(rows + tok * L::kBytes + L::kV), vp + (tt + tok) * a.ld_v, sub * v_piece, v_end, 4 * v_piece, v_piece);
                } else {
                    copy_values(rows + L::kV, vp + tt * a.ld_v, a.ld_v, left, lane, vn, 32);
                }
                if (tok < left) {
                    if (KIND == 1) b_next = static_cast<const T *>(a.b_pre)[(tt + tok) * a.ld_b + h];
                    if (KIND != 0) a_next = static_cast<const T *>(a.a_pre)[(tt + tok) * a.ld_a + h];
                }
            }
            cp_async_commit();
        };
        auto scalars = [&](int t0, unsigned char *buf) {
            const int left = min(mine, n - t0 - w * mine);
            if (KIND == 0) {
                const float inv_tau = 1.0f / a.tau;
                unsigned char *rows = buf + w * mine * L::kBytes;
                // eight or four decays at a time, all loads before the first store: of one channel's tokens, or of one token's channels where a
                // warp has few tokens
                if (mine > 4) {
                    for (int c = lane; c < D; c += 32) {
                        const float zb = a.z_bias[h * D + c];
                        float z[8];
#pragma unroll
                        for (int e = 0; e < 8; ++e) z[e] = to_f(reinterpret_cast<const T *>(rows + max(0, min(e, left - 1)) * L::kBytes + L::kZ)[c]) + zb;
#pragma unroll
                        for (int e = 0; e < 8; ++e) z[e] = expf(log_sigmoid(z[e]) * inv_tau);
#pragma unroll
                        for (int e = 0; e < 8; ++e)
                            if (e < left) reinterpret_cast<float *>(rows + e * L::kBytes + L::kDecay)[c] = z[e];
                    }
                } else {
                    for (int i = 0; i < left; ++i)
                        for (int c = lane; c < D; c += 128) {
                            float z[4];
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                const int at = min(c + 32 * e, D - 1);
                                z[e] = to_f(reinterpret_cast<const T *>(rows + i * L::kBytes + L::kZ)[at]) + a.z_bias[h * D + at];
                            }
#pragma unroll
                            for (int e = 0; e < 4; ++e) z[e] = expf(log_sigmoid(z[e]) * inv_tau);
#pragma unroll
                            for (int e = 0; e < 4; ++e)
                                if (c + 32 * e < D) reinterpret_cast<float *>(rows + i * L::kBytes + L::kDecay)[c + 32 * e] = z[e];
                        }
                }
            }
            unsigned char *row = buf + (w * mine + min(tok, mine - 1)) * L::kBytes;
            // four lanes a token, every fourth piece of its rows each: a lane's pieces in order, then the lanes by xor-shuffles
            uint64_t sq2 = 0, sk2 = 0, dot2 = 0;
#pragma unroll 4
            for (int p = sub; p < L::kRowBytes / 16; p += 4) {
                constexpr int E = 16 / static_cast<int>(sizeof(T));
                uint64_t qv[E / 2], kv[E / 2];
                const uint4 qr = *reinterpret_cast<const uint4 *>(row + p * 16), kr = *reinterpret_cast<const uint4 *>(row + L::kK + p * 16);
                unpack<E>(&qr, qv, T{});
                unpack<E>(&kr, kv, T{});
#pragma unroll
                for (int e = 0; e < E / 2; ++e) {
                    if (KIND == 1) {
                        sq2 = fma2(qv[e], qv[e], sq2);
                        sk2 = fma2(kv[e], kv[e], sk2);
                    }
                    dot2 = fma2(qv[e], kv[e], dot2);
                }
            }
            float x, y, sq, sk, dot;
            upk2(sq2, x, y), sq = x + y;
            upk2(sk2, x, y), sk = x + y;
            upk2(dot2, x, y), dot = x + y;
#pragma unroll
            for (int o = 1; o < 4; o <<= 1) {
                if (KIND == 1) {
                    sq += __shfl_xor_sync(0xffffffffu, sq, o);
                    sk += __shfl_xor_sync(0xffffffffu, sk, o);
                }
                dot += __shfl_xor_sync(0xffffffffu, dot, o);
            }
            if (sub == 0 && tok < left) {
                float4 *s = reinterpret_cast<float4 *>(row + L::kScalars);
                float2 *scale = HAND ? &out_scale[t0 / chunk & 3][w * mine + tok] : nullptr;
                if (KIND == 0) {
                    s[0] = make_float4(a.q_scale, dot * a.q_scale, 0.f, 0.f);
                } else if (KIND == 2) {
                    const float step = softplusf_(to_f(a_now) + dtb);
                    const float g = expf(neg_rate * step);
                    if (HAND) *scale = make_float2(g * a.q_scale, 1.f);   // what is added comes whole
                    s[0] = make_float4(g, step, g * a.q_scale, dot * a.q_scale);
                } else {
                    const float fq = a.q_scale / sqrtf(sq + a.unit_eps), fk = 1.0f / sqrtf(sk + a.unit_eps);   // unit length per head, the query scaled
                    const float g = expf(neg_rate * softplusf_(to_f(a_now) + dtb));
                    s[0] = make_float4(g, g * fk, sigmoidf_(to_f(b_now)), fk);
                    if (HAND) *scale = make_float2(g * fq, dot * fq * fk);
                    s[1] = make_float4(g * fq, dot * fq * fk, 0.f, 0.f);
                }
            }
        };
        // the read-outs of this warp's tokens of chunk t0: the parts by a binary tree, as lanes add them by xor-shuffles
        [[maybe_unused]] auto read_out = [&](int t0) {
            const int left = min(mine, n - t0 - w * mine), c = t0 / chunk;
            const float *from = read_outs + ((c & 1) * chunk + w * mine) * RO::kFloats;
            const int64_t out_ld = static_cast<int64_t>(H) * V;
            float *out = a.out + (static_cast<int64_t>(q0) + t0 + w * mine) * out_ld + h * V + jb;
#pragma unroll 2
            for (int i = lane; i < left * COLS; i += 32) {
                const int t = i / COLS, col = i % COLS;
                const float *r = from + t * RO::kFloats + col;
                float o[PW];
#pragma unroll
                for (int p = 0; p < PW; ++p) o[p] = r[p * RO::kPart];
#pragma unroll
                for (int x = 1; x < PW; x <<= 1)
#pragma unroll
                    for (int p = 0; p < PW; p += 2 * x) o[p] += o[p + x];
                const float2 f = out_scale[c & 3][w * mine + t];
                if (jb + col < V) out[t * out_ld + col] = fmaf(f.x, o[0], f.y * r[RO::kAdd]);
            }
        };
        issue(0, sm);
        a_now = a_next, b_now = b_next;
        issue(chunk, sm + chunk_bytes);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncwarp();
        scalars(0, sm);
        __syncthreads();
        int cur = 0;
        for (int t0 = 0; t0 < n; t0 += chunk) {
            const int nxt = cur + 1 == kScanBuffers ? 0 : cur + 1, far = nxt + 1 == kScanBuffers ? 0 : nxt + 1;
            a_now = a_next, b_now = b_next;
            issue(t0 + 2 * chunk, sm + far * chunk_bytes);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncwarp();
            if (t0 + chunk < n) scalars(t0 + chunk, sm + nxt * chunk_bytes);
            if constexpr (HAND)
                if (t0 > 0) read_out(t0 - chunk);
            cur = nxt;
            __syncthreads();
        }
        if constexpr (HAND) read_out((n - 1) / chunk * chunk);
        return;
    }
    // ---- compute: rows part * R + r of columns j and j + 1 ----
    const int part = lane / CW, jl = (warp * CW + lane % CW) * 2, j = jb + jl;
    const float skip = KIND == 2 && a.skip ? a.skip[h] : 0.f;
    float *S_g = a.state + static_cast<int64_t>(a.state_slots[b]) * a.state_stride + static_cast<int64_t>(h) * D * V;
    const bool pair_ok = V % 2 == 0 && reinterpret_cast<uintptr_t>(S_g) % 8 == 0;
    using Tile = StateTile<R, PW, NW>;
    const bool through = SHORT && V % 4 == 0 && reinterpret_cast<uintptr_t>(S_g) % 16 == 0;
    float *tile = reinterpret_cast<float *>(sm + buffers * chunk_bytes);
    // the compute warps' pieces of 16 bytes of the CTA's columns, a row's one after the other
    auto each_piece = [&](auto f) {
        constexpr int kPer = COLS / 4;
        for (int i = threadIdx.x; i < D * kPer; i += 32 * NW) {
            const int row = i / kPer, c = i % kPer * 4;
            if (jb + c < V) f(tile + Tile::at(row, c), S_g + static_cast<int64_t>(row) * V + jb + c);
        }
    };
    uint64_t Sa[R / 2], Sb[R / 2];
    if (a.context_lens[b] == 0) {
#pragma unroll
        for (int i = 0; i < R / 2; ++i) Sa[i] = Sb[i] = 0;
    } else if (through) {
        each_piece([](float *t, const float *g) { cp_async_16(smem_u32(t), g, 16); });
        cp_async_commit();
        cp_async_wait_all();
        asm volatile("bar.sync 1, %0;" ::"n"(32 * NW) : "memory");
#pragma unroll
        for (int i = 0; i < R / 2; ++i) {
            float2 x[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int row = part * R + 2 * i + e;
                x[e] = make_float2(0.f, 0.f);
                if (row < D && j < V) x[e] = *reinterpret_cast<const float2 *>(tile + Tile::at(row, jl));
            }
            Sa[i] = pk2(x[0].x, x[1].x);
            Sb[i] = pk2(x[0].y, x[1].y);
        }
    } else {
#pragma unroll
        for (int i = 0; i < R / 2; ++i) {
            float2 x[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int row = part * R + 2 * i + e;
                const float *p = S_g + static_cast<int64_t>(row) * V + j;
                x[e] = make_float2(0.f, 0.f);
                if (row < D) {
                    if (pair_ok) {
                        if (j < V) x[e] = *reinterpret_cast<const float2 *>(p);
                    } else {
                        if (j < V) x[e].x = p[0];
                        if (j + 1 < V) x[e].y = p[1];
                    }
                }
            }
            Sa[i] = pk2(x[0].x, x[1].x);
            Sb[i] = pk2(x[0].y, x[1].y);
        }
    }
    const int jo = jb + jl + (part & 1);                          // the column whose read-out this lane writes (parts 0 and 1)
    const int64_t out_ld = static_cast<int64_t>(H) * V;
    float *out = a.out + static_cast<int64_t>(q0 - 1) * out_ld + h * V + jo;   // of the token before the one in hand
    const bool writes = part < 2 && jo < V;
    // The read-out of a token: a lane's sums go to the staging warps (HAND), or its
    // sums over the lanes are shuffled beside the next token's, so that their latencies are one.  Each of two
    // neighbouring parts takes one column: o_mine + the neighbour's o_give, over the lanes, times o_scale, plus o_add.
    float o_mine = 0.f, o_give = 0.f, o_scale = 0.f, o_add = 0.f;
    __syncthreads();
    int cur = 0;
    for (int t0 = 0; t0 < n; t0 += chunk) {
        const unsigned char *buf = sm + cur * chunk_bytes;
        [[maybe_unused]] float *ro_t = nullptr;
        if constexpr (HAND) ro_t = read_outs + (t0 / chunk & 1) * chunk * RO::kFloats + part * RO::kPart + jl;
        const int nt = min(chunk, n - t0);
        struct {
            uint4 k[NP], q[NP];
            float4 s0;
            float2 s1;
            float va, vb;
            ulonglong2 d[KIND == 0 ? R / 4 : 1];
        } tk;
        auto fetch = [&](int i) {
            const unsigned char *row = buf + i * L::kBytes;
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                tk.k[p] = *reinterpret_cast<const uint4 *>(row + L::kK + (part * NP + p) * 16);
                tk.q[p] = *reinterpret_cast<const uint4 *>(row + (part * NP + p) * 16);
            }
            if (KIND == 0) {
#pragma unroll
                for (int p = 0; p < R / 4; ++p) tk.d[p] = *reinterpret_cast<const ulonglong2 *>(row + L::kDecay + part * R * 4 + p * 16);
            }
            tk.s0 = *reinterpret_cast<const float4 *>(row + L::kScalars);
            if (KIND == 1 && !HAND) tk.s1 = *reinterpret_cast<const float2 *>(row + L::kScalars + 16);
            fetch_pair(reinterpret_cast<const T *>(row + L::kV) + jl, tk.va, tk.vb);
        };
        if (!SHORT) fetch(0);
        constexpr int kUnroll = SHORT ? 1 : HAND ? (KIND == 1 ? 6 : 8) : 4;   // delta rule, handed over, 4, 5, 6, 7, 8: 725, 716, 701, 728, 711 us (16: 1148, the instruction cache, whose edge an edit of the loop moves: time these again then)
#pragma unroll kUnroll
        for (int i = 0; i < nt; ++i) {
            if (SHORT) fetch(i);   // registers for more warps instead of a token ahead
            uint64_t k2[R / 2], q2[R / 2], d2[KIND == 0 ? R / 2 : 1];
            unpack<R>(tk.k, k2, T{});
            unpack<R>(tk.q, q2, T{});
            if (KIND == 0) {
#pragma unroll
                for (int p = 0; p < R / 4; ++p) {
                    d2[2 * p] = tk.d[p].x;
                    d2[2 * p + 1] = tk.d[p].y;
                }
            }
            const float4 s0 = tk.s0;
            const float2 s1 = tk.s1;
            const float va = tk.va, vb = tk.vb;
            if (!SHORT) fetch(min(i + 1, nt - 1));
            float o = o_mine;
            float ua, ub, wa, wb;                                  // written rows of both columns, before and with the key's length
            uint64_t g2 = 0;
            if (KIND == 1) {
                float ka = row_sum<R>(Sa, k2), kb = row_sum<R>(Sb, k2);
                if (!HAND) o += __shfl_xor_sync(0xffffffffu, o_give, CW);
#pragma unroll
                for (int x = CW; x < 32; x <<= 1) {
                    ka += __shfl_xor_sync(0xffffffffu, ka, x);
                    kb += __shfl_xor_sync(0xffffffffu, kb, x);
                    if (!HAND && x > CW) o += __shfl_xor_sync(0xffffffffu, o, x);
                }
                ua = s0.z * fmaf(-s0.y, ka, va);                   // the decayed state's answer to k
                ub = s0.z * fmaf(-s0.y, kb, vb);
                wa = s0.w * ua;
                wb = s0.w * ub;
                g2 = pk2(s0.x, s0.x);
            } else {
                if (!HAND) {
                    o += __shfl_xor_sync(0xffffffffu, o_give, CW);
#pragma unroll
                    for (int x = 2 * CW; x < 32; x <<= 1) o += __shfl_xor_sync(0xffffffffu, o, x);
                }
                wa = ua = KIND == 2 ? s0.y * va : va;
                wb = ub = KIND == 2 ? s0.y * vb : vb;
                if (KIND == 2) g2 = pk2(s0.x, s0.x);
                if (KIND == 0) {
#pragma unroll
                    for (int p = 0; p < R / 2; ++p) q2[p] = mul2(q2[p], d2[p]);
                }
            }
            if (!HAND) {
                if (writes && t0 + i > 0) *out = fmaf(o_scale, o, o_add);
                out += out_ld;
            }
            const float qa = row_sum<R>(Sa, q2), qb = row_sum<R>(Sb, q2);
            if constexpr (HAND) {
                *reinterpret_cast<float2 *>(ro_t + i * RO::kFloats) = make_float2(qa, qb);
                const float add_a = KIND == 2 ? fmaf(skip, va, s0.w * ua) : ua, add_b = KIND == 2 ? fmaf(skip, vb, s0.w * ub) : ub;
                if (part == 0) *reinterpret_cast<float2 *>(ro_t + i * RO::kFloats + RO::kAdd) = make_float2(add_a, add_b);
            } else {
                o_mine = (part & 1) ? qb : qa;
                o_give = (part & 1) ? qa : qb;
                o_scale = KIND == 1 ? s1.x : (KIND == 2 ? s0.z : s0.x);
                o_add = (KIND == 1 ? s1.y : (KIND == 2 ? s0.w : s0.y)) * ((part & 1) ? ub : ua);
                if (KIND == 2) o_add = fmaf(skip, (part & 1) ? vb : va, o_add);
            }
            const uint64_t wa2 = pk2(wa, wa), wb2 = pk2(wb, wb);
#pragma unroll
            for (int p = 0; p < R / 2; ++p) {
                Sa[p] = fma2(KIND == 0 ? d2[p] : g2, Sa[p], mul2(k2[p], wa2));
                Sb[p] = fma2(KIND == 0 ? d2[p] : g2, Sb[p], mul2(k2[p], wb2));
            }
        }
        cur = cur + 1 == kScanBuffers ? 0 : cur + 1;
        __syncthreads();
    }
    if (!HAND) {
        o_mine += __shfl_xor_sync(0xffffffffu, o_give, CW);
#pragma unroll
        for (int x = 2 * CW; x < 32; x <<= 1) o_mine += __shfl_xor_sync(0xffffffffu, o_mine, x);
        if (writes) *out = fmaf(o_scale, o_mine, o_add);
    }
#pragma unroll
    for (int i = 0; i < R / 2; ++i) {
        float2 x[2];
        upk2(Sa[i], x[0].x, x[1].x);
        upk2(Sb[i], x[0].y, x[1].y);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int row = part * R + 2 * i + e;
            float *p = S_g + static_cast<int64_t>(row) * V + j;
            if (row < D) {
                if (through) {
                    *reinterpret_cast<float2 *>(tile + Tile::at(row, jl)) = x[e];
                } else if (pair_ok) {
                    if (j < V) *reinterpret_cast<float2 *>(p) = x[e];
                } else {
                    if (j < V) p[0] = x[e].x;
                    if (j + 1 < V) p[1] = x[e].y;
                }
            }
        }
    }
    if (through) {   // a warp stores other warps' entries
        asm volatile("bar.sync 1, %0;" ::"n"(32 * NW) : "memory");
        each_piece([](const float *t, float *g) { *reinterpret_cast<float4 *>(g) = *reinterpret_cast<const float4 *>(t); });
    }
}

// the longest portion where every one of the B sequences has a token (one without makes another longer: nothing but speed may depend on this)
int64_t longest_portion(const atoma_state_scan_args &a) { return std::max<int64_t>(1, a.T - (a.B - 1)); }

template <typename T, int KIND, int R, int PW, int NW, int NB, bool SHORT = false>
cudaError_t launch_scan(const atoma_state_scan_args &a, cudaStream_t stream) {
    using L = Staged<T, KIND, R, PW, NW>;
    // staged tokens per buffer: at most 32, no more than the longest portion can have, and NB CTAs' buffers fit one SM
    constexpr int kOutBytes = kHandOver<T, KIND, R, PW, NW, SHORT> ? 2 * ReadOut<PW, NW>::kFloats * 4 : 0;
    const int64_t fit = 200 * 1024 / NB / (kScanBuffers * L::kBytes + kOutBytes);
    const int chunk = SHORT ? 4 : static_cast<int>(std::max<int64_t>(4, std::min<int64_t>({32, (longest_portion(a) + 3) / 4 * 4, fit / 4 * 4})));
    const int buffers = a.T <= chunk ? 1 : kScanBuffers;   // a step of one chunk fills the first only (whatever share of it is whose: a sequence may have no token)
    const size_t smem = static_cast<size_t>(buffers) * chunk * L::kBytes + (SHORT ? StateTile<R, PW, NW>::kBytes : chunk * kOutBytes);
    if (smem > 48 * 1024) cudaFuncSetAttribute(state_scan_kernel<T, KIND, R, PW, NW, NB, SHORT>, cudaFuncAttributeMaxDynamicSharedMemorySize, 208 * 1024);
    // copies in pieces of 16 bytes where every row and size allows it, else of 4, else value by value
    const int64_t size = sizeof(T);
    auto row = [&](const void *p, int64_t ld, int64_t cols, int64_t piece) {
        return !p || (reinterpret_cast<uintptr_t>(p) % piece == 0 && ld * size % piece == 0 && cols * size % piece == 0);
    };
    auto rows = [&](int64_t piece) { return row(a.q, a.ld_q, a.dim, piece) && row(a.k, a.ld_k, a.dim, piece) && (KIND != 0 || row(a.z, a.ld_z, a.dim, piece)); };
    const int piece = rows(16) ? 16 : (rows(4) ? 4 : 0), v_piece = row(a.v, a.ld_v, a.vdim, 16) ? 16 : (row(a.v, a.ld_v, a.vdim, 4) ? 4 : 0);
    const dim3 grid(static_cast<unsigned>((a.vdim + L::kCols - 1) / L::kCols), static_cast<unsigned>(a.H), static_cast<unsigned>(a.B));
    return launch_ex(state_scan_kernel<T, KIND, R, PW, NW, NB, SHORT>, grid, dim3(32 * (NW + kStagers)), smem, stream, a, chunk, buffers, piece, v_piece);
}

// How the state is split.  Sixteen rows a lane need the fewest instructions per entry and one shuffle fewer; eight rows a lane put the state on
// twice the warps, and serve steps that leave half of the SMs idle (us, eight / sixteen: delta rule of 16 heads, 2000 tokens 289 / 363; state space of
// 32 heads, 4000 tokens 365 / 518; where sixteen fill the SMs once it is 876 / 727, 301 / 266), and steps of more than a wave whose heads are too narrow
// for the columns of eight warps (32 sequences of 40 tokens, 16 heads of 64 x 64, eight rows / sixteen in wide CTAs 41 / 66, 32 heads of 64 x 32 41 / 117).  CTAs of eight
// warps share the staging and keep two warps a scheduler: for more than a wave of CTAs (500 + 500 tokens 194 / 164); between one and two waves a long
// portion stays with the narrow CTAs, since the sequences' lengths, which only the device knows, may leave wide ones alone on an SM (900, 700, 300 and 105
// tokens of 16 heads 193 / 285, 500 + 500 tokens of 32 heads the other way round).  Steps of four tokens a sequence and less in the mean go by kShort, though one of them
// may be long (32 sequences of 1, 2, 4 tokens, eight rows or wide CTAs / short, us: 113 / 60, 117 / 68, 125 / 80; 31 of one token beside one of 60 129 / 97).
enum class Split { kEight, kSixteen, kSixteenWide, kShort };

template <typename T, int KIND>
cudaError_t launch_split(const atoma_state_scan_args &a, Split split, cudaStream_t stream) {
    if (split == Split::kShort)
        return a.dim <= 64    ? launch_scan<T, KIND, 8, 8, 4, 4, true>(a, stream)
               : a.dim <= 128 ? launch_scan<T, KIND, 8, 16, 4, 4, true>(a, stream)
               : a.dim <= 256 ? launch_scan<T, KIND, 8, 32, 4, 4, true>(a, stream)
                              : launch_scan<T, KIND, 16, 32, 4, 2, true>(a, stream);
    if (split == Split::kEight)
        return a.dim <= 64 ? launch_scan<T, KIND, 8, 8, 4, 2>(a, stream) : a.dim <= 128 ? launch_scan<T, KIND, 8, 16, 4, 2>(a, stream) : launch_scan<T, KIND, 8, 32, 4, 2>(a, stream);
    if (split == Split::kSixteenWide)
        return a.dim <= 64 ? launch_scan<T, KIND, 16, 4, 8, 1>(a, stream) 
               : a.dim <= 128 ? launch_scan<T, KIND, 16, 8, 8, 1>(a, stream)
               : a.dim <= 256 ? launch_scan<T, KIND, 16, 16, 8, 1>(a, stream)
                              : launch_scan<T, KIND, 16, 32, 8, 1>(a, stream);
    return a.dim <= 64    ? launch_scan<T, KIND, 16, 4, 4, 1>(a, stream)
           : a.dim <= 128 ? launch_scan<T, KIND, 16, 8, 4, 1>(a, stream)
           : a.dim <= 256 ? launch_scan<T, KIND, 16, 16, 4, 1>(a, stream)
                          : launch_scan<T, KIND, 16, 32, 4, 1>(a, stream);
}

template <typename T>
cudaError_t launch_kind(const atoma_state_scan_args &a, Split split, cudaStream_t stream) {
    return a.kind == 0 ? launch_split<T, 0>(a, split, stream) : a.kind == 1 ? launch_split<T, 1>(a, split, stream) : launch_split<T, 2>(a, split, stream);
}

}  // namespace

bool hyb_state_scan(const atoma_state_scan_args &a, cudaStream_t stream) {
    if (a.T <= 0 || a.B <= 0) return true;
    if (!hybrid::known_dtype(a.dtype, "atoma_state_scan")) return false;
    const bool gla = a.kind == 0, delta = a.kind == 1, ssm = a.kind == 2;
    if ((!gla && !delta && !ssm) || !a.q || !a.k || !a.v || !a.state || !a.state_slots || !a.query_start || !a.context_lens || !a.out || a.H <= 0 ||
        a.dim <= 0 || a.vdim <= 0 || a.state_stride < a.H * a.dim * a.vdim || (gla && (!a.z || !a.z_bias || !(a.tau > 0.f))) ||
        (delta && !a.b_pre) ||
        (!gla && (!a.a_pre || !a.a_log || !a.dt_bias || a.G <= 0 || a.H % a.G))) {
        set_status(kErrInvalidArg, "atoma_state_scan: null argument, unknown kind %d, or a state row shorter than heads * dim * vdim", a.kind);
        return false;
    }
    if (a.dim > 512) {
        set_status(kErrUnsupported, "atoma_state_scan: a key size of %lld exceeds 512", static_cast<long long>(a.dim));
        return false;
    }
    const int pw = a.dim <= 64 ? 4 : (a.dim <= 128 ? 8 : (a.dim <= 256 ? 16 : 32)), cols = 256 / pw, sms = current_device_info().sm_count;
    const int64_t ctas = (a.vdim + cols - 1) / cols * a.H * a.B;
    Split split = Split::kSixteen;
    if (a.T <= 4 * a.B && !(g_hybrid_debug & 16)) split = Split::kShort;
    else if (a.dim <= 256 && (ctas * 2 <= sms || (ctas > sms && a.vdim <= cols)) && !(g_hybrid_debug & 16)) split = Split::kEight;
    else if (ctas > (a.dim > 256 || longest_portion(a) <= 256 ? sms : 2 * sms)) split = Split::kSixteenWide;
    const cudaError_t e = a.dtype == ATOMA_DTYPE_BF16 ? launch_kind<__nv_bfloat16>(a, split, stream) : launch_kind<float>(a, split, stream);
    return hybrid::launched(e, "state_scan_kernel");
}

}  // namespace atoma

using namespace atoma;

extern "C" void atoma_state_scan(const atoma_state_scan_args *args, atoma_stream_t stream) {
    clear_status();
    if (!args) {
        set_status(kErrInvalidArg, "atoma_state_scan: args is NULL");
        return;
    }
    hyb_state_scan(*args, static_cast<cudaStream_t>(stream));
}
