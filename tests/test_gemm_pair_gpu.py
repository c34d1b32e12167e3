"""The prompt-sized GEMM on CTA pairs (more than 128 tokens) against float64 on the same 16-bit inputs, at the edges of its tiles: token
chunks and weight tiles that end raggedly, K inside and across 64-wide blocks, strided operands, and the gated activations of its epilogue.

Tolerance per element: half a unit of the output's last place and 4e-6 of sum_k |x w| for the float32 sums (as test_gemm_gpu.py); behind an
activation the two products are rounded to 16 bits first: a relative 2^-8 of |gate| and |up| moves act(gate) up by at most
2^-8 (1.1 |gate| + |act(gate)|) |up| (1.1 bounds the derivative of silu and gelu), and the output's own rounding follows."""
import numpy as np
import pytest
import torch

from atoma_infer_b200 import _lib, hybrid_ops, ops
from helpers import randn_t, t2f32, ulp16
from test_gemm_gpu import _check

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF = torch.bfloat16


@pytest.mark.parametrize("T,N,K", [
    (129, 8, 64),          # the fewest tokens, one weight group
    (159, 264, 128),       # a second weight tile of 8 rows
    (160, 256, 72),        # K ends 8 into its second block
    (257, 1000, 200),
    (513, 250, 1024),      # columns that miss the 4-wide stores
    (1023, 3000, 328),     # more tiles than pairs, every edge ragged
    (4097, 264, 64),       # more than 16 chunks: two groups of the raster
    (192, 3072, 16384),    # the last tokens that a long K sends to the split-K kernel, and the first that it does not
    (193, 3072, 16384),
])
def test_against_float64(T, N, K):
    x = randn_t((T, K), 1, BF, DEV)
    w = randn_t((N, K), 2, BF, DEV, scale=K ** -0.5)
    _check(x, w, ops.gemm_tn(x, w), f"pair gemm T={T} N={N} K={K}")
    assert _lib.lib().atoma_gemm_pair_timeouts() == 0


def test_strided_operands_stay_inside_their_views():
    T, N, K = 300, 520, 192
    x = randn_t((T, K + 64), 3, BF, DEV)[:, 24:24 + K]
    w = randn_t((N, K + 8), 4, BF, DEV, scale=K ** -0.5)[:, 8:]
    wide = torch.full((T + 2, N + 40), 7.0, dtype=BF, device=DEV)
    y = wide[1:-1, 13:13 + N]        # rows that no 8-byte store can take
    ops.gemm_tn(x, w, out=y)
    _check(x, w, y, "strided")
    wide[1:-1, 13:13 + N] = 7.0
    assert bool((wide == 7.0).all())


@pytest.mark.parametrize("dtype", [BF, torch.float16])
@pytest.mark.parametrize("T,F,K,act", [(129, 8, 64, "silu"), (257, 136, 128, "silu"), (300, 264, 192, "clamped"), (520, 1048, 320, "silu")])
def test_gated_activations(dtype, T, F, K, act):
    if act == "clamped" and dtype != BF:
        pytest.skip("the clamped form is bfloat16 only")
    x = randn_t((T, K), 5, dtype, DEV)
    w = randn_t((2 * F, K), 6, dtype, DEV, scale=K ** -0.5)
    bias = randn_t((2 * F,), 7, torch.float32, DEV, scale=0.5) if act == "clamped" else None
    if act == "clamped":
        L = _lib.lib()
        got = torch.empty((T, F), dtype=dtype, device=DEV)
        L.atoma_gate_up_clamped(x.data_ptr(), w.data_ptr(), bias.data_ptr(), got.data_ptr(), T, F, K, K, K, F, 1.0, 1.702, 1.0, 1,
                                torch.cuda.current_stream().cuda_stream)
        assert L.atoma_last_status() == 0
    else:
        got = ops.gate_up_silu(x, w)
    xe, we = t2f32(x).astype(np.float64), t2f32(w).astype(np.float64)
    z, mag = xe @ we.T, np.abs(xe) @ np.abs(we).T
    plain = z                        # what is rounded to 16 bits: the products before their biases
    if bias is not None:
        z = z + bias.double().cpu().numpy()
    g, u = z[:, :F], z[:, F:]
    if act == "clamped":
        g, u = np.minimum(g, 1.0), np.clip(u, -1.0, 1.0) + 1.0
    a = g / (1 + np.exp(-(1.702 if act == "clamped" else 1.0) * g))
    half = 2.0 ** (-8 if dtype == BF else -11)
    slack = lambda v, m: half * np.abs(v) + 4e-6 * m
    gs, us = slack(plain[:, :F], mag[:, :F]), slack(plain[:, F:], mag[:, F:])
    bound = 0.5 * ulp16(a * u, dtype == BF) * 1.01 + 1.1 * gs * np.abs(u) + np.abs(a) * us + 1.1 * gs * us + 1e-6
    diff = np.abs(t2f32(got).astype(np.float64) - a * u)
    assert (diff <= bound).all(), f"worst excess {(diff - bound).max():.3e}"
    assert _lib.lib().atoma_gemm_pair_timeouts() == 0


@pytest.mark.parametrize("dtype", [BF, torch.float16])
def test_activation_is_float32(dtype):
    """Rows of x with one entry make both products exact, so a result differs from the rounded float64 one only where float32's error reaches over the
    middle of two neighbours: with four operations of half to one unit (2^-24; 1.1e-7 of the value in the mean) and neighbours 2^-8 to 2^-7 (2^-11 to 2^-10) of the
    value apart, in the share 2 x 1.1e-7 x 2^7.5 of the entries."""
    T, F, K = 192, 32768, 64
    x = torch.zeros((T, K), dtype=dtype, device=DEV)
    x[torch.arange(T), torch.arange(T) % K] = torch.tensor([0.5, 1.0, 2.0], dtype=dtype, device=DEV).repeat_interleave(K)
    w = randn_t((2 * F, K), 12, dtype, DEV, scale=2.0)
    got = ops.gate_up_silu(x, w)
    z = x.double() @ w.double().T
    want = (z[:, :F] / (1 + torch.exp(-z[:, :F])) * z[:, F:]).to(dtype)
    share = (got != want).double().mean().item()
    assert share < 2.2e-7 * 2.0 ** (7.5 if dtype == BF else 10.5), share


def test_activation_of_extreme_gates():
    """Gates whose exponential is huge, infinite or NaN: what float32 gives for g / (1 + e^-g) u, up to the exponential's 2 ulp and the rounding to bfloat16."""
    gates = [-300.0, -100.0, -89.0, -88.5, -88.0, -87.5, -87.0, -60.0, -0.0, 60.0, 300.0, float("-inf"), float("inf"), float("nan")]
    T, K, F = 129, 64, 16
    x, w = torch.zeros((T, K), dtype=BF, device=DEV), torch.zeros((2 * F, K), dtype=BF, device=DEV)
    for i, g in enumerate(gates):                  # column i of w alone meets row i of x; an infinity comes from a product that overflows
        big = abs(g) == float("inf")
        x[i, i] = 3e38 if big else 1.0
        w[i, i] = (3.0 if g > 0 else -3.0) if big else g
        w[F + i, i] = 2e-38 if big else 1.5
    got = ops.gate_up_silu(x, w)
    z = x.float() @ w.float().T
    g, u = z[:, :F].to(BF).float(), z[:, F:].to(BF).float()
    want = (g / (1 + torch.exp(-g)) * u).to(BF)
    for i, name in enumerate(gates):
        a, b = got[i, i].item(), want[i, i].item()
        assert (a != a and b != b) or a == b or abs(a - b) <= abs(b) * 2.0 ** -7, (name, a, b)


@pytest.mark.parametrize("scale_input", [False, True])
@pytest.mark.parametrize("T,E,top,W,F", [
    (1, 3, 2, 64, 64),         # two chunks of one row
    (33, 70, 3, 72, 136),      # more experts than chosen, K that ends inside a block, chunks of up to 64 rows
    (300, 5, 4, 136, 264),     # an expert that most tokens choose (even chunks), chunks of every width
])
def test_grouped_by_expert(T, E, top, W, F, scale_input):
    """Routed experts: crowded and empty ones, and a token that meets the same expert twice.  The bound follows the path's
    roundings: inputs (when scaled) and the activation to bfloat16 (2^-8 each of the sums' magnitudes), each pair's row to bfloat16."""
    g = torch.Generator().manual_seed(11)
    index = torch.stack([torch.randperm(E, generator=g)[:top] if top <= E else torch.zeros(top, dtype=torch.long) for _ in range(T)])
    index[: 2 * T // 3, 0] = 1
    index[T // 2:, 1] = 1
    weight = torch.rand((T, top), generator=g) + 0.1
    h = randn_t((T, W), 8, BF, DEV)
    gu = randn_t((E * 2 * F, W), 9, BF, DEV, scale=W ** -0.5).reshape(E, 2 * F, W)
    dn = randn_t((E * W, F), 10, BF, DEV, scale=F ** -0.5).reshape(E, W, F)
    got = hybrid_ops.moe_experts(h, index.to(torch.int32).to(DEV), weight.to(DEV), gu, dn, 0.0, 1.0, 0.0, scale_input=scale_input).double().cpu()
    hd, gud, dnd = h.double().cpu(), gu.double().cpu(), dn.double().cpu()
    want, bound = torch.zeros(T, W, dtype=torch.float64), torch.full((T, W), 1e-6, dtype=torch.float64)
    for t in range(T):
        for k in range(top):
            e, w = int(index[t, k]), float(weight[t, k])
            x = hd[t] * w if scale_input else hd[t]
            z = gud[e] @ x
            dz = (2.0 ** -8 if scale_input else 0.0) * (gud[e].abs() @ x.abs()) + 4e-6 * (gud[e].abs() @ x.abs())
            a = z[:F] / (1 + torch.exp(-z[:F])) * z[F:]
            da = 1.1 * dz[:F] * z[F:].abs() + z[:F].abs() * dz[F:] + 1.1 * dz[:F] * dz[F:] + 2.0 ** -8 * a.abs() * 1.01
            y = dnd[e] @ a
            dy = dnd[e].abs() @ da + 4e-6 * (dnd[e].abs() @ a.abs())
            s = 1.0 if scale_input else w
            want[t] += s * y
            bound[t] += s * dy + 2.0 ** -8 * (s * y).abs() + 2.0 ** -8 * s * dy
    diff = (got - want).abs()
    assert (diff <= bound).all(), f"worst excess {float((diff - bound).max()):.3e}"
    assert _lib.lib().atoma_gemm_pair_timeouts() == 0
