"""Per-head norms, rotation and cache write, a warp per share of a token's heads, against the general kernel (debug flag 2): wholly turned heads in both orders,
shares that end inside the queries, the keys and the values, several rounds a share (many tokens) and fewer heads than a round.

Bound: as both kernels form the same float32 expressions and differ in the order of a head's sum of squares, one unit of the last place of bfloat16 (2^-7 of the
value) and 2e-5 of the largest entry where a rotation cancels."""
import pytest
import torch

from atoma_infer_b200 import hybrid_ops as ops
from helpers import randn_t

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF = torch.bfloat16


@pytest.mark.parametrize("T,H,G,D,interleaved,bias", [
    (37, 32, 8, 128, True, False),       # a share is one round
    (37, 7, 7, 64, False, True),         # rounds of four heads, seven of them
    (700, 33, 11, 128, False, True),     # shares that cross from queries to keys to values
    (700, 33, 11, 256, True, False),
    (6001, 12, 4, 64, True, True),       # a warp takes the whole token
    (6001, 10, 2, 128, False, False),
])
def test_shares_against_the_general_kernel(T, H, G, D, interleaved, bias):
    N = (H + 2 * G) * D
    proj = randn_t((T, N), 1, BF, DEV)
    vec = lambda n, seed, mean: randn_t((n,), seed, torch.float32, DEV, scale=0.1) + mean
    freq, low = torch.logspace(0, -4, D // 2, device=DEV), vec(D // 2, 4, 0.0) * 1e-8
    pos, slots = torch.arange(T, device=DEV) * 7, torch.randperm(T, generator=torch.Generator().manual_seed(7)).to(DEV)
    slots[T // 2] = -1
    out = []
    for flags in (0, 2):
        k, v = (torch.full((T, G, D), 9.0, dtype=BF, device=DEV) for _ in range(2))
        ops.debug_flags(flags)
        try:
            q = ops.qkv_headnorm_rope_cache(proj, 0, H * D, (H + G) * D, vec(D, 5, 1.0), vec(D, 6, 1.0), freq, None, interleaved, pos, slots, k, v, H, G, D, D, 1e-5,
                                            bias=vec(N, 2, 0.0) if bias else None, qk_freq_lo=low)
        finally:
            ops.debug_flags(0)
        out.append((q, k, v))
    for got, want in zip(*((x.float() for x in o) for o in out)):
        assert bool(((got - want).abs() <= want.abs() * 2.0 ** -7 + 2e-5 * want.abs().max()).all())
