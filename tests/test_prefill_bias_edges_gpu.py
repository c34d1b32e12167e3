"""Long portions of prompt attention where a path of the softmax begins or ends: distance tables that end inside, at and beyond what is kept in shared memory,
and rows whose largest score grows from one tile of keys to the next, or by more than the reference maximum may lag behind, against float64.

Bound: the weights are rounded to bfloat16 (2^-8 of the weighted mean of |v| at most), as is the result; 1e-5 for the float32 sums, 2^-22 of the largest score
in the exponent."""
import math

import pytest
import torch

from atoma_infer_b200 import hybrid_ops as ho
from atoma_infer_b200 import ops
from helpers import randn_t

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def check(got, want, mean, score=0.0):
    diff, bound = (got.double() - want).abs(), (2.0 ** -8 * 1.01 + 1e-5 + 2.0 ** -22 * score) * mean + 2.0 ** -8 * 1.01 * want.abs() + 1e-6
    assert bool((diff <= bound).all()), f"worst excess {float((diff - bound).max()):.3e}"


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("rows,window", [(1, 0), (127, 0), (300, 500), (2048, 0), (2049, 0), (2200, 2000)])
def test_tables_that_end_inside_a_tile(D, rows, window):
    H, G, bs, seqs = 4, 2, 16, ((0, 300), (1931, 389))
    T, pages = sum(n for _, n in seqs), [-(-(c + n) // bs) for c, n in seqs]
    table = torch.zeros((2, max(pages)), dtype=torch.int32)
    table[0, :pages[0]], table[1] = torch.arange(pages[0]), torch.arange(pages[0], sum(pages))
    kc, vc = randn_t((sum(pages) * bs, G, D), 1, torch.bfloat16, DEV), randn_t((sum(pages) * bs, G, D), 2, torch.bfloat16, DEV)
    q, dist = randn_t((T, H * D), 3, torch.bfloat16, DEV), randn_t((rows, H), 5, torch.float32, DEV)
    pos = torch.cat([torch.arange(c, c + n) for c, n in seqs]).to(DEV)
    tseq = torch.arange(2, dtype=torch.int32).repeat_interleave(torch.tensor([n for _, n in seqs])).to(DEV)
    got = ho.softmax_attention_paged(q, kc, vc, pos, tseq, table.to(DEV), H, G, D, D, bs, D ** -0.5, window=window, dist_bias=dist, long_min_q=128)
    t0 = 0
    for b, (c, n) in enumerate(seqs):
        slot = (table[b].long()[torch.arange(c + n) // bs] * bs + torch.arange(c + n) % bs).to(DEV)
        k, v = (x[slot].double().transpose(0, 1).repeat_interleave(H // G, 0) for x in (kc, vc))
        i, j = c + torch.arange(n, device=DEV)[:, None], torch.arange(c + n, device=DEV)[None]
        hidden = (j > i) | ((i - j >= window) if window else (j > i))
        s = torch.bmm(q[t0:t0 + n].double().reshape(n, H, D).transpose(0, 1), k.transpose(1, 2)) * D ** -0.5
        w = torch.softmax((s + dist.double()[(i - j).clamp(0, rows - 1)].permute(2, 0, 1)).masked_fill(hidden[None], -math.inf), 2)
        check(got[t0:t0 + n], *((torch.bmm(w, x).transpose(0, 1).reshape(n, H * D)) for x in (v, v.abs())))
        t0 += n
    assert ho.prefill_timeouts() == 0


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("step", [0.5, 6.0, 40.0])
def test_scores_that_grow_from_tile_to_tile(D, step):
    """The score of a row's keys rises by `step` (in units of log 2) from one tile of 128 keys to the next, in some rows only."""
    H, G, n = 4, 2, 700
    q = 0.3 * randn_t((n, H, D), 1, torch.bfloat16, DEV)
    k = 0.3 * randn_t((n, G, D), 2, torch.bfloat16, DEV)
    v = randn_t((n, G, D), 3, torch.bfloat16, DEV)
    q[:, :, 0] = (torch.arange(n, device=DEV) % 3 == 0).to(q.dtype)[:, None] * 4.0
    k[:, :, 0] = (step * math.log(2.0) * D ** 0.5 / 4.0 * (torch.arange(n, device=DEV) // 128).float())[:, None].to(k.dtype)
    start = torch.tensor([0, n], dtype=torch.int32, device=DEV)
    got = ops.flash_attn_varlen(q, k, v, start, start, n, n, D ** -0.5, True)
    rep = lambda x: x.double().transpose(0, 1).repeat_interleave(H // G, 0)
    s = torch.bmm(q.double().transpose(0, 1), rep(k).transpose(1, 2)) * D ** -0.5
    s = s.masked_fill(torch.ones(n, n, dtype=torch.bool, device=DEV).triu(1), -math.inf)
    w = torch.softmax(s, 2)
    check(got, *(torch.bmm(w, x).transpose(0, 1) for x in (rep(v), rep(v).abs())), score=float(s[s > -math.inf].abs().max()))
    assert ho.prefill_timeouts() == 0
