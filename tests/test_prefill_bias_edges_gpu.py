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


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("rows,n,context", [(2210, 300, 2100), (2049, 200, 2250), (4096, 700, 3700), (3000, 400, 1900)])
def test_tables_longer_than_their_copy(D, rows, n, context):
    """Tiles whose distances lie within the copy of the first rows and the rows behind it, across their end, between there and the table's end, and beyond that."""
    H, G, bs, m = 4, 2, 16, n + context
    kc, vc = randn_t((-(-m // bs) * bs, G, D), 1, torch.bfloat16, DEV), randn_t((-(-m // bs) * bs, G, D), 2, torch.bfloat16, DEV)
    q, dist = randn_t((n, H * D), 3, torch.bfloat16, DEV), randn_t((rows, H), 5, torch.float32, DEV)
    table, pos = torch.arange(-(-m // bs), dtype=torch.int32, device=DEV)[None], context + torch.arange(n, device=DEV)
    got = ho.softmax_attention_paged(q, kc, vc, pos, torch.zeros(n, dtype=torch.int32, device=DEV), table, H, G, D, D, bs, D ** -0.5, dist_bias=dist, long_min_q=128)
    k, v = (x[:m].double().transpose(0, 1).repeat_interleave(H // G, 0) for x in (kc, vc))
    i, j = pos[:, None], torch.arange(m, device=DEV)[None]
    s = torch.bmm(q.double().reshape(n, H, D).transpose(0, 1), k.transpose(1, 2)) * D ** -0.5
    w = torch.softmax((s + dist.double()[(i - j).clamp(0, rows - 1)].permute(2, 0, 1)).masked_fill((j > i)[None], -math.inf), 2)
    check(got, *((torch.bmm(w, x).transpose(0, 1).reshape(n, H * D)) for x in (v, v.abs())))
    assert ho.prefill_timeouts() == 0


def halves(case, n, step, dev):
    """What 64 keys at a time (a thread's share of a tile) add to the score, in units of log 2."""
    h = torch.arange(n, device=dev) // 64
    if case == "rising":
        return step * h.float()
    low = (h % 2 == 1) if case == "first" else (h % 2 == 0) if case == "second" else ((h // 2 + h) % 2 == 1)   # the half that never holds the largest score
    return step * (h // 2).float() - 24.0 * low.float()


@pytest.mark.parametrize("case", ["rising", "first", "second", "alternate"])
@pytest.mark.parametrize("D,step,form", [(64, 3.0, "paged"), (128, 12.0, "paged"), (64, 12.0, "bias"), (128, 3.0, "bias"), (128, 12.0, "bias")])
def test_largest_scores_in_one_half_of_the_tiles(D, step, form, case):
    """Two threads share a row's scores where pages or a distance table are read: each has to learn of the other's maximum, in every tile and behind the last."""
    H, G, n, bs = 4, 2, 900, 16
    pages = -(-n // bs)
    q = 0.3 * randn_t((n, H, D), 1, torch.bfloat16, DEV)
    kc = 0.3 * randn_t((pages, bs, G, D), 2, torch.bfloat16, DEV)
    vc = randn_t((pages, bs, G, D), 3, torch.bfloat16, DEV)
    order = torch.randperm(pages, generator=torch.Generator().manual_seed(4)).to(DEV)
    slot = order[torch.arange(n, device=DEV) // bs] * bs + torch.arange(n, device=DEV) % bs
    q[:, :, 0] = (torch.arange(n, device=DEV) % 3 != 1).to(q.dtype)[:, None] * 4.0
    kc.view(-1, G, D)[slot, :, 0] = (halves(case, n, step, DEV) * math.log(2.0) * D ** 0.5 / 4.0)[:, None].to(kc.dtype)
    k, v = (x.reshape(-1, G, D)[slot].double().transpose(0, 1).repeat_interleave(H // G, 0) for x in (kc, vc))
    i, j = torch.arange(n, device=DEV)[:, None], torch.arange(n, device=DEV)[None]
    s = torch.bmm(q.double().transpose(0, 1), k.transpose(1, 2)) * D ** -0.5
    table = order.to(torch.int32)[None].contiguous()
    if form == "paged":
        start = torch.tensor([0, n], dtype=torch.int32, device=DEV)
        got = ops.flash_attn_varlen_with_block_table(q, kc, vc, None, start, start, n, n, D ** -0.5, None, 0, table)
    else:
        dist = randn_t((300, H), 5, torch.float32, DEV)
        pos, tseq = torch.arange(n, device=DEV), torch.zeros(n, dtype=torch.int32, device=DEV)
        got = ho.softmax_attention_paged(q.reshape(n, H * D), kc.view(-1, G, D), vc.view(-1, G, D), pos, tseq, table, H, G, D, D, bs, D ** -0.5, dist_bias=dist, long_min_q=128)
        s = s + dist.double()[(i - j).clamp(0, 299)].permute(2, 0, 1)
    s = s.masked_fill((j > i)[None], -math.inf)
    w = torch.softmax(s, 2)
    check(got.reshape(n, H, D), *(torch.bmm(w, x).transpose(0, 1) for x in (v, v.abs())), score=float(s[s > -math.inf].abs().max()))
    assert ho.prefill_timeouts() == 0
