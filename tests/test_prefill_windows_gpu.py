"""Long portions of windowed softmax attention with a distance table and a gate, in several query tiles and sequences, against float64: narrow windows, whose grid
goes head by head, and wide ones, whose grid goes over all heads.

Bound: the weights are rounded to bfloat16 (2^-8 of the weighted mean of |v| at most), as are the result and, where kept tokens are merged, the sums before
them; 1e-5 for the float32 sums."""
import pytest
import torch

from atoma_infer_b200 import hybrid_ops as ops
from helpers import randn_t

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("window,keep", [(40, 4), (87, 0), (600, 4), (0, 0)])
def test_against_float64(D, window, keep):
    H, G, bs, rows, seqs = 6, 3, 16, 50, ((0, 700), (300, 513), (5, 257))
    each = [-(-(c + n) // bs) for c, n in seqs]
    pool = torch.randperm(sum(each), generator=torch.Generator().manual_seed(1)).to(torch.int32)
    table, at = torch.zeros((len(seqs), max(each)), dtype=torch.int32), 0
    for b, m in enumerate(each):
        table[b, :m] = pool[at:at + m]
        at += m
    T = sum(n for _, n in seqs)
    kc, vc = randn_t((sum(each) * bs, G, D), 1, torch.bfloat16, DEV), randn_t((sum(each) * bs, G, D), 2, torch.bfloat16, DEV)
    q, gate, dist = randn_t((T, H * D), 3, torch.bfloat16, DEV), randn_t((T, H * D), 4, torch.bfloat16, DEV), randn_t((rows, H), 5, torch.float32, DEV)
    pos = torch.cat([torch.arange(c, c + n) for c, n in seqs]).to(DEV)
    tseq = torch.arange(len(seqs), dtype=torch.int32).repeat_interleave(torch.tensor([n for _, n in seqs])).to(DEV)
    got = ops.softmax_attention_paged(q, kc, vc, pos, tseq, table.to(DEV), H, G, D, D, bs, D ** -0.5, window=window, keep_first=keep, dist_bias=dist, gate=gate,
                                      long_min_q=128).double()
    t0 = 0
    for b, (c, n) in enumerate(seqs):
        p = torch.arange(c + n)
        slot = (table[b].long()[p // bs] * bs + p % bs).to(DEV)
        k, v = (x[slot].double().transpose(0, 1).repeat_interleave(H // G, 0) for x in (kc, vc))
        i, j = c + torch.arange(n, device=DEV)[:, None], torch.arange(c + n, device=DEV)[None]
        hidden = (j > i) | ((i - j >= window) & (j >= keep) if window else j > i)
        s = torch.bmm(q[t0:t0 + n].double().reshape(n, H, D).transpose(0, 1), k.transpose(1, 2)) * D ** -0.5
        w = torch.softmax((s + dist.double()[(i - j).clamp(0, rows - 1)].permute(2, 0, 1)).masked_fill(hidden[None], -float("inf")), 2)
        gt = torch.sigmoid(gate[t0:t0 + n].double())
        want, mean = ((torch.bmm(w, x).transpose(0, 1).reshape(n, H * D)) * gt for x in (v, v.abs()))
        diff, bound = (got[t0:t0 + n] - want).abs(), (2.0 ** -8 * 1.01 + 1e-5) * mean + 2.0 ** -7 * 1.01 * want.abs() + 1e-6
        assert bool((diff <= bound).all()), f"sequence {b}: worst excess {float((diff - bound).max()):.3e}"
        t0 += n
    assert ops.prefill_timeouts() == 0
