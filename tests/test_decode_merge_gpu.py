"""Decode attention whose partial results are merged: no more than one merge takes, several groups of them, heads of one to sixteen queries, sequences that
share a step, against float64.

Bound: the weights are rounded to bfloat16 (2^-8 of the weighted mean of |v| at most), as is the result; 1e-5 for the float32 sums."""
import pytest
import torch

from atoma_infer_b200 import ops
from helpers import randn_t

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("H,G,D,lens", [
    (32, 8, 64, [16]), (32, 8, 128, [130]), (32, 8, 64, [777]), (32, 8, 128, [1030]), (32, 8, 128, [2100]), (8, 8, 64, [4000]), (128, 8, 128, [2500]),
    (72, 8, 64, [1500, 3]), (8, 1, 128, [5000]), (16, 2, 64, [2600, 700]), (32, 8, 128, [3000, 1, 0, 900]), (32, 8, 64, [300] * 20),
])
def test_against_float64(H, G, D, lens):
    page = 16
    pages = [-(-n // page) for n in lens]
    kv = randn_t((2, sum(pages) + 1, page, G, D), 1, torch.bfloat16, DEV)
    q = randn_t((len(lens), 1, H, D), 2, torch.bfloat16, DEV)
    pool, at = torch.randperm(sum(pages), generator=torch.Generator().manual_seed(3)).to(torch.int32), 0
    table = torch.zeros((len(lens), max(pages)), dtype=torch.int32)
    for b, m in enumerate(pages):
        table[b, :m] = pool[at:at + m]
        at += m
    args = (q, kv[0], kv[1], None, D ** -0.5, table.to(DEV), torch.tensor(lens, dtype=torch.int32, device=DEV), True)
    got = ops.flash_attn_kv_cache_full(*args)
    assert ops.last_mha_path() == "decode_paged"
    assert torch.equal(ops.flash_attn_kv_cache_full(*args), got)       # whoever arrives last, and the counters are clean again
    for b, n in enumerate(lens):
        p = torch.arange(n)
        rows = (table[b].long()[p // page] * page + p % page).to(DEV)
        k, v = (x.reshape(-1, G, D)[rows].double().transpose(0, 1).repeat_interleave(H // G, 0) for x in kv)
        w = torch.softmax(torch.bmm(q[b, 0].double()[:, None], k.transpose(1, 2)) * D ** -0.5, 2)
        want, mean = (torch.bmm(w, x)[:, 0] for x in (v, v.abs()))
        diff, bound = (got[b].double().reshape(H, D) - want).abs(), (2.0 ** -8 * 1.01 + 1e-5) * mean + 2.0 ** -8 * 1.01 * want.abs() + 1e-6
        assert bool((diff <= bound).all()), f"{n} keys: worst excess {float((diff - bound).max()):.3e}"
