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


def one_sequence(H, G, D, n, dtype, width, others=0):
    """One sequence of n keys in a table of `width` pages, with `others` empty sequences behind it: output, log-sum-exp, and the same in float64."""
    page, need = 16, -(-n // 16)
    kv = randn_t((2, need + 1, page, G, D), 1, dtype, DEV)
    q = randn_t((1 + others, 1, H, D), 2, dtype, DEV)
    table = torch.zeros((1 + others, width), dtype=torch.int32, device=DEV)
    table[0, :need] = torch.randperm(need, generator=torch.Generator().manual_seed(3)).to(torch.int32).to(DEV)
    lens = torch.tensor([n] + [0] * others, dtype=torch.int32, device=DEV)
    out, lse = ops.flash_attn_kv_cache_full(q, kv[0], kv[1], None, D ** -0.5, table, lens, True, with_lse=True)
    assert ops.last_mha_path() == "decode_paged"
    p = torch.arange(n, device=DEV)
    k = kv[0].reshape(-1, G, D)[table[0].long()[p // page] * page + p % page].double().transpose(0, 1).repeat_interleave(H // G, 0)
    want = torch.logsumexp(torch.bmm(q[0, 0].double()[:, None], k.transpose(1, 2)) * D ** -0.5, 2)
    return out[0].clone(), lse.reshape(1 + others, H)[0].clone(), want.reshape(H)


@pytest.mark.parametrize("H,G,D,n,dtype,groups", [
    (32, 8, 64, 300, torch.bfloat16, False), (32, 8, 64, 777, torch.bfloat16, False), (32, 8, 64, 1020, torch.float16, False), (32, 8, 128, 480, torch.float16, False),
    (8, 8, 128, 150, torch.bfloat16, False), (128, 8, 128, 360, torch.bfloat16, False), (128, 8, 128, 390, torch.float16, True), (72, 8, 64, 310, torch.bfloat16, False), (16, 16, 64, 1500, torch.float16, False),
    (32, 8, 64, 4000, torch.float16, True), (128, 8, 128, 2500, torch.bfloat16, True), (8, 1, 128, 5000, torch.float16, True), (48, 24, 128, 2600, torch.float16, True),
])
def test_bits_follow_the_keys_alone(H, G, D, n, dtype, groups):
    # A sequence's keys lie on the same CTAs whatever its table could hold and however many empty sequences are beside it.  Up to a number of partials (groups = False)
    # they are merged in one order, whichever kernel does it: a wide table alone, an exact one, and six empty sequences take different ones.
    need = -(-n // 16)
    out, lse, want = one_sequence(H, G, D, n, dtype, need)
    # scores of 64 and 128 products in float32, weights and sums within a few units of 2^-22, the logarithm within 2^-21
    assert float((lse.double() - want).abs().max()) < 5e-5
    for width, others in ((need + 300, 0),) if groups else ((need + 300, 0), (need, 6), (need + 300, 6)):
        o, s, _ = one_sequence(H, G, D, n, dtype, width, others)
        assert torch.equal(o, out) and torch.equal(s, lse), (width, others)
