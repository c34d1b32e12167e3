"""Prompt attention through block tables on the tensor-memory prefill kernel: against the same kernel on pages in order, where every output must be the
same to the bit whatever the pages' size and order, and against float64.  Cache rows that belong to no sequence hold NaN: none may reach a
product."""
import pytest
import torch

from atoma_infer_b200 import hybrid_ops, ops
from helpers import randn_t

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("H,G,page,news,contexts", [
    (4, 2, 16, (129, 1, 256), (0, 700, 128)),          # one row past a tile, a decoded token, whole tiles behind whole tiles
    (3, 1, 48, (300, 33, 127), (5, 0, 129)),           # pages that straddle tiles
    (2, 2, 256, (640,), (1000,)),                      # pages of two tiles, two query tiles and a half
    (8, 8, 16, (32, 31), (0, 95)),                     # less than one tile
])
def test_same_bits_whatever_the_pages(D, dtype, H, G, page, news, contexts):
    lens = [n + c for n, c in zip(news, contexts)]
    T = sum(news)
    q = randn_t((T, H, D), 1, dtype, DEV)
    k, v = randn_t((sum(lens), G, D), 2, dtype, DEV), randn_t((sum(lens), G, D), 3, dtype, DEV)
    each = [-(-n // page) for n in lens]
    pool = torch.randperm(sum(each) + 2, generator=torch.Generator().manual_seed(4)).to(torch.int32)
    kc, vc = (torch.full((sum(each) + 2, page, G, D), float("nan"), dtype=dtype, device=DEV) for _ in range(2))
    table, used, row = torch.zeros((len(lens), max(each)), dtype=torch.int32), 0, 0
    for b, n in enumerate(lens):
        table[b, :each[b]] = pool[used:used + each[b]]
        at = torch.arange(n)
        slot = (table[b].long()[at // page] * page + at % page).to(DEV)
        kc.view(-1, G, D)[slot], vc.view(-1, G, D)[slot] = k[row:row + n], v[row:row + n]
        used, row = used + each[b], row + n
    starts = lambda x: torch.tensor([sum(x[:i]) for i in range(len(x) + 1)], dtype=torch.int32, device=DEV)
    args = (starts(news), starts(lens), max(news), max(lens), D ** -0.5)
    got = ops.flash_attn_varlen_with_block_table(q, kc, vc, None, *args, None, 0, table.to(DEV))
    assert ops.last_mha_path() == "prefill_tc"
    wide = -(-max(lens) // 16) * 16                    # one page per sequence
    kw, vw = (torch.full((len(lens), wide, G, D), float("nan"), dtype=dtype, device=DEV) for _ in range(2))
    at = 0
    for b, n in enumerate(lens):
        kw[b, :n], vw[b, :n] = k[at:at + n], v[at:at + n]
        at += n
    order = torch.arange(len(lens), dtype=torch.int32, device=DEV)[:, None]
    assert torch.equal(got, ops.flash_attn_varlen_with_block_table(q, kw, vw, None, *args, None, 0, order))
    _check(got, q, k, v, news, contexts)
    assert hybrid_ops.prefill_timeouts() == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("H,G,page,news,contexts,gathered", [
    (4, 2, 16, (256,), (1792,), True),                           # the shortest step that is gathered
    (3, 1, 48, (300, 1, 33), (2100, 0, 1991), False),            # what so few rows save is not sure to pay for three sequences' keys
    (2, 2, 256, (1000, 640), (1100, 1408), False),
    (2, 1, 48, (4000, 3900, 1), (0, 100, 2500), True),           # pages that straddle tiles, a decoded token, a sequence that ends inside a tile
    (2, 1, 16, (3000, 2950), (72, 122), True),                   # both end with a whole tile
    (32, 32, 16, (256,), (1792,), False),                        # many key heads: the copy is the larger part
])
def test_gathered_steps_give_the_bits_of_pages(dtype, H, G, page, news, contexts, gathered):
    """A bound on the longest sequence that would take too much scratch leaves the step on its pages, as does a capture, whose graph may be replayed beside other work on the
    capture's stream; rows behind a sequence's end and unused pages hold NaN."""
    D, lens = 128, [n + c for n, c in zip(news, contexts)]
    q = randn_t((sum(news), H, D), 1, dtype, DEV)
    each = [-(-n // page) for n in lens]
    pool = torch.randperm(sum(each) + 2, generator=torch.Generator().manual_seed(4)).to(torch.int32)
    kc, vc = (torch.full((sum(each) + 2, page, G, D), float("nan"), dtype=dtype, device=DEV) for _ in range(2))
    k, v = randn_t((sum(lens), G, D), 2, dtype, DEV), randn_t((sum(lens), G, D), 3, dtype, DEV)
    table, used, row = torch.zeros((len(lens), max(each)), dtype=torch.int32), 0, 0
    for b, n in enumerate(lens):
        table[b, :each[b]] = pool[used:used + each[b]]
        at = torch.arange(n)
        slot = (table[b].long()[at // page] * page + at % page).to(DEV)
        kc.view(-1, G, D)[slot], vc.view(-1, G, D)[slot] = k[row:row + n], v[row:row + n]
        used, row = used + each[b], row + n
    starts = lambda x: torch.tensor([sum(x[:i]) for i in range(len(x) + 1)], dtype=torch.int32, device=DEV)
    args = q, kc, vc, None, starts(news), starts(lens)
    table = table.to(DEV)

    def run(longest, longest_q=max(news)):
        ops.reset_launch_count()
        return ops.flash_attn_varlen_with_block_table(*args, longest_q, longest, D ** -0.5, None, 0, table)

    got = run(max(lens))
    assert ops.last_mha_path() == "prefill_tc" and ops.launch_count() == (2 if gathered else 1)      # a copy, then the products
    assert torch.equal(got, run(1 << 22)) and ops.launch_count() == 1
    if len(news) == 1:                                                         # a loose bound on the portion saves nothing
        assert torch.equal(got, run(max(lens), max(news) + 8192)) and ops.launch_count() == (2 if gathered else 1)
    assert torch.equal(got, run(2048))                                         # a bound that some sequences exceed
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        again = run(max(lens))
    assert ops.launch_count() == 1
    graph.replay()
    assert torch.equal(got, again)
    _check(got, q, k, v, news, contexts)
    assert hybrid_ops.prefill_timeouts() == 0


def _check(got, q, k, v, news, contexts):
    """Against float64; k, v: the sequences' rows one after the other.  Bound: the weights are rounded to 16 bits (2^-8 or 2^-11 of the value at most), as is
    the result; 1e-5 for the float32 sums."""
    H, G, D = q.shape[1], k.shape[1], q.shape[2]
    unit, at, row = 2.0 ** (-8 if q.dtype == torch.bfloat16 else -11), 0, 0
    for b, (n, c) in enumerate(zip(news, contexts)):
        i = torch.arange(n + c, device=DEV)
        kb, vb = (t[row:row + n + c].double().transpose(0, 1).repeat_interleave(H // G, 0) for t in (k, v))
        s = torch.bmm(q[at:at + n].double().transpose(0, 1), kb.transpose(1, 2)) * D ** -0.5
        w = torch.softmax(s.masked_fill(i[None, None] > (c + torch.arange(n, device=DEV))[None, :, None], -float("inf")), 2)
        want, mean = torch.bmm(w, vb).transpose(0, 1), torch.bmm(w, vb.abs()).transpose(0, 1)
        diff = (got[at:at + n].double() - want).abs()
        bound = (unit * 1.01 + 1e-5) * mean + unit * 1.01 * want.abs() + 1e-6
        assert bool((diff <= bound).all()), f"sequence {b}: worst excess {float((diff - bound).max()):.3e}"
        at, row = at + n, row + n + c


@pytest.mark.parametrize("D", [64, 128])
def test_large_queries_keep_the_precision(D):
    """Scores of four times unit size, where a few weights carry a row: the largest one is 1 and is not rounded, so that the error against float64 is little more
    than the result's own rounding, 2^-8 / sqrt(12) of a value between two powers of two in the mean square (1.66e-3 of the norm), as on the tile kernel
    (1.73e-3); with the maximum corrected from 2^8 on it is 2.09e-3."""
    n, H, G = 1500, 8, 2
    q, k, v = randn_t((n, H, D), 1, torch.bfloat16, DEV, scale=4.0), randn_t((n, G, D), 2, torch.bfloat16, DEV), randn_t((n, G, D), 3, torch.bfloat16, DEV)
    starts = torch.tensor([0, n], dtype=torch.int32, device=DEV)
    pages = lambda t: torch.cat([t, t.new_zeros((4, G, D))]).view(94, 16, G, D)
    got = ops.flash_attn_varlen_with_block_table(q, pages(k), pages(v), None, starts, starts, n, n, D ** -0.5, None, 0, torch.arange(94, dtype=torch.int32, device=DEV)[None])
    assert ops.last_mha_path() == "prefill_tc"
    kb, vb = (t.double().transpose(0, 1).repeat_interleave(H // G, 0) for t in (k, v))
    s = torch.bmm(q.double().transpose(0, 1), kb.transpose(1, 2)) * D ** -0.5
    w = torch.softmax(s.masked_fill(torch.ones((n, n), dtype=torch.bool, device=DEV).triu(1), -float("inf")), 2)
    want = torch.bmm(w, vb).transpose(0, 1)
    assert ((got.double() - want).norm() / want.norm()).item() < 1.85e-3


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("news,contexts,path", [
    # 30 sequences of 32 heads, on both sides of every line of short_for_prefill
    ((1, 64, 64, 65, 128, 128, 129, 1, 1, 300) * 3, (255, 192, 193, 0, 64, 65, 63, 1023, 1024, 0) * 3, "prefill_tc"),
    ((33, 1, 64) * 4, (0, 200, 192) * 4, "tile"),      # nothing but short sequences
])
def test_short_sequences_of_a_wide_step(D, dtype, news, contexts, path):
    """Steps of many sequences, whose short ones the tile kernel serves (heads of 64: beside the prefill kernel), against float64."""
    H, G, page = 32, 8, 16
    lens = [n + c for n, c in zip(news, contexts)]
    T = sum(news)
    q = randn_t((T, H, D), 1, dtype, DEV)
    each = [-(-n // page) for n in lens]
    pool = torch.randperm(sum(each), generator=torch.Generator().manual_seed(4)).to(torch.int32)
    kc, vc = randn_t((sum(each), page, G, D), 2, dtype, DEV), randn_t((sum(each), page, G, D), 3, dtype, DEV)
    table, used = torch.zeros((len(lens), max(each)), dtype=torch.int32), 0
    for b, n in enumerate(each):
        table[b, :n] = pool[used:used + n]
        used += n
    starts = lambda x: torch.tensor([sum(x[:i]) for i in range(len(x) + 1)], dtype=torch.int32, device=DEV)
    got = ops.flash_attn_varlen_with_block_table(q, kc, vc, None, starts(news), starts(lens), max(news), max(lens), D ** -0.5, None, 0, table.to(DEV))
    assert ops.last_mha_path() == path
    rows = torch.cat([table[b].long()[torch.arange(n) // page] * page + torch.arange(n) % page for b, n in enumerate(lens)]).to(DEV)
    _check(got, q, kc.reshape(-1, G, D)[rows], vc.reshape(-1, G, D)[rows], news, contexts)
