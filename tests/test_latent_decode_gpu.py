"""Latent attention of decoded tokens (equal runs of key tiles over the SMs, merged where a sequence is shared) against float64, at the edges
of its tiles, runs and head paddings.  Cache rows that no sequence owns hold NaN.  Debug flag 128 takes the kernel whatever the step's size; without it
the step's own choice of a kernel is held against the same bounds.

Bound per output entry: the queries, the weights and the cache are bfloat16 operands of float32 sums.  The oracle takes the queries rounded as the kernels
round them, so what is left is the weights' rounding, 2^-8 of the weighted mean of |c| at most, and 1e-4 of that mean for the float32 scores and sums.
That is tight enough to miss a tile: each oracle is also held against itself without one tile of 64 keys, which has to be outside the bound."""
import math

import pytest
import torch

from atoma_infer_b200 import _lib, hybrid_ops as ops
from helpers import randn_t

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _attend(flags, *args, **kw):
    ops.debug_flags(flags)
    try:
        return ops.latent_attention_paged(*args, **kw)
    finally:
        ops.debug_flags(0)


@pytest.mark.parametrize("H,R,out_cols,bs,window,sink,lens", [
    (32, 576, 512, 16, 0, False, (4096, 1, 64, 65, 2000, 127)),        # many CTAs share the long ones, several short ones share a CTA
    (17, 192, 128, 16, 100, True, (1, 99, 100, 101, 700)),             # heads padded to 32, a window that starts inside a page, a sink
    (16, 512, 0, 32, 0, True, (333,) * 7),                             # rows without a tail
    (1, 128, 0, 48, 65, False, (64, 66, 5000)),                        # one head, a window of one key more than a tile
    (12, 320, 256, 16, 0, False, tuple(range(1, 161))),                # more sequences than CTAs take one at a time
    (32, 256, 128, 16, 0, True, (30000,)),                             # one sequence over all SMs
])
@pytest.mark.parametrize("flags", [128, 0])
def test_against_float64(H, R, out_cols, bs, window, sink, lens, flags):
    g = torch.Generator().manual_seed(3)
    each = [-(-n // bs) for n in lens]
    pool = torch.randperm(sum(each) + 1, generator=g).to(torch.int32)
    table, at = torch.zeros((len(lens), max(each)), dtype=torch.int32), 0
    cache = torch.full(((sum(each) + 1) * bs, R), float("nan"), dtype=torch.bfloat16)
    rows = []
    for b, n in enumerate(lens):
        table[b, :each[b]] = pool[at:at + each[b]]
        at += each[b]
        p = torch.arange(n)
        slot = table[b].long()[p // bs] * bs + p % bs
        cache[slot] = torch.randn((n, R), generator=g).to(torch.bfloat16)
        rows.append(cache[slot].double())
        if window:                                # rows that have left the window, some of them beside its first key
            cache[slot[:max(0, n - window)]] = float("nan")
    q = torch.randn((len(lens), H, R), generator=g) * (8.0 / R ** 0.5)
    sinks = torch.randn(H, generator=g) if sink else None
    scale = 0.3
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    pos = torch.tensor([n - 1 for n in lens], device=DEV)
    got = _attend(flags, q.reshape(len(lens), -1).to(DEV), cache.to(DEV), pos, i32(list(range(len(lens)))), table.to(DEV), sinks.to(DEV) if sink else None, H, R, bs,
                  window, scale, 1, query_start=i32(list(range(len(lens) + 1))), max_seq_len=max(lens), out_cols=out_cols).double().cpu()
    cols = out_cols or R
    for b, c in enumerate(rows):
        c = c[-window:] if window else c
        s = q[b].to(torch.bfloat16).double() @ c.T * scale
        m = s.max(1, keepdim=True).values
        w = torch.exp(s - m)
        den = w.sum(1, keepdim=True) + (torch.exp(sinks.double()[:, None] - m) if sink else 0.0)
        want, mean = w / den @ c[:, :cols], w / den @ c[:, :cols].abs()
        bound = (2.0 ** -8 * 1.01 + 1e-4) * mean + 1e-6
        diff = (got[b, :, :cols] - want).abs()
        assert bool((diff <= bound).all()), f"sequence {b}: worst excess {float((diff - bound).max()):.3e}"
        if len(c) > 64:
            at = 64 * (len(c) // 128)
            w[:, at:at + 64] = 0.0
            den = den - torch.exp(s - m)[:, at:at + 64].sum(1, keepdim=True)
            assert bool(((w / den @ c[:, :cols] - want).abs() > bound).any())
    assert _lib.lib().atoma_latent_decode_timeouts() == 0


@pytest.mark.parametrize("lens", [(4096,), (200,) * 3, (65, 64, 3000)])
@pytest.mark.parametrize("where", ["query", "cached row"])
def test_nan_stays_nan(lens, where):
    """One NaN in a query, or in one cached row: every sum of that head (of all heads) is NaN whether one CTA served the sequence or several whose
    runs were merged, and the other sequences' are not."""
    H, R, bs = 8, 192, 16
    each = [-(-n // bs) for n in lens]
    table, at = torch.zeros((len(lens), max(each)), dtype=torch.int32), 0
    for b, n in enumerate(each):
        table[b, :n] = torch.arange(at, at + n)
        at += n
    cache = randn_t((at * bs, R), 1, torch.bfloat16, DEV)
    q = randn_t((len(lens), H, R), 2, torch.float32, DEV, scale=R ** -0.5)
    hit, i32 = len(lens) - 1, lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    if where == "query":
        q[hit, 3, 100] = float("nan")
    else:
        cache[int(table[hit, 1]) * bs + 5] = float("nan")
    out = _attend(128, q.reshape(len(lens), -1), cache, torch.tensor([n - 1 for n in lens], device=DEV), i32(list(range(len(lens)))), table.to(DEV), None, H, R,
                  bs, 0, 0.3, 1, query_start=i32(list(range(len(lens) + 1))), max_seq_len=max(lens), out_cols=128)[:, :, :128]
    want = torch.zeros((len(lens), H), dtype=torch.bool, device=DEV)
    want[hit, slice(3, 4) if where == "query" else slice(None)] = True
    assert torch.equal(out.isnan().all(2), want) and torch.equal(out.isnan().any(2), want)


@pytest.mark.parametrize("T,H,n,R,row,gated", [(1, 3, 32, 64, 64, False), (33, 2, 64, 192, 256, True), (64, 5, 128, 512, 576, True), (65, 2, 32, 128, 128, False)])
def test_values_of_a_few_tokens(T, H, n, R, row, gated):
    """Operands rounded to bfloat16 (2^-8 of the input), float32 sums, one rounding of the result; 65 tokens take the general path."""
    o = randn_t((T, H, row), 1, torch.float32, DEV)
    w = randn_t((H * n, R), 2, torch.bfloat16, DEV, scale=R ** -0.5)
    gate = randn_t((T, H * n), 3, torch.bfloat16, DEV) if gated else None
    got = ops.latent_expand_values(o, w, H, n, R, torch.bfloat16, gate=gate).double().cpu()
    x, wd = o.double().cpu()[..., :R], w.double().cpu().reshape(H, n, R)
    s = torch.sigmoid(gate.double().cpu()) if gated else 1.0
    want = torch.einsum("thr,hnr->thn", x, wd).reshape(T, -1) * s
    mag = torch.einsum("thr,hnr->thn", x.abs(), wd.abs()).reshape(T, -1)
    assert bool(((got - want).abs() <= 2.0 ** -8 * want.abs() + (2.0 ** -8 + 4e-6) * mag * 1.01).all())


@pytest.mark.parametrize("T,H,dim,rot,pairs,interleaved,rank", [(1, 3, 128, 64, 32, False, 512), (31, 2, 64, 32, 7, True, 64), (33, 5, 48, 8, 4, False, 192), (64, 4, 128, 0, 0, False, 128), (64, 1, 256, 16, 0, True, 64)])
def test_absorbed_queries_of_few_tokens(T, H, dim, rot, pairs, interleaved, rank):
    """One launch for up to 64 tokens: the bits of the product in 64-token tiles and the rotation behind it, which a step of one token more takes."""
    q = randn_t((65, H * (dim + rot)), 1, torch.bfloat16, DEV)
    w = randn_t((H * dim, rank), 2, torch.bfloat16, DEV)
    freq = (10000.0 ** (-torch.arange(pairs, dtype=torch.float32) / max(pairs, 1))).to(DEV) if pairs else None
    low = (torch.arange(pairs, dtype=torch.float32) * 1e-9).to(DEV) if pairs else None
    pos = torch.arange(65, device=DEV) * 97
    run = lambda n: ops.latent_query_absorb_rope(q[:n], w, freq, interleaved, pos[:n], H, dim, rot, rank, freq_lo=low, amplitude=1.25)
    got, want = run(T), run(65)
    assert torch.equal(got, want[:T])
    exact = torch.einsum("thd,hdr->thr", q[:T].double().view(T, H, -1)[..., :dim], w.double().view(H, dim, rank))
    assert (got[..., :rank].double() - exact).norm() <= 1e-5 * exact.norm()
