"""Sigmoid attention with talking heads over prompt portions (the talk matrix as a product of split pieces, keys in segments) against float64.

Bound per output entry: a score is a float32 sum of bfloat16 products, a weight and the mix are within 1e-5 of sum_g |talk| a_g; the mixed weight is
rounded to bfloat16 (8 bits: 2^-8 of it at most) before it meets the value, the result once more."""
import pytest
import torch

from atoma_infer_b200 import _lib
from atoma_infer_b200 import hybrid_ops as ops
from helpers import randn_t

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
F64 = torch.float64


@pytest.mark.parametrize("H,G,D,V,bs,seqs,cap,slopes,bias", [
    (32, 8, 64, 64, 16, ((0, 33), (40, 1), (1000, 17)), 30.0, True, -1.0),      # a row past two tiles, a decoded token, a portion over two segments
    (16, 2, 48, 32, 16, ((1500, 20), (511, 2), (0, 16)), 0.0, False, 0.0),      # three segments, one that ends at a row block's last key; no cap, no slopes
    (32, 32, 16, 64, 8, ((600, 5),), 5.0, True, -10.0),                         # one head per key head; weights near 5e-5
    (16, 16, 64, 16, 16, ((0, 700),), 8.0, True, 0.0),                          # a prompt whose later rows take two segments
    (32, 8, 64, 64, 4, ((0, 33), (1000, 17)), 30.0, True, -1.0),                # pages that hold no run of eight keys: the kernel of other head sizes
    (32, 8, 48, 32, 16, ((0, 700), (1500, 20)), 8.0, True, -1.0),               # ... whose later rows take two segments, then three
])
def test_against_float64(H, G, D, V, bs, seqs, cap, slopes, bias):
    def edit(talk):
        talk[1] *= 1e-4                  # rows of other sizes
        talk[2] *= 300.0
        talk[3] = 0.0

    _compare(H, G, D, V, bs, seqs, cap, slopes, bias, edit, 1e-9)


@pytest.mark.parametrize("H", [16, 32])
def test_small_weights_keep_their_bits(H):
    """Heads whose weights are near e^-40 everywhere: the mix is float32's, whatever the weights' size."""
    _compare(H, 4, 64, 64, 16, ((0, 40), (700, 20)), 8.0, False, -40.0, lambda talk: None, 0.0)


@pytest.mark.parametrize("H", [16, 32])
def test_small_talk_rows(H):
    """Rows of the talk matrix far below and far above one, down to float32's smallest normal values (their outputs may be flushed to zero: 1e-36)."""
    def edit(talk):
        for h, scale in enumerate([1e-10, 1e-25, 2.0 ** -110, 2.0 ** -121, 2.0 ** -125, 1e10, 1e20, 1e30]):
            talk[h] *= scale

    _compare(H, 4, 64, 64, 16, ((0, 40), (700, 20)), 8.0, True, -1.0, edit, 1e-36)


def _compare(H, G, D, V, bs, seqs, cap, slopes, bias, edit, floor):
    g = torch.Generator().manual_seed(2)
    each = [-(-(c + n) // bs) for c, n in seqs]
    pool = torch.randperm(sum(each), generator=g).to(torch.int32)
    table, at = torch.zeros((len(seqs), max(each)), dtype=torch.int32), 0
    for b, n in enumerate(each):
        table[b, :n] = pool[at:at + n]
        at += n
    kc, vc = randn_t((sum(each) * bs, G, D), 1, torch.bfloat16, DEV), randn_t((sum(each) * bs, G, V), 2, torch.bfloat16, DEV)
    T = sum(n for _, n in seqs)
    q = randn_t((T, H * D), 3, torch.bfloat16, DEV)
    sl = torch.tensor([2.0 ** (-8.0 * (h + 1) / H) for h in range(H)], device=DEV) if slopes else None
    hb = randn_t((H,), 4, torch.float32, DEV, scale=0.5) + bias
    talk = torch.eye(H, device=DEV) + randn_t((H, H), 5, torch.float32, DEV, scale=0.3)
    edit(talk)
    pos = torch.cat([torch.arange(c, c + n) for c, n in seqs]).to(DEV)
    tseq = torch.arange(len(seqs), dtype=torch.int32).repeat_interleave(torch.tensor([n for _, n in seqs])).to(DEV)
    out = ops.sigmoid_attention_paged(q, kc, vc, pos, tseq, table.to(DEV), sl, hb, talk, H, G, D, V, bs, D ** -0.5, cap, max(n for _, n in seqs)).double()
    t0 = 0
    for b, (c, n) in enumerate(seqs):
        p = torch.arange(c + n)
        slot = (table[b].long()[p // bs] * bs + p % bs).to(DEV)
        k, v = (x[slot].double().transpose(0, 1).repeat_interleave(H // G, 0) for x in (kc, vc))
        z = torch.bmm(q[t0:t0 + n].double().reshape(n, H, D).transpose(0, 1), k.transpose(1, 2)) * D ** -0.5
        if cap:
            z = cap * torch.tanh(z / cap)
        gap = (c + torch.arange(n, device=DEV)[:, None] - torch.arange(c + n, device=DEV)[None]).double()
        if slopes:
            z = z - sl.double()[:, None, None] * gap
        w = torch.sigmoid(z + hb.double()[:, None, None]) * (gap >= 0)
        mixed = (talk.double() @ w.reshape(H, -1)).reshape(w.shape)
        slack = 2.0 ** -8 * mixed.abs() + 1e-5 * (talk.double().abs() @ w.reshape(H, -1)).reshape(w.shape)
        flat = lambda x: x.transpose(0, 1).reshape(n, H * V)
        want, bound = flat(torch.bmm(mixed, v)), flat(torch.bmm(slack, v.abs()))
        diff = (out[t0:t0 + n] - want).abs()
        excess = diff - (bound + 2.0 ** -8 * want.abs() + floor)
        assert bool((excess <= 0).all()), f"sequence {b}: worst excess {float(excess.max()):.3e}"
        t0 += n


@pytest.mark.parametrize("H,D,others", [
    (32, 64, ((4000, 3),)),                        # a longer sequence beside it
    (16, 16, ((0, 4000), (0, 3000), (0, 3000))),   # a step of many tokens, whose CTAs take all segments of their rows
    (32, 64, ((20000, 900),)),                     # sums that take more than one run of tokens
    (32, 64, ((0, 9600),)),                        # ... whose CTAs take all segments, of the shorter ones
    (32, 48, ((0, 9600), (20000, 40))),            # the kernel of other head sizes
])
def test_a_position_does_not_depend_on_the_step(H, D, others):
    """The same bits for a sequence alone, beside others, and read in two portions that end anywhere."""
    G, bs, n = 8, 16, 1301
    seqs = [(0, n)] + list(others)
    each = [-(-(c + m) // bs) for c, m in seqs]
    table, at = torch.zeros((len(seqs), max(each)), dtype=torch.int32), 0
    for b, m in enumerate(each):
        table[b, :m] = torch.arange(at, at + m)
        at += m
    kc, vc = (randn_t((at * bs, G, D), i, torch.bfloat16, DEV) for i in (1, 2))
    q = randn_t((sum(m for _, m in seqs), H * D), 3, torch.bfloat16, DEV)
    hb, talk = randn_t((H,), 4, torch.float32, DEV), torch.eye(H, device=DEV) + randn_t((H, H), 5, torch.float32, DEV, scale=0.3)

    def run(rows, seqs, table, longest=None):
        pos = torch.cat([torch.arange(c, c + m) for c, m in seqs]).to(DEV)
        tseq = torch.arange(len(seqs), dtype=torch.int32).repeat_interleave(torch.tensor([m for _, m in seqs])).to(DEV)
        return ops.sigmoid_attention_paged(rows, kc, vc, pos, tseq, table.to(DEV), None, hb, talk, H, G, D, D, bs, D ** -0.5, 8.0, max(m for _, m in seqs), None, longest)

    alone = run(q[:n], seqs[:1], table[:1])
    wide = torch.cat([table[:1], torch.zeros((1, 1100), dtype=torch.int32)], 1)   # ... or in a wide table, its length unknown: single segments' sums do not fit at once
    assert torch.equal(run(q[:n], seqs[:1], wide, 0), alone)
    assert torch.equal(run(q, seqs, table)[:n], alone)
    assert torch.equal(run(q[:701], [(0, 701)], table[:1]), alone[:701])
    assert torch.equal(run(q[701:n], [(701, 600)], table[:1]), alone[701:])


@pytest.mark.parametrize("G", [1, 2, 8])
def test_same_bits_whatever_the_pages(G):
    """32 heads of 64: pages of whole 16-key tiles go by TMA, others by pieces; cache rows that belong to no sequence hold NaN."""
    H, D, seqs = 32, 64, ((0, 49), (30, 2), (1007, 17), (512, 16), (495, 1))
    lens = [c + n for c, n in seqs]
    T = sum(n for _, n in seqs)
    q, talk = randn_t((T, H * D), 3, torch.bfloat16, DEV), torch.eye(H, device=DEV) + randn_t((H, H), 5, torch.float32, DEV, scale=0.3)
    k, v = (randn_t((sum(lens), G, D), i, torch.bfloat16, DEV) for i in (1, 2))
    hb = randn_t((H,), 4, torch.float32, DEV)
    pos = torch.cat([torch.arange(c, c + n) for c, n in seqs]).to(DEV)
    tseq = torch.arange(len(seqs), dtype=torch.int32).repeat_interleave(torch.tensor([n for _, n in seqs])).to(DEV)
    outs = []
    for bs in (16, 24, 48, 8):
        each = [-(-n // bs) for n in lens]
        pool = torch.randperm(sum(each), generator=torch.Generator().manual_seed(bs)).to(torch.int32)
        kc, vc = (torch.full((sum(each) * bs, G, D), float("nan"), dtype=torch.bfloat16, device=DEV) for _ in range(2))
        table, used, row = torch.zeros((len(seqs), max(each)), dtype=torch.int32), 0, 0
        for b, n in enumerate(lens):
            table[b, :each[b]] = pool[used:used + each[b]]
            at = torch.arange(n)
            slot = (table[b].long()[at // bs] * bs + at % bs).to(DEV)
            kc[slot], vc[slot] = k[row:row + n], v[row:row + n]
            used, row = used + each[b], row + n
        outs.append(ops.sigmoid_attention_paged(q, kc, vc, pos, tseq, table.to(DEV), None, hb, talk, H, G, D, D, bs, D ** -0.5, 8.0, 49))
    assert torch.isfinite(outs[0]).all() and all(torch.equal(o, outs[0]) for o in outs[1:])


@pytest.mark.parametrize("H,G,bs", [(32, 8, 16), (32, 2, 24), (16, 4, 16)])
def test_one_cache_as_keys_and_values(H, G, bs):
    """A cache that serves as both gives the bits of two caches with the same rows: by TMA (pages of whole 16-key tiles), by pieces, and for 16 heads."""
    D, seqs = 64, ((0, 49), (300, 2))
    each = [-(-(c + n) // bs) for c, n in seqs]
    table = torch.zeros((2, max(each)), dtype=torch.int32)
    table[0, :each[0]], table[1, :each[1]] = torch.arange(each[0]), torch.arange(each[0], sum(each))
    kc, q = randn_t((sum(each) * bs, G, D), 1, torch.bfloat16, DEV), randn_t((51, H * D), 3, torch.bfloat16, DEV)
    hb, talk = randn_t((H,), 4, torch.float32, DEV), torch.eye(H, device=DEV) + randn_t((H, H), 5, torch.float32, DEV, scale=0.3)
    pos = torch.cat([torch.arange(c, c + n) for c, n in seqs]).to(DEV)
    tseq = torch.tensor([0] * 49 + [1] * 2, dtype=torch.int32, device=DEV)
    run = lambda vc: ops.sigmoid_attention_paged(q, kc, vc, pos, tseq, table.to(DEV), None, hb, talk, H, G, D, D, bs, D ** -0.5, 8.0, 49)
    given_up = _lib.lib().atoma_kernel_timeouts()
    assert torch.equal(run(kc), run(kc.clone())) and _lib.lib().atoma_kernel_timeouts() == given_up


@pytest.mark.parametrize("H,D", [(16, 32), (32, 64)])
def test_capture_on_a_stream_without_scratch(H, D):
    """A long prompt captured on a stream that has run nothing: segments need scratch that cannot be had there, whole rows need none."""
    G, bs, n = 2, 16, 1100
    kc, vc, q = (randn_t((1104, *s), i, torch.bfloat16, DEV) for i, s in enumerate([(G, D), (G, D), (H * D,)]))
    table, pos, tseq = torch.arange(69, dtype=torch.int32, device=DEV)[None], torch.arange(n, device=DEV), torch.zeros(n, dtype=torch.int32, device=DEV)
    talk, hb = randn_t((H, H), 5, torch.float32, DEV), torch.zeros(H, device=DEV)
    starts = torch.tensor([0, n], dtype=torch.int32, device=DEV)
    run = lambda: ops.sigmoid_attention_paged(q[:n], kc, vc, pos, tseq, table, None, hb, talk, H, G, D, D, bs, D ** -0.5, 0.0, n, starts, n)
    want, graph = run().double(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=torch.cuda.Stream()):
        got = run()
    graph.replay()
    torch.cuda.synchronize()
    # one sum in another order, then one rounding to bfloat16 each
    assert bool(((got.double() - want).abs() <= 2.0 ** -7 * want.abs() + 1e-4).all())
