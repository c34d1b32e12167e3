"""The gated delta rule with keys of 65 to 128 entries: odd and single value columns, portions around a staged chunk of 32 tokens, both splits of the
rows over lanes, and the same bits however a sequence is cut into steps."""
import pytest
import torch

import surinex_oracle as so

pytestmark = pytest.mark.gpu
DEV = "cuda"


def i32(xs):
    return torch.tensor(xs, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("D,V", [(65, 1), (72, 33), (100, 31), (127, 2), (128, 65)])
def test_both_splits_against_float64(dtype, D, V):
    from atoma_infer_b200 import hybrid_ops as ops

    H, G, cuts = 4, 2, [4, 1, 31, 33, 7, 3]
    n = sum(cuts)
    g = torch.Generator().manual_seed(1000 * D + V)
    q, k = (torch.randn(n, G * D, generator=g).to(torch.bfloat16) for _ in range(2))
    v, b, a = (torch.randn(n, c, generator=g).to(torch.bfloat16) for c in (H * V, H, H))
    a_log, dt = torch.randn(H, generator=g) * 0.5 - 1.0, torch.randn(H, generator=g) * 0.5
    decay = torch.exp(-torch.exp(a_log.double()) * so.softplus(a.double() + dt.double()))
    want = so.delta_recurrence(so.unit_length(q.double().reshape(n, G, D)) * D ** -0.5, so.unit_length(k.double().reshape(n, G, D)),
                               v.double().reshape(n, H, V), so.sigma(b.double()), decay).reshape(n, H * V)
    x = [t.to(dtype).to(DEV) for t in (q, k, v, b, a)]
    outs = []
    try:
        for flags in (16, 0):        # 16: never the split of eight rows a lane, which serves a step of few CTAs
            ops.debug_flags(flags)
            state, got, lo = torch.full((2, H * D * V), 7.0, device=DEV), [], 0
            for c in cuts:
                got.append(ops.delta_rule_scan(*(t[lo:lo + c] for t in x), a_log.to(DEV), dt.to(DEV), D ** -0.5, state, i32([1]), i32([0, c]), i32([lo]),
                                               H, G, D, V))
                lo += c
            outs.append((torch.cat(got), state))
    finally:
        ops.debug_flags(0)
    # float32 throughout: some 128 + 5 terms and 79 decaying steps, 2^-24 each, of which the norm of the error keeps far less
    assert ((outs[0][0].double().cpu() - want).norm() / want.norm()).item() < 2e-5
    # both splits add in the same order
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])
    assert (outs[0][1][0] == 7.0).all()


@pytest.mark.parametrize("flags", [0, 16])
@pytest.mark.parametrize("D,V", [(128, 128), (100, 33), (64, 64)])
def test_cuts_do_not_change_the_bits(D, V, flags):
    """Outputs and state of 77 tokens read at once, token by token, and in portions that end anywhere, alone and beside another sequence."""
    from atoma_infer_b200 import hybrid_ops as ops

    H, G, n = 4, 2, 77
    g = torch.Generator().manual_seed(5)
    x = [torch.randn(n, c, generator=g).to(torch.bfloat16).to(DEV) for c in (G * D, G * D, H * V, H, H)]
    a_log, dt = (torch.randn(H, generator=g) * 0.5 - 1.0).to(DEV), (torch.randn(H, generator=g) * 0.5).to(DEV)

    def run(cuts, beside=0):
        state, out, lo = torch.zeros((2, H * D * V), device=DEV), [], 0
        for c in cuts:
            rows = [torch.cat([t[lo:lo + c], t[:beside]]) for t in x]
            slots, starts, ctx = ([0, 1], [0, c, c + beside], [lo, 0]) if beside else ([0], [0, c], [lo])
            out.append(ops.delta_rule_scan(*rows, a_log, dt, D ** -0.5, state, i32(slots), i32(starts), i32(ctx), H, G, D, V)[:c])
            lo += c
        return torch.cat(out), state[0]

    ops.debug_flags(flags)
    try:
        want = run([n])
        for cuts, beside in (([1] * n, 0), ([4, 1, 31, 33, 8], 0), ([2, 75], 0), ([50, 27], 9)):
            got = run(cuts, beside)
            assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]), cuts
    finally:
        ops.debug_flags(0)
