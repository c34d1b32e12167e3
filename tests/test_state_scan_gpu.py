"""The matrix-state scans on every split of the state over lanes and warps, and on every way their rows are copied: the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def i32(xs):
    return torch.tensor(xs, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("D,V", [(64, 128), (128, 64), (72, 8), (50, 34), (33, 7), (256, 16), (300, 24)])
@pytest.mark.parametrize("rule", ["gla", "delta", "ssm"])
def test_splits_and_copies_give_the_same_bits(rule, D, V, dtype):
    """One sequence of 70 tokens (two chunks and a rest) alone, with sixteen rows a lane, among enough sequences for the CTAs of eight warps, and in
    columns of a wider matrix that start at an odd element (value by value) or at an even one (pieces of four bytes)."""
    from atoma_infer_b200 import hybrid_ops as ops

    H, n, B = 4, 70, 90
    G = H if rule == "gla" else 2
    g = torch.Generator().manual_seed(D + V)
    rnd = lambda c: torch.randn(n, c, generator=g).to(torch.bfloat16).to(dtype).to(DEV)
    q, k, v, z, b, a = rnd(G * D), rnd(G * D), rnd(H * V), rnd(H * D), rnd(H), rnd(H)
    k *= D ** -0.5 if rule != "delta" else 1.0
    per_head = [torch.randn(H, generator=g).to(DEV) * 0.5 - 1.0 for _ in range(3)]
    zb = torch.randn(H * D, generator=g).to(DEV)

    def run(rows, starts, flags=0):
        """Every sequence in its own slot, from zero; (outputs, states)."""
        q, k, v, z, b, a = rows
        S = len(starts) - 1
        state = torch.full((S, H * D * V), 3.0, device=DEV)
        at = (state, i32(list(range(S))), i32(starts), i32([0] * S), H)
        ops.debug_flags(flags)
        try:
            if rule == "gla":
                return ops.gla_scan(q, k, v, z, zb, 6.0, D ** -0.5, *at, D, V), state
            if rule == "delta":
                return ops.delta_rule_scan(q, k, v, b, a, per_head[0], per_head[1], D ** -0.5, *at, G, D, V), state
            return ops.ssm_scan(v, k, q, a, per_head[0], per_head[1], per_head[2], *at, G, D, V), state
        finally:
            ops.debug_flags(0)

    rows = [q, k, v, z, b, a]
    out, state = run(rows, [0, n])
    assert torch.isfinite(out).all() and torch.isfinite(state).all()
    sixteen = run(rows, [0, n], 16)
    assert torch.equal(sixteen[0], out) and torch.equal(sixteen[1], state)
    many = [torch.cat([t] + [t[:6]] * (B - 1)) for t in rows]            # six tokens each: no step of short portions, so the first one's chunks go through the CTAs of eight warps
    wide = run(many, [0] + [n + 6 * b for b in range(B)])
    assert torch.equal(wide[0][:n], out) and torch.equal(wide[1][0], state[0])
    short = [torch.cat([t] + [t[:1]] * (B - 1)) for t in rows]           # the portions of the others have one token: the mean is below four, short CTAs
    few = run(short, [0] + list(range(n, n + B)))
    assert torch.equal(few[0][:n], out) and torch.equal(few[1][0], state[0])
    for shift in (1, 2):
        padded = []
        for t in rows:
            m = torch.zeros(n, t.shape[1] + 3, dtype=dtype, device=DEV)
            m[:, shift:shift + t.shape[1]] = t
            padded.append(m[:, shift:shift + t.shape[1]])
        moved = run(padded, [0, n])
        assert torch.equal(moved[0], out) and torch.equal(moved[1], state), shift


@pytest.mark.parametrize("n,empty", [(10, 2), (5, 3), (33, 30)])
@pytest.mark.parametrize("D", [64, 128])
def test_sequences_without_a_token(n, empty, D):
    """A portion that is longer than the step's tokens shared out, one to every sequence, would allow."""
    from atoma_infer_b200 import hybrid_ops as ops

    H, V = 4, 64
    g = torch.Generator().manual_seed(n)
    q, k, v, z = (torch.randn(n, c, generator=g).to(torch.bfloat16).to(DEV) for c in (H * D, H * D, H * V, H * D))
    zb = torch.randn(H * D, generator=g).to(DEV)
    outs = []
    for starts in ([0, n], [0] + [n] * (empty + 1), [0] * (empty + 1) + [n]):
        S = len(starts) - 1
        state = torch.zeros((S, H * D * V), device=DEV)
        out = ops.gla_scan(q, k, v, z, zb, 6.0, D ** -0.5, state, i32(list(range(S))), i32(starts), i32([0] * S), H, D, V)
        outs.append((out, state[starts.index(n) - 1]))
    assert all(torch.equal(o, outs[0][0]) and torch.equal(s, outs[0][1]) for o, s in outs[1:])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("D,V", [(64, 128), (64, 64), (64, 32), (128, 64), (72, 8), (50, 34), (33, 7), (256, 16), (300, 24), (512, 12)])
@pytest.mark.parametrize("rule", ["gla", "delta", "ssm"])
def test_short_steps_give_the_bits_of_long_ones(rule, D, V, dtype):
    """A portion of 23 tokens at once, among enough others for the wide CTAs, and in steps of one to four tokens, whose states pass through shared memory where
    their rows are whole pieces of 16 bytes; states of an odd pitch, which are not."""
    from atoma_infer_b200 import hybrid_ops as ops

    H, n, B = 4, 23, 80
    G = H if rule == "gla" else 2
    g = torch.Generator().manual_seed(D + V)
    rnd = lambda c: torch.randn(n, c, generator=g).to(torch.bfloat16).to(dtype).to(DEV)
    rows = [rnd(G * D), rnd(G * D), rnd(H * V), rnd(H * D), rnd(H), rnd(H)]
    rows[1] *= D ** -0.5 if rule != "delta" else 1.0
    per_head = [torch.randn(H, generator=g).to(DEV) * 0.5 - 1.0 for _ in range(3)]
    zb = torch.randn(H * D, generator=g).to(DEV)
    before = torch.randn(H * D * V, generator=g).to(DEV)

    def step(rows, state, slots, starts, contexts):
        q, k, v, z, b, a = rows
        at = (state, i32(slots), i32(starts), i32(contexts), H)
        if rule == "gla":
            return ops.gla_scan(q, k, v, z, zb, 6.0, D ** -0.5, *at, D, V)
        if rule == "delta":
            return ops.delta_rule_scan(q, k, v, b, a, per_head[0], per_head[1], D ** -0.5, *at, G, D, V)
        return ops.ssm_scan(v, k, q, a, per_head[0], per_head[1], per_head[2], *at, G, D, V)

    def states(count, pitch=0):
        s = torch.full((count, H * D * V + pitch), 3.0, device=DEV)
        s[:, :H * D * V] = before
        return s

    state = states(1)
    out = step(rows, state, [0], [0, n], [7])
    assert torch.isfinite(out).all() and torch.isfinite(state).all()
    many = [torch.cat([t] + [t[:6]] * (B - 1)) for t in rows]            # six tokens a sequence: no short step
    wide = states(B)
    assert torch.equal(step(many, wide, list(range(B)), [0] + [n + 6 * b for b in range(B)], [7] * B)[:n], out) and torch.equal(wide[0], state[0])
    for pitch in (0, 1):
        cut, t0, k = states(2, pitch), 0, 0
        while t0 < n:
            m = min(1 + k % 4, n - t0)
            part = step([t[t0:t0 + m].contiguous() for t in rows], cut, [1], [0, m], [7 + t0])
            assert torch.equal(part, out[t0:t0 + m]), (t0, m, pitch)
            t0, k = t0 + m, k + 1
        assert torch.equal(cut[1, :H * D * V], state[0]) and bool((cut[:, H * D * V:] == 3.0).all()) and torch.equal(cut[0, :H * D * V], before)
    fresh = states(1)                                                     # no context: what the slot held does not count
    whole = states(1)
    a, b = step(rows, whole, [0], [0, n], [0]), step([t[:1] for t in rows], fresh, [0], [0, 1], [0])
    assert torch.equal(a[:1], b)


def test_gla_decay_against_float64():
    """One token with k = 0 on a state of ones: the state that is left is the decay, sigmoid(z)^(1 / tau)."""
    from atoma_infer_b200 import hybrid_ops as ho

    H, D, V = 64, 64, 64
    z = torch.linspace(-85.0, 85.0, H * D, device=DEV)
    z[:7] = torch.tensor([0.0, -0.0, 1e-6, -1e-6, 1e-30, -17.3, 17.3], device=DEV)
    zeros = lambda n: torch.zeros((1, n), device=DEV)
    i32 = lambda *x: torch.tensor(x, dtype=torch.int32, device=DEV)
    for tau in (1.0, 16.0):
        state = torch.ones((1, H * D * V), device=DEV)
        ho.gla_scan(zeros(H * D), zeros(H * D), zeros(H * V), z[None].contiguous(), torch.zeros(H * D, device=DEV), tau, 1.0, state, i32(0), i32(0, 1), i32(5), H, D, V)
        log = torch.nn.functional.logsigmoid(z.double()) / tau
        got, want = state.reshape(H * D, V)[:, 0].double(), torch.exp(log)
        # the logarithm and its quotient by tau are rounded to float32 each, its term log(1 + x) <= log 2 is within three units, the exponential within two
        bound = log.abs() * 2.0 ** -23 + 2.1 * 2.0 ** -24 / tau + 2.0 ** -22
        assert bool(((got / want - 1.0).abs() <= bound).all())
        assert torch.equal(state.reshape(H * D, V), state.reshape(H * D, V)[:, :1].expand(-1, V))
