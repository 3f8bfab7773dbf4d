"""The recurrences over long prompt portions in chunks of 64 tokens (gated_chunks.cu, delta_chunks.cu) against the same recurrences
walked token by token in float64: portions that end inside a chunk, on its edge and one token beyond, beside short portions and single tokens
that the walk keeps; head sizes on and off the kernels' padding; states that are not zero at the start.

The bound: every output is a sum of at most T rounded products whose factors are themselves products of at most T decays, so its error
against float64 grows at worst with T units of 2^-24 and in practice with the root of that; 2e-5 of the result's root mean square is about 8 sqrt(T)
units at 640 tokens."""

import numpy as np
import pytest
import torch

from tests.conftest import cuda_or_skip

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def in_chunks(monkeypatch):
    """Every portion that may run in chunks does, whether or not it pays."""
    import sllm_b200.ops as ops
    monkeypatch.setattr(ops, "_chunks_pay", lambda *a: True)


REL = 2e-5
LENS = [640, 1, 96, 200, 63, 64 * 2 + 1, 128, 95]
SLOTS = [5, 0, 3, 8, 1, 7, 2, 6]


def _step(dev, lens, slots):
    from tests.test_rososun import _step as make
    return make(dev, lens, slots)


def _spans():
    starts = np.concatenate([[0], np.cumsum(LENS)])
    return [(int(a), int(b), s) for a, b, s in zip(starts[:-1], starts[1:], SLOTS)]


def _close(got, want, what):
    got, want = got.double(), want.double()
    assert torch.isfinite(got).all(), what
    err = (got - want).abs().max() / want.pow(2).mean().sqrt()
    assert err < 40 * REL, f"{what}: {float(err)} of the root mean square at worst"
    err = (got - want).norm() / want.norm()
    assert err < REL, f"{what}: {float(err)}"


def _walk(q, k, v, keep, S, p=None, w=None):
    """float64, [T, H, d]: S <- keep S - w (p^T S) + k v^T, o = S^T q."""
    out = torch.empty_like(v)
    for t in range(q.shape[0]):
        gone = w[t][:, :, None] * torch.einsum("hi,hij->hj", p[t], S)[:, None] if p is not None else 0.0
        S = S * keep[t][:, :, None] - gone + k[t][:, :, None] * v[t][:, None, :]
        out[t] = torch.einsum("hij,hi->hj", S, q[t])
    return out, S


def _state(g, H, dk, dv, dev):
    return torch.randn(10, H, dk, dv, device=dev, generator=g)


def _check(run, terms, H, dk, dv, dev, g):
    """``run(state, step) -> o``; ``terms(a, b)``: float64 (q, k, v, keep[, p, w]) of a span's tokens."""
    state = _state(g, H, dk, dv, dev)
    before = state.clone()
    o = run(state, _step(dev, LENS, SLOTS)).reshape(-1, H, dv)
    for a, b, slot in _spans():
        want, last = _walk(*[x[:, :, :] if x.dim() == 3 else x for x in terms(a, b)[:4]], before[slot].double(), *terms(a, b)[4:])
        _close(o[a:b], want, f"outputs of {b - a} tokens")
        _close(state[slot], last, f"state after {b - a} tokens")
    untouched = [s for s in range(10) if s not in SLOTS]
    assert torch.equal(state[untouched], before[untouched])


SIZES = [(64, 64, 3), (128, 128, 2), (128, 64, 2), (64, 128, 2), (40, 24, 3), (72, 100, 2), (17, 5, 2)]


@pytest.mark.parametrize("dk,dv,H", SIZES)
@pytest.mark.parametrize("hard", [False, True])
def test_gated_linear_attention_in_chunks(dk, dv, H, hard):
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    g = torch.Generator(device=dev).manual_seed(dk + 3 * dv)
    T, off = sum(LENS), 3
    proj = torch.randn(T, off + H * (2 * dk + dv), device=dev, generator=g)
    z = torch.randn(T, H * dk, device=dev, generator=g) * (40.0 if hard else 1.0) + (0.0 if hard else 2.0)      # hard: decays from one down to e^-20
    offs = (off, off + H * dk, off + 2 * H * dk)

    def terms(a, b):
        q, k, v = (proj[a:b, o:o + H * n].double().reshape(b - a, H, n) for o, n in zip(offs, (dk, dk, dv)))
        return q * dk ** -0.5, k, v, (torch.nn.functional.logsigmoid(z[a:b].double()) / 8.0).exp().reshape(b - a, H, dk)
    _check(lambda state, step: ops.gated_linear_attention(proj, offs, z, state, step, H, dk, dv, dk ** -0.5, 8.0), terms, H, dk, dv, dev, g)


@pytest.mark.parametrize("dk,dv,H", SIZES)
def test_decay_linear_attention_in_chunks(dk, dv, H):
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    g = torch.Generator(device=dev).manual_seed(dk + 5 * dv)
    T = sum(LENS)
    proj = torch.randn(T, H * (2 * dk + dv), device=dev, generator=g)
    decay = torch.tensor([1.0 - 2.0 ** (-2.0 - 4 * h) for h in range(H)], device=dev)
    offs = (0, H * dk, 2 * H * dk)
    silu = torch.nn.functional.silu

    def terms(a, b):
        q, k, v = (silu(proj[a:b, o:o + H * n].double()).reshape(b - a, H, n) for o, n in zip(offs, (dk, dk, dv)))
        return q, k, v, decay.double()[None, :, None].expand(b - a, H, 1)
    _check(lambda state, step: ops.decay_linear_attention(proj, offs, decay, state, step, H, dk, dv), terms, H, dk, dv, dev, g)


@pytest.mark.parametrize("dk,dv,H", SIZES)
@pytest.mark.parametrize("hard", [False, True])
def test_forget_gate_attention_in_chunks(dk, dv, H, hard):
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    g = torch.Generator(device=dev).manual_seed(dk + 7 * dv)
    T = sum(LENS)
    proj = torch.randn(T, H * (2 * dk + dv), device=dev, generator=g)
    bias = torch.randn(H * dk, device=dev, generator=g) * (30.0 if hard else 1.0)
    lower = torch.rand(H * dk, device=dev, generator=g) * (0.0 if hard else 0.9)
    offs = (0, H * dk, 2 * H * dk)

    def terms(a, b):
        q, z, v = (proj[a:b, o:o + H * n].double().reshape(b - a, H, n) for o, n in zip(offs, (dk, dk, dv)))
        f = (lower + (1 - lower) * torch.sigmoid(proj[a:b, offs[1]:offs[1] + H * dk] + bias)).double().reshape(b - a, H, dk)
        return torch.nn.functional.silu(q), 1 - f, v, f
    _check(lambda state, step: ops.forget_gate_attention(proj, offs, bias, lower, state, step, H, dk, dv), terms, H, dk, dv, dev, g)


@pytest.mark.parametrize("dk,dv,H,G", [(64, 64, 4, 2), (128, 128, 2, 1), (128, 64, 2, 2), (64, 128, 2, 1), (40, 24, 3, 3), (100, 72, 2, 1)])
@pytest.mark.parametrize("hard", [False, True])
def test_gated_delta_rule_in_chunks(dk, dv, H, G, hard):
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    g = torch.Generator(device=dev).manual_seed(dk + 11 * dv)
    T = sum(LENS)
    qkv = torch.randn(T, 2 * G * dk + H * dv, device=dev, generator=g)
    gates = torch.randn(T, 2 * H + 1, device=dev, generator=g)
    a_log = torch.rand(H, device=dev, generator=g) * (6.0 if hard else 2.0)       # hard: decays down to zero
    dt_bias = torch.randn(H, device=dev, generator=g) - (0.0 if hard else 3.0)
    offs = (0, G * dk, 2 * G * dk)

    def terms(a, b):
        n = b - a
        q, k = (qkv[a:b, o:o + G * dk].double().reshape(n, G, dk) for o in offs[:2])
        q, k = (x / (x.pow(2).sum(-1, keepdim=True) + 1e-6).sqrt() for x in (q, k))
        q, k = (x.repeat_interleave(H // G, 1) for x in (q * dk ** -0.5, k))
        v = qkv[a:b, offs[2]:].double().reshape(n, H, dv)
        beta = torch.sigmoid(gates[a:b, :H].double())[:, :, None]
        keep = torch.exp(-torch.exp(a_log.double()) * torch.nn.functional.softplus(gates[a:b, H + 1:].double() + dt_bias.double()))[:, :, None]
        return q, k, beta * v, keep, k, beta * keep * k
    _check(lambda state, step: ops.gated_delta_rule(qkv, offs, gates, 0, H + 1, a_log, dt_bias, state, step, H, G, dk, dv, dk ** -0.5),
           terms, H, dk, dv, dev, g)


@pytest.mark.parametrize("d,H", [(64, 3), (40, 2), (17, 5)])
@pytest.mark.parametrize("hard", [False, True])
def test_delta_rule_in_chunks(d, H, hard):
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    g = torch.Generator(device=dev).manual_seed(d + 13 * H)
    T, C = sum(LENS), H * d
    proj = torch.randn(T, 4 * C, device=dev, generator=g)
    decay = torch.randn(T, C, device=dev, generator=g) * 2 + (20.0 if hard else -2.0)      # hard: every channel's decay at its smallest
    bias = torch.randn(C, device=dev, generator=g)

    def terms(a, b):
        r, k, v, z = (proj[a:b, o * C:(o + 1) * C].double().reshape(b - a, H, d) for o in range(4))
        u = k / (k.pow(2).sum(-1, keepdim=True) + 1e-6).sqrt()
        keep = torch.exp(-np.exp(-0.5) * torch.sigmoid(decay[a:b].double())).reshape(b - a, H, d)
        return r, k, v, keep, u, torch.sigmoid(z + bias.double().reshape(H, d)) * u
    _check(lambda state, step: ops.delta_rule(proj, (0, C, 2 * C, 3 * C), decay, bias, state, step, H, d, d), terms, H, d, d, dev, g)


# ---- single tokens ------------------------------------------------------------------------------------------------------

TOKEN_SIZES = [(64, 64, 3), (128, 128, 2), (128, 64, 2), (64, 128, 2), (40, 24, 3), (72, 100, 2), (17, 4, 2)]


@pytest.mark.parametrize("dk,dv,H", TOKEN_SIZES)
@pytest.mark.parametrize("kind", ["general_delta", "gated_delta", "gated", "fixed", "forget_gate"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_one_token_of_every_request(kind, dk, dv, H, dtype):
    """Against float64: a sum of at most 128 products beside the state; 2e-6 of the state's size, and the output's rounding."""
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    g = torch.Generator(device=dev).manual_seed(dk + dv + H)
    slots = [4, 0, 7, 2, 9]
    S, G = len(slots), H if kind != "gated_delta" or H % 2 else H // 2
    rand = lambda *shape: torch.randn(*shape, device=dev, generator=g)  # noqa: E731
    K, V = G * dk, H * dv
    proj, state = rand(S, 5 + 2 * K + V + H * dk + 3), rand(10, H, dk, dv)
    offs = (5, 5 + K, 5 + 2 * K, 5 + 2 * K + V)
    decay, bias, a, gain, gate, gates = rand(S, H * dk), rand(H * dk), rand(H * dk), rand(V), rand(S, V + 2), rand(S, 2 * H + 1)
    q, k, v, z = (proj[:, o:o + n].double().reshape(S, h, -1) for o, n, h in zip(offs, (K, K, V, H * dk), (G, G, H, H)))
    kw, p, w, silu = {}, None, None, torch.nn.functional.silu
    unit = lambda x: x / (x.pow(2).sum(-1, keepdim=True) + 1e-6).sqrt()  # noqa: E731
    if kind == "general_delta":
        keep = torch.exp(-np.exp(-0.5) * torch.sigmoid(decay.double())).reshape(S, H, dk)
        p, w = unit(k), torch.sigmoid(z + a.double().reshape(H, dk)) * unit(k)
        kw = {"decay": decay, "a": a}
    elif kind == "gated_delta":
        a, bias = a[:H].contiguous(), bias[:H].contiguous()
        q, k = (unit(x).repeat_interleave(H // G, 1) for x in (q, k))
        q, beta = q * 0.3, torch.sigmoid(gates[:, :H].double())[:, :, None]
        keep = torch.exp(-torch.exp(a.double()) * torch.nn.functional.softplus(gates[:, H + 1:].double() + bias.double()))[:, :, None]
        p, w, v = k, beta * keep * k, beta * v
        kw = {"a": a, "bias": bias, "gates": gates, "off_b": 0, "off_dt": H + 1, "key_heads": G, "q_scale": 0.3}
    elif kind == "gated":
        q, keep = q * 0.3, (torch.nn.functional.logsigmoid(decay.double()) / 8).exp().reshape(S, H, dk)
        kw = {"decay": decay, "q_scale": 0.3, "tau": 8.0}
    elif kind == "fixed":
        a = torch.rand(H, device=dev, generator=g)
        q, k, v, keep = silu(q), silu(k), silu(v), a.double()[None, :, None]
        kw = {"a": a}
    else:
        a = torch.rand(H * dk, device=dev, generator=g)
        keep = (a.double() + (1 - a.double()) * torch.sigmoid(k.reshape(S, -1) + bias.double())).reshape(S, H, dk)
        q, k = silu(q), 1 - keep
        kw = {"a": a, "bias": bias}
    before = state.clone()
    old = state[slots].double()
    gone = w[..., None] * torch.einsum("shi,shij->shj", p, old)[:, :, None] if p is not None else 0.0
    new = old * keep[..., None] - gone + k[..., None] * v[:, :, None]
    o = torch.einsum("shij,shi->shj", new, q)
    step = _step(dev, [1] * S, slots)
    raw = ops.recurrence_token(kind, proj, offs, state, step, H, dk, dv, torch.float32, **kw)
    assert torch.equal(state[[1, 3, 5, 6, 8]], before[[1, 3, 5, 6, 8]])
    size = float(new.abs().max())
    torch.testing.assert_close(state[slots].double(), new, rtol=0, atol=2e-6 * size)
    torch.testing.assert_close(raw.double().reshape(S, H, dv), o, rtol=2e-5, atol=2e-5 * float(o.abs().max()))
    for act, f in (("sigmoid", torch.sigmoid), ("silu", silu), ("none", None)):
        state.copy_(before)
        wide = torch.zeros(S, V + 7, device=dev, dtype=dtype)
        ops.recurrence_token(kind, proj, offs, state, step, H, dk, dv, dtype, norm=(gain, 1e-5, None if f is None else gate, 2, act), out=wide,
                             out_off=3, **kw)
        want = (o / (o.pow(2).mean(-1, keepdim=True) + 1e-5).sqrt()).reshape(S, V) * gain.double()
        want = want if f is None else want * f(gate[:, 2:].double())
        tol = 1e-4 if dtype == torch.float32 else 1e-2
        torch.testing.assert_close(wide[:, 3:3 + V].double(), want, rtol=tol, atol=tol)
        assert not wide[:, :3].any() and not wide[:, 3 + V:].any()


@pytest.mark.parametrize("lens", [[1, 1, 1], [130, 1, 97]])
def test_states_off_the_16_byte_boundary(lens):
    """A state that is a view at an odd float is taken by every form, as it is where it starts on 16 bytes."""
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    g = torch.Generator(device=dev).manual_seed(8)
    H, d = 3, 64
    proj = torch.randn(sum(lens), 3 * H * d, device=dev, generator=g)
    decay = torch.tensor([0.5, 0.9, 0.99], device=dev)
    step = _step(dev, lens, [2, 0, 3])
    state = torch.randn(4, H, d, d, device=dev, generator=g)
    off = torch.zeros(state.numel() + 1, device=dev)[1:].view_as(state).copy_(state)
    assert off.is_contiguous() and off.data_ptr() % 16 != 0
    offs = (0, H * d, 2 * H * d)
    want = ops.decay_linear_attention(proj, offs, decay, state, step, H, d, d)
    got = ops.decay_linear_attention(proj, offs, decay, off, step, H, d, d)
    torch.testing.assert_close(got, want, rtol=2e-5, atol=2e-5 * float(want.abs().max()))
    torch.testing.assert_close(off, state, rtol=2e-5, atol=2e-5 * float(state.abs().max()))


@pytest.mark.parametrize("short", ["a", "bias", "gain", "gate"])
def test_vectors_that_do_not_fit_are_refused(short):
    """As `forget_gate_attention` refuses them: the kernel would read past their ends."""
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    H, d, S = 3, 64, 2
    x = {"a": torch.zeros(H * d, device=dev), "bias": torch.zeros(H * d, device=dev), "gain": torch.zeros(H * d, device=dev), "gate": torch.zeros(S, H * d, device=dev)}
    proj, state = torch.zeros(S, 3 * H * d, device=dev), torch.zeros(3, H, d, d, device=dev)
    run = lambda: ops.recurrence_token("forget_gate", proj, (0, H * d, 2 * H * d), state, _step(dev, [1] * S, [0, 1]), H, d, d, torch.float32,  # noqa: E731
                                       a=x["a"], bias=x["bias"], norm=(x["gain"], 1e-5, x["gate"], 0, "silu"))
    run()
    x[short] = x[short][:-1].contiguous()
    with pytest.raises(ops.KernelError):
        run()


@pytest.mark.parametrize("kind", ["gated", "fixed", "forget_gate", "gated_delta", "general_delta"])
def test_chunks_within_a_bound_on_their_scratch(monkeypatch, kind):
    """A step whose chunks would hold more than the bound runs them in groups, with the same bits and scratch for one group; where there is no room even for that
    the portions are walked, as they were before there were chunks."""
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    g = torch.Generator(device=dev).manual_seed(3)
    H, d, T = 2, 64, sum(LENS)
    C = H * d
    proj, z, v1, v2 = (torch.randn(*s, device=dev, generator=g) for s in ((T, 4 * C), (T, C), (C,), (C,)))
    lower, head, heads = torch.rand(C, device=dev, generator=g) * 0.9, torch.tensor([0.9, 0.99], device=dev), torch.zeros(H, device=dev) - 2
    offs = (0, C, 2 * C)
    run = {"gated": lambda s, t: ops.gated_linear_attention(proj, offs, z, s, t, H, d, d, 0.1, 8.0),
           "fixed": lambda s, t: ops.decay_linear_attention(proj, offs, head, s, t, H, d, d),
           "forget_gate": lambda s, t: ops.forget_gate_attention(proj, offs, v1, lower, s, t, H, d, d),
           "gated_delta": lambda s, t: ops.gated_delta_rule(proj, offs, z, 0, H, heads, heads, s, t, H, H, d, d, 0.1),
           "general_delta": lambda s, t: ops.delta_rule(proj, offs + (3 * C,), z, v2, s, t, H, d, d)}[kind]
    before = _state(g, H, d, d, dev)
    want_state = before.clone()
    want = run(want_state, _step(dev, LENS, SLOTS))
    per = 4 * H * (d * (d + 1) if kind in ("gated", "fixed", "forget_gate") else int(ops.lib().sllm_delta_chunked_scratch(d, d)))
    sizes, empty = [], ops._scratch
    for chunks in (1, 3, 4, 11):
        with monkeypatch.context() as m:
            m.setattr(ops, "CHUNK_SCRATCH_BYTES", chunks * per + per - 4)
            m.setattr(ops, "_scratch", lambda floats, device: sizes.append(4 * floats) or empty(floats, device))
            state = before.clone()
            assert torch.equal(run(state, _step(dev, LENS, SLOTS)), want) and torch.equal(state, want_state)
        assert per <= sizes.pop() <= chunks * per and not sizes
    with monkeypatch.context() as m:
        m.setattr(ops, "_scratch", lambda floats, device: None)
        state = before.clone()
        got = run(state, _step(dev, LENS, SLOTS))
    _close(got, want, "walked")
    _close(state, want_state, "states walked")
