"""The norms whose rows lie in registers, at the edges of their forms (one vector, whole blocks, one channel too many, rows in great number), against float64.  The bounds: a sum
of W squares in float32 is good to (W + 8) 2^-24 of itself, its root to half of that, a product of three roundings; bfloat16 rounds to 2^-8 of the result."""

import pytest
import torch

from tests.conftest import cuda_or_skip

pytestmark = pytest.mark.gpu


class _Step:
    def __init__(self, lens, dev):
        ends = torch.tensor(lens).cumsum(0)
        self.q_start = torch.cat([torch.zeros(1, dtype=torch.int64), ends]).to(device=dev, dtype=torch.int32)
        self.seq_of_token = torch.repeat_interleave(torch.arange(len(lens)), torch.tensor(lens)).to(device=dev, dtype=torch.int32)
        self.state_slots = torch.arange(len(lens), device=dev, dtype=torch.int32).flip(0).contiguous()


def _close(got, want, scale, W):
    eps = 2.0 ** -8 if got.dtype == torch.bfloat16 else 0.0
    return bool(((got.double() - want).abs() <= (eps + (W + 16) * 2.0 ** -24) * scale + 1e-30).all())


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T", [1, 3, 300])
@pytest.mark.parametrize("W", [4, 100, 128, 2048, 4096, 4100, 8192, 8196, 16388, 1001])
def test_rows_in_registers(W, T, dtype):
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    g = torch.Generator(device=dev).manual_seed(W + T)
    rand = lambda *s: torch.randn(*s, device=dev, generator=g)  # noqa: E731
    x, term, a, b, eps = rand(T, W), rand(2, T, W), rand(W), rand(W), 1e-5
    norm = lambda v: v * torch.rsqrt(v.pow(2).mean(-1, keepdim=True) + eps)  # noqa: E731
    # one norm, with and without partial sums to add
    for delta in (None, term[0].contiguous(), term):
        stream = x.clone()
        want = x.double() + (0 if delta is None else delta.double().sum(0) if delta.dim() == 3 else delta.double())
        y = ops.add_rmsnorm(stream, delta, a, eps, dtype)
        assert bool(((stream.double() - want).abs() <= 2.0 ** -22 * (x.abs() + term.abs().sum(0))).all())
        want = norm(stream.double()) * a
        assert _close(y, want, want.abs(), W)
    # two norms of a row
    p, q = ops.norm_pair(x, a, b, eps, dtype)
    for got, gain in ((p, a), (q, b)):
        assert _close(got, norm(x.double()) * gain, (norm(x.double()) * gain).abs(), W)
    # a norm before the term joins the stream and one behind it
    for t in (term[0].contiguous(), term):
        stream = x.clone()
        h = ops.post_add_norm(stream, t, a, eps, b, eps, dtype)
        add = norm((t.double().sum(0) if t.dim() == 3 else t.double())) * a
        assert bool(((stream.double() - (x + add)).abs() <= (W + 16) * 2.0 ** -24 * (x.abs() + add.abs() + 1)).all())
        want = norm(stream.double()) * b
        assert _close(h, want, want.abs(), W)


def test_wide_rows_keep_their_16_byte_loads():
    """The form a norm takes (0: a channel a load; 1, 2: one or two vectors of four a thread, in registers; 3: vectors of four, read twice; 4: many rows), on both sides of every border."""
    cuda_or_skip()
    from sllm_b200.ops._lib import lib
    form = lib().sllm_add_rmsnorm_form
    for H, few, many in ((4, 1, 4), (4096, 1, 4), (4100, 2, 4), (8192, 2, 4), (8196, 3, 4), (16384, 3, 4), (16388, 3, 3), (32768, 3, 3)):
        assert [form(1, H, 0, 1), form(63, H, 1, 1), form(64, H, 1, 1), form(64, H, 2, 1), form(64, H, 1, 0)] == [few, few, many, few, 0]
        assert form(1, H + 1, 0, 1) == form(64, H + 2, 0, 1) == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("lens", [[1], [1, 1, 1], [2, 5, 1], [200, 150, 1]])
@pytest.mark.parametrize("W,groups", [(128, 1), (512, 4), (2048, 4), (4096, 4), (2048, 16), (384, 3), (4608, 4), (640, 4)])
def test_groups_of_pieces_with_and_without_the_shift(W, groups, lens, dtype):
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    T, eps = sum(lens), 1e-5
    g = torch.Generator(device=dev).manual_seed(W + T)
    x, gain, mix = torch.randn(T, W, device=dev, generator=g), torch.randn(W, device=dev, generator=g), torch.rand(W, device=dev, generator=g)
    state = torch.randn(len(lens) + 1, W, device=dev, generator=g)
    step, before = _Step(lens, dev), state.clone()
    xd = x.double().reshape(T, groups, W // groups)
    h = (xd * torch.rsqrt(xd.pow(2).mean(-1, keepdim=True) + eps)).reshape(T, W) * gain
    plain = ops.group_norm_shift(x, None, gain, dtype, groups=groups, eps=eps)
    assert _close(plain, h, h.abs(), W // groups)
    got, shifted = ops.group_norm_shift(x, None, gain, dtype, groups=groups, eps=eps, mix=mix, state=state, step=step)
    assert torch.equal(got, plain)
    prev = torch.cat([h[:1], h[:-1]])
    for r, start in enumerate(step.q_start[:-1].tolist()):
        prev[start] = before[step.state_slots[r]].double()
    want = h + (prev - h) * mix
    assert _close(shifted, want, h.abs() + prev.abs(), W // groups)
    for r in range(len(lens)):
        last = int(step.q_start[r + 1]) - 1
        assert _close(state[step.state_slots[r]], h[last], h[last].abs(), W // groups)
    assert torch.equal(state[-1], before[-1])
