"""The weight-streaming product's other forms: CTAs that walk more than one group of rows (matrices of many rows) or take four side by side, clusters that share the columns
(matrices of few), and the gate|up product with its activation, at row counts and reductions that leave remainders of both.  The bounds: K float32
additions of exact products, 2^-24 of the sum of their magnitudes each; for the activation also 2^-8 of the result, its bfloat16 rounding."""

import pytest
import torch

from tests.conftest import cuda_or_skip

pytestmark = pytest.mark.gpu


def _product(dev, M, N, K):
    g = torch.Generator(device=dev).manual_seed(M + N + K)
    x = torch.randn(M, K, device=dev, generator=g).bfloat16()
    w = (torch.randn(N, K, device=dev, generator=g) / K ** 0.5).bfloat16()
    b = torch.randn(N, device=dev, generator=g)
    y = x.double() @ w.double().T + b
    bound = (K + 1) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T + b.abs())
    return g, x, w, b, y, bound


@pytest.mark.parametrize("M", [1, 8, 9, 16])
@pytest.mark.parametrize("N,K", [(24, 2080), (200, 4128), (1000, 4160), (2048, 1056), (5000, 64), (9480, 96), (10001, 320), (33000, 32), (18944, 64), (18945, 352)])
def test_rows_and_columns_in_parts(M, N, K):
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    g, x, w, b, y, bound = _product(dev, M, N, K)
    got = ops.linear_ws(x, w, b, torch.float32)
    assert bool(((got - y).abs() <= bound).all())
    stream = torch.randn(M, N, device=dev, generator=g)
    added = stream.clone()
    ops.linear_ws(x, w, b, torch.float32, residual=added)
    assert bool(((added - (stream + y)).abs() <= bound + 2.0 ** -23 * (stream.abs() + y.abs())).all())
    gain = torch.randn(N, device=dev, generator=g)
    again = stream.clone()
    xg, owed = ops.linear_ws(x, w, b, torch.float32, residual=again, next_gain=gain)
    assert torch.equal(again, added) and torch.equal(xg, (added * gain).bfloat16())
    torch.testing.assert_close(owed.ssq[:, :owed.parts].double().sum(1), added.double().pow(2).sum(1), rtol=N * 2.0 ** -24, atol=0)
    alone = M - 1 if M <= 8 else M - 9                       # (from 9 tokens on the rows may be dealt in another form)
    assert torch.equal(ops.linear_ws(x[alone:].contiguous(), w, b, torch.float32)[-1], got[-1])


@pytest.mark.parametrize("M", [1, 8, 9, 16])
@pytest.mark.parametrize("N,K", [(16, 32), (4736, 96), (4752, 320), (8208, 1056), (9728, 896), (11264, 2048), (22016, 64), (37888, 96)])
@pytest.mark.parametrize("act", ["silu", "gelu_tanh"])
def test_gate_and_up_with_their_activation(M, N, K, act):
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    _, x, w, b, y, bound = _product(dev, M, N, K)
    gate, up = y.reshape(M, N // 16, 2, 8).unbind(2)
    gate_off, up_off = bound.reshape(M, N // 16, 2, 8).unbind(2)
    fn = torch.nn.functional.silu if act == "silu" else lambda v: torch.nn.functional.gelu(v, approximate="tanh")
    want = fn(gate) * up
    # both activations rise by at most 1.13 a unit; the float32 activation itself is good to 1e-5 of its argument
    off = 2.0 ** -8 * want.abs() + 1.2 * (gate_off * up.abs() + up_off * gate.abs()) + 1e-5 * gate.abs() * up.abs() + 1e-30
    got = ops.linear_ws_gated(x, w, b, act).reshape(M, N // 16, 8)
    assert bool(((got - want).abs() <= off).all())
    alone = M - 1 if M <= 8 else M - 9
    assert torch.equal(ops.linear_ws_gated(x[alone:].contiguous(), w, b, act)[-1], got[-1].reshape(-1))


@pytest.mark.parametrize("M", [17, 24, 25, 32])
@pytest.mark.parametrize("N,K,takes", [(896, 896, True), (896, 4864, True), (2048, 5632, True), (2048, 544, True), (1536, 8192, False), (1000, 480, False)])
def test_more_tokens_on_small_matrices(M, N, K, takes):
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    assert ops.ws_supports(M, N, K) == takes
    g, x, w, b, y, bound = _product(dev, M, N, K)
    assert bool(((ops.linear_ws(x, w, b, torch.float32) - y).abs() <= bound).all())
    stream = torch.randn(M, N, device=dev, generator=g)
    added = stream.clone()
    ops.linear_ws(x, w, b, torch.float32, residual=added)
    assert bool(((added - (stream + y)).abs() <= bound + 2.0 ** -23 * (stream.abs() + y.abs())).all())


@pytest.mark.parametrize("M", [1, 8, 9, 16, 24])
@pytest.mark.parametrize("N,K", [(256, 1024), (1000, 1536), (2048, 1536), (512, 2048), (130, 2080), (2048, 2048), (20000, 1024), (19000, 1280)])
def test_around_the_reductions_that_are_cut(M, N, K):
    """Reductions on both sides of the lines from which clusters share them and from which rows are walked."""
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    g, x, w, b, y, bound = _product(dev, M, N, K)
    assert bool(((ops.linear_ws(x, w, b, torch.float32) - y).abs() <= bound).all())
    stream = torch.randn(M, N, device=dev, generator=g)
    added = stream.clone()
    ops.linear_ws(x, w, b, torch.float32, residual=added)
    assert bool(((added - (stream + y)).abs() <= bound + 2.0 ** -23 * (stream.abs() + y.abs())).all())


@pytest.mark.parametrize("N,K,slices", [(2560, 2560, True), (3072, 3072, True), (2048, 2048, False), (4096, 2048, False), (3584, 3584, False)])
def test_partial_sums_for_those_who_add_them(N, K, slices):
    """17 to 32 tokens and rows for one to one and a half CTAs an SM: a consumer that adds partial sums gets slices of K, one that cannot the whole product, and both
    are the product."""
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    if ops.num_sms() != 148:
        pytest.skip("the sizes are those of 148 SMs")
    _, x, w, _, y, bound = _product(dev, 24, N, K)
    y, bound = x.double() @ w.double().T, bound + 1
    parts = ops.linear(x, w, None, torch.float32, True)
    assert (parts.dim() == 3) == slices and ops.can_accumulate(x, w) == (not slices)
    for got in (parts.double().sum(0) if slices else parts, ops.linear(x, w, None, torch.float32)):
        assert got.dim() == 2 and float((got - y).norm() / y.norm()) < 1e-5


@pytest.mark.parametrize("M", [1, 8, 9, 16])
@pytest.mark.parametrize("N,K", [(8208, 128), (9728, 896), (17920, 1536), (22016, 4096)])
@pytest.mark.parametrize("parts", [1, 56, 296, 592])
def test_gate_and_up_with_a_norm_owed_on_their_input(M, N, K, parts):
    """Groups of rows side by side and one after the other, with the tokens' partial sums of squares of every size of table a producer leaves.  The bound: that of the
    product, times the row's scale, 2^-20 more for the scale's own sum and root."""
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    g, x, w, b, _, _ = _product(dev, M, N, K)
    ssq = torch.full((M, (parts + 3) & ~3), float("nan"), device=dev)          # (what lies beyond the parts is never read)
    ssq[:, :parts] = torch.rand(M, parts, device=dev, generator=g) * 4 * K / parts
    eps = 1e-5
    scale = (ssq[:, :parts].double().sum(1, keepdim=True) / K + eps).rsqrt()
    plain = x.double() @ w.double().T
    y = plain * scale + b
    bound = (K + 1) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T * scale + b.abs()) + 2.0 ** -20 * plain.abs() * scale
    for act, fn in (("silu", torch.nn.functional.silu), ("gelu_tanh", lambda v: torch.nn.functional.gelu(v, approximate="tanh"))):
        gate, up = y.reshape(M, N // 16, 2, 8).unbind(2)
        gate_off, up_off = bound.reshape(M, N // 16, 2, 8).unbind(2)
        want = fn(gate) * up
        off = 2.0 ** -8 * want.abs() + 1.2 * (gate_off * up.abs() + up_off * gate.abs()) + 1e-5 * gate.abs() * up.abs() + 1e-30
        got = ops.linear_ws_gated(x, w, b, act, scale=ops.RowScale(ssq, parts, eps, K)).reshape(M, N // 16, 8)
        assert bool(((got - want).abs() <= off).all())


@pytest.mark.parametrize("M", [17, 24, 32])
@pytest.mark.parametrize("N,K", [(896, 896), (896, 4864), (2048, 5632), (2048, 2048)])
def test_the_next_norms_input_from_more_tokens(M, N, K):
    """17 to 32 tokens on small matrices, the columns shared by clusters: the stream, the next norm's input and its partial sums, as the dispatch has them made."""
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    g, x, w, b, y, bound = _product(dev, M, N, K)
    assert ops.can_accumulate_norm(x, w)
    stream, gain = torch.randn(M, N, device=dev, generator=g), torch.randn(N, device=dev, generator=g)
    added = stream.clone()
    xg, owed = ops.linear_accumulate_norm(x, w, b, added, gain, 1e-6)
    assert bool(((added - (stream + y)).abs() <= bound + 2.0 ** -23 * (stream.abs() + y.abs())).all())
    assert torch.equal(xg, (added * gain).bfloat16()) and owed.width == N and owed.eps == 1e-6 and owed.parts <= ops.MAX_SCALE_PARTS_ROWS32
    torch.testing.assert_close(owed.ssq[:, :owed.parts].double().sum(1), added.double().pow(2).sum(1), rtol=N * 2.0 ** -24, atol=0)


@pytest.mark.parametrize("M", [1, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("N,K", [(16, 128), (1000, 896), (4864, 896), (7168, 1536), (7184, 1536), (9728, 896), (200, 3200), (64, 6400), (8192, 1664)])
def test_streams_with_resident_activations(M, N, K):
    """The streaming kernel where all activations fit its shared memory and just beyond: plain, with the activation, with a norm owed on the input (tables of one, some and
    many partial sums, the rest of them never read), rows and tokens that leave remainders."""
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    g, x, w, b, y, bound = _product(dev, M, N, K)
    assert bool(((ops.linear_stream(x, w, b, torch.float32) - y).abs() <= bound).all())
    if N % 16:
        return
    for parts in (0, 1, 57, 592):
        scale, plain, off = 1.0, x.double() @ w.double().T, (K + 1) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)
        if parts == 0:
            got = ops.linear_stream(x, w, None, torch.bfloat16, silu=True)
        else:
            ssq = torch.full((M, (parts + 3) & ~3), float("nan"), device=dev)
            ssq[:, :parts] = torch.rand(M, parts, device=dev, generator=g) * 4 * K / parts
            scale = (ssq[:, :parts].double().sum(1, keepdim=True) / K + 1e-5).rsqrt()
            got = torch.empty(M, N // 2, dtype=torch.bfloat16, device=dev)
            ops.call("sllm_linear_stream_silu_scaled", x.data_ptr(), w.data_ptr(), got.data_ptr(), M, N, K, *ops.RowScale(ssq, parts, 1e-5, K).args(), ops._stream())
        z, zo = plain * scale, off * scale + 2.0 ** -20 * (plain * scale).abs()
        gate, up = z.reshape(M, N // 16, 2, 8).unbind(2)
        gate_off, up_off = zo.reshape(M, N // 16, 2, 8).unbind(2)
        want = torch.nn.functional.silu(gate) * up
        lim = 2.0 ** -8 * want.abs() + 1.2 * (gate_off * up.abs() + up_off * gate.abs()) + 1e-5 * gate.abs() * up.abs() + 1e-30
        assert bool(((got.reshape(M, N // 16, 8) - want).abs() <= lim).all())


@pytest.mark.parametrize("M", [1, 16, 33, 128])
@pytest.mark.parametrize("N,K", [(1, 8), (8, 2048), (9, 4096), (15, 4104), (8, 264), (7, 11008)])
def test_few_columns(M, N, K):
    """Products narrower than a tile: no library kernel, both result types, with and without a bias."""
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    _, x, w, b, y, bound = _product(dev, M, N, K)
    before = ops.launches["library"]
    assert bool(((ops.linear(x, w, b, torch.float32) - y).abs() <= bound).all())
    plain = y - b
    assert bool(((ops.linear(x, w, None, torch.bfloat16) - plain).abs() <= bound + 2.0 ** -8 * plain.abs()).all())
    assert ops.launches["library"] == before


def test_few_columns_of_what_the_kernel_does_not_read():
    """Few columns of another type or off a 16-byte border, a bias that is broadcast or of another type: the library's product takes them, as it takes any; operands that do not fit one another and
    a bias of another length are refused."""
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    g = torch.Generator(device=dev).manual_seed(3)
    for dtype in (torch.float16, torch.float64):
        x, w = torch.randn(5, 64, device=dev, generator=g, dtype=torch.float32).to(dtype), torch.randn(9, 64, device=dev, generator=g, dtype=torch.float32).to(dtype)
        want = x.double() @ w.double().T
        assert bool(((ops.linear(x, w, None, dtype) - want).abs() <= torch.finfo(dtype).eps * want.abs() + 65 * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)).all())
    x, w = torch.randn(5, 64, device=dev, generator=g).bfloat16(), torch.randn(9, 64, device=dev, generator=g).bfloat16()
    b = torch.randn(9, device=dev, generator=g)
    y, bound = x.double() @ w.double().T, 66 * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T) + 2.0 ** -22
    shifted = torch.empty(5 * 64 + 1, device=dev, dtype=torch.bfloat16)[1:].view(5, 64).copy_(x)
    for xs, bias in ((shifted, b), (x, b[:1]), (x, b.bfloat16()), (x, b.double())):
        before = ops.launches["library"]
        assert bool(((ops.linear(xs, w, bias, torch.float32) - (y + bias.double())).abs() <= bound + 2.0 ** -22 * (y.abs() + bias.abs())).all())
        assert ops.launches["library"] == before + 1
    for xs, ws, bias in ((x, w[:, :56].contiguous(), None), (x[:, :56].contiguous(), w, None), (x, w, b[:8].contiguous()), (x, w.reshape(9, 8, 8), None)):
        with pytest.raises((RuntimeError, ops.KernelError)):
            ops.linear(xs, ws, bias, torch.float32)


def test_which_streams_keep_their_activations():
    """The line between the two streaming kernels (whose sums have the same order and so the same bits), on both sides of each of its borders, for 148 SMs."""
    import sllm_b200.ops as ops
    cuda_or_skip()
    if ops.num_sms() != 148:
        pytest.skip("the sizes are those of 148 SMs")
    form = ops.lib().sllm_linear_stream_resident
    store, silu = 0, 1
    for M, N, K, epilogue, scaled, want in [
            (1, 9472, 256, store, 0, 1), (1, 9488, 256, store, 0, 0), (8, 1024, 256, silu, 1, 0), (32, 1024, 256, silu, 0, 0), (32, 1024, 384, silu, 0, 0), (32, 1024, 512, silu, 0, 1),
            (32, 7168, 896, store, 0, 1), (32, 7184, 896, store, 0, 0), (32, 7184, 896, silu, 1, 1), (8, 18944, 384, store, 0, 1), (8, 18960, 384, store, 0, 0),
            (8, 28416, 1536, store, 0, 1), (8, 32000, 1536, store, 0, 0), (8, 40960, 1536, store, 0, 1), (8, 151936, 1536, store, 0, 1), (8, 28416, 896, silu, 1, 0), (8, 18944, 896, silu, 1, 1),
            (16, 18944, 2048, store, 0, 1), (16, 18960, 2048, store, 0, 0), (16, 32000, 2048, store, 0, 0), (16, 4736, 3200, store, 0, 1), (16, 4752, 3200, store, 0, 0), (16, 64, 3328, store, 0, 0),
            (8, 4736, 6400, store, 0, 1), (8, 4752, 6400, store, 0, 0), (8, 9472, 4864, store, 0, 1), (8, 4752, 4608, store, 0, 0), (8, 64, 6528, store, 0, 0), (33, 64, 128, store, 0, 0)]:
        assert form(M, N, K, epilogue, scaled) == want, (M, N, K, epilogue, scaled)


def _silu_of(z, off):
    """silu(gate) * up of rows interleaved by eight, in float64, and how far it is off where gate and up are off by ``off``."""
    M, N = z.shape
    gate, up = z.reshape(M, N // 16, 2, 8).unbind(2)
    gate_off, up_off = off.reshape(M, N // 16, 2, 8).unbind(2)
    want = torch.nn.functional.silu(gate) * up
    lim = 2.0 ** -8 * want.abs() + 1.2 * (gate_off * up.abs() + up_off * gate.abs()) + 1e-5 * gate.abs() * up.abs() + 1e-30
    return want.reshape(M, N // 2), lim.reshape(M, N // 2)


@pytest.mark.parametrize("M", [16, 17, 32, 33])
@pytest.mark.parametrize("N,K", [(12272, 1024), (12288, 1024), (6144, 2048), (14080, 896), (18944, 1024), (19072, 1024)])
def test_medium_matrices_of_17_to_32_tokens(M, N, K, monkeypatch):
    """Both sides of the lines between the streaming kernel and the one on tensor memory (2^23.6 elements, 1,024 columns with the activation, one tile an SM): which one runs, with and without the
    activation, and what neither leaves is refused."""
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    g, x, w, b, y, bound = _product(dev, M, N, K)
    ran = []
    for name in ("linear_tc", "linear_stream", "linear_ws"):
        monkeypatch.setattr(ops, name, lambda *a, _f=getattr(ops, name), _n=name, **k: (ran.append(_n), _f(*a, **k))[1])
    on_tensor_memory = 17 <= M <= 32 and N * K >= 12 << 20 and -(-N // 128) <= ops.num_sms()
    assert bool(((ops.linear(x, w, b, torch.float32) - y).abs() <= bound).all())
    if 17 <= M <= 32:
        assert ran == ["linear_tc" if on_tensor_memory else "linear_stream"]
    if M <= 32:
        with pytest.raises(ops.KernelError):                  # (no kernel for few tokens leaves float16)
            ops.linear(x, w, b, torch.float16)
    ran.clear()
    plain, off = x.double() @ w.double().T, (K + 1) * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)
    want, lim = _silu_of(plain, off)
    assert bool(((ops.linear_silu_mul(x, w, 8, torch.bfloat16) - want).abs() <= lim).all())
    if 17 <= M <= 32:
        assert ran == ["linear_tc" if on_tensor_memory and K >= 1024 else "linear_stream"]
    if M <= 32:                                              # an input whose norm is owed is taken on either side
        ssq = torch.rand(M, 56, device=dev, generator=g) * 4 * K / 56
        scale = (ssq.double().sum(1, keepdim=True) / K + 1e-5).rsqrt()
        want, lim = _silu_of(plain * scale, off * scale + 2.0 ** -20 * (plain * scale).abs())
        assert ops.silu_scaled_supports(x, w, 8, torch.bfloat16)
        assert bool(((ops.linear_silu_mul(x, w, 8, torch.bfloat16, scale=ops.RowScale(ssq, 56, 1e-5, K)) - want).abs() <= lim).all())
        assert ops.silu_scaled_pays(x, w, 8, torch.bfloat16) == (not (on_tensor_memory and (N, K) in ((6144, 2048), (18944, 1024))))


def test_rotary_epilogue_behind_the_kernel_that_makes_positions_and_slots():
    """Positions and slots that the kernel just before writes are the ones that count, call after call: the same queries, keys and values as from buffers that were there long before."""
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    g = torch.Generator(device=dev).manual_seed(5)
    M, K, nq, nkv, hd, ps, pages = 8, 256, 4, 2, 64, 16, 40
    x, w = torch.randn(M, K, device=dev, generator=g).bfloat16(), torch.randn((nq + 2 * nkv) * hd, K, device=dev, generator=g).bfloat16()
    b, table = torch.randn((nq + 2 * nkv) * hd, device=dev, generator=g), torch.randn(4096, 2, hd // 2, device=dev, generator=g)
    many = [(torch.randint(0, 4096, (M,), device=dev, generator=g, dtype=torch.int32), torch.randperm(pages * ps, device=dev, generator=g)[:M].int()) for _ in range(40)]

    def caches():
        return [torch.zeros(pages, nkv, ps, hd, device=dev, dtype=torch.bfloat16) for _ in range(2)]
    call = lambda pos, slots, kv: ops.linear_rope_kv_write(x, w, b, pos, table, hd, nq, nkv, hd, slots, *kv)  # noqa: E731
    kept, made = caches(), caches()
    torch.cuda.synchronize()
    want = [call(pos, slots, kept) for pos, slots in many]
    pos, slots = torch.zeros(M, device=dev, dtype=torch.int32), torch.zeros(M, device=dev, dtype=torch.int32)
    got = []
    for p, s in many:
        torch.add(p, 0, out=pos)
        torch.add(s, 0, out=slots)
        got.append(call(pos, slots, made))
    assert all(torch.equal(a, c) for a, c in zip(got, want)) and all(torch.equal(a, c) for a, c in zip(made, kept))


def test_rotary_epilogue_of_17_to_32_tokens_with_a_norm_owed():
    """Only where the norm is owed, up to 1,024 columns and rows for two CTAs an SM; the product itself is tested with the kernels."""
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    cache, table = torch.empty(4, 2, 16, 64, device=dev, dtype=torch.bfloat16), torch.empty(8, 2, 32, device=dev)

    def takes(M, nq, nkv, K, owed):
        x, w = torch.empty(M, K, device=dev, dtype=torch.bfloat16), torch.empty((nq + 2 * nkv) * 64, K, device=dev, dtype=torch.bfloat16)
        return ops.qkv_rope_supports(x, w, table, 64, nq, nkv, 64, cache, owed=owed)
    for M, nq, nkv, K, plain, owed in [(16, 14, 2, 896, True, True), (17, 14, 2, 896, False, True), (32, 14, 2, 1024, False, True), (17, 14, 2, 1056, False, False), (33, 14, 2, 896, False, False)]:
        assert (takes(M, nq, nkv, K, False), takes(M, nq, nkv, K, True)) == (plain, owed), (M, nq, nkv, K)
    if ops.num_sms() == 148:
        assert takes(32, 14, 30, 1024, True) and not takes(32, 14, 31, 1024, True)
