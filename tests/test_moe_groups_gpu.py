"""A mixture of experts with the tokens sorted by expert (moe_groups.cu, the grouped form of gemm_pair.cu): the sorting itself, the grouped product
with each of its epilogues, and whole mixtures in both forms, against one another and against float64 (the bound: two bfloat16 roundings of each input and
activation, 2^-8 of the terms' root sum of squares at worst, so 1e-2 of the result's)."""

import pytest
import torch

from tests.conftest import cuda_or_skip

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,top,E", [(1, 1, 1), (300, 2, 8), (257, 8, 8), (1000, 3, 40), (64, 1, 200), (2048, 2, 8)])
@pytest.mark.parametrize("lopsided", [False, True])
def test_every_choice_has_a_row_among_its_experts(T, top, E, lopsided):
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    g = torch.Generator(device=dev).manual_seed(T + E)
    score = torch.rand(T, E, device=dev, generator=g)
    if lopsided:
        score[:, 0] += 2
    idx = score.topk(top, -1).indices.int().contiguous()
    place, tile_expert, row_token = ops.moe_assign(idx, E)
    assert len(place.unique()) == T * top
    assert torch.equal(tile_expert[(place // 256).long()], idx)
    assert torch.equal(row_token[place.long()], torch.arange(T, device=dev, dtype=torch.int32)[:, None].expand(T, top))
    assert int((row_token >= 0).sum()) == T * top
    used = int(((torch.bincount(idx.flatten().long(), minlength=E) + 255) // 256).sum())
    assert int((tile_expert >= 0).sum()) == used and bool((tile_expert[used:] == -1).all())


@pytest.mark.parametrize("N,K,E", [(256, 64, 3), (1408, 192, 8), (72, 2048, 5), (520, 128, 2)])
@pytest.mark.parametrize("act", [None, "float", "gelu", "silu"])
def test_grouped_product(N, K, E, act):
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    if act == "silu" and N % 16:
        pytest.skip("the gated epilogue takes whole blocks of 8 pairs")
    g = torch.Generator(device=dev).manual_seed(N + K)
    tiles = torch.tensor([e for e in range(E) for _ in range(1 + e % 2)] + [-1, -1], dtype=torch.int32, device=dev)
    x = torch.randn(256 * len(tiles), K, device=dev, generator=g).bfloat16()
    rows = torch.randn(E * N, K, device=dev, generator=g).bfloat16() / K ** 0.5                # experts below one another
    got = ops.gemm_pair_grouped(x, rows, tiles, N, K, N, 0, torch.float32 if act == "float" else torch.bfloat16, act=None if act == "float" else act)
    cols = rows.reshape(E, N, K).transpose(0, 1).reshape(N, E * K).contiguous()                # experts beside one another
    side = ops.gemm_pair_grouped(x, cols, tiles, N, K, 0, K, torch.float32 if act == "float" else torch.bfloat16, act=None if act == "float" else act)
    ops.check_tcgen05_status()
    live = int((tiles >= 0).sum()) * 256
    y = torch.cat([x[256 * i:256 * (i + 1)].double() @ rows[N * int(e):N * (int(e) + 1)].double().T for i, e in enumerate(tiles.tolist()) if e >= 0])
    if act == "gelu":
        y = torch.nn.functional.gelu(y)
    if act == "silu":
        gate, up = y.reshape(live, N // 16, 2, 8).unbind(2)
        y = (torch.nn.functional.silu(gate) * up).reshape(live, N // 2)
    tol = 2e-5 if act == "float" else 1e-2
    torch.testing.assert_close(got[:live].double(), y, rtol=tol, atol=tol)
    assert torch.equal(got[:live], side[:live])


@pytest.mark.parametrize("M,N,K,cols,at", [(129, 72, 64, 128, 8), (300, 256, 200, 264, 64), (2048, 3584, 328, 1024, 512), (700, 2048, 64, 72, 0), (513, 520, 1000, 1000, 0)])
def test_a_product_with_some_of_a_matrixs_columns(M, N, K, cols, at):
    """The same bits as with these columns as a matrix of their own, whatever stands in the columns beside them."""
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    g = torch.Generator(device=dev).manual_seed(M + N)
    x = torch.randn(M, K, device=dev, generator=g).bfloat16()
    own = (torch.randn(N, K, device=dev, generator=g) / K ** 0.5).bfloat16()
    w = torch.full((N, cols), float("nan"), device=dev).bfloat16()
    w[:, at:at + K] = own
    for dtype in (torch.float32, torch.bfloat16):
        got, want = ops.gemm_pair(x, w, None, dtype, w_col=at), ops.gemm_pair(x, own, None, dtype)
        ops.check_tcgen05_status()
        assert torch.equal(got, want)
    for bad in (-8, at + 4, cols - K + 8):
        with pytest.raises(ops.KernelError):
            ops.gemm_pair(x, w, None, torch.float32, w_col=bad)


CASES = [("routed_experts", {"experts": 8, "top": 2, "groups": 4, "keep": 2, "scale": 2.0, "expert_ff": 192, "shared_ff": 384}),
         ("routed_experts", {"experts": 6, "top": 3, "scale": 1.0, "expert_ff": 64}),
         ("gated_experts", {"experts": 8, "top": 2, "expert_ff": 128, "limit": 7.0}),
         ("gated_experts", {"experts": 5, "top": 1, "expert_ff": 192, "activation": "silu", "scale": 2.0}),
         ("gated_experts", {"experts": 8, "top": 2, "expert_ff": 128, "activation": "silu", "router_bias": True, "shared_ff": 256})]


@pytest.mark.parametrize("kind,params", CASES)
@pytest.mark.parametrize("T", [129, 700])
def test_a_mixture_sorted_by_expert(monkeypatch, kind, params, T):
    import sllm_b200.ops as ops
    from sllm_b200.config.plan import PartSpec
    from sllm_b200.models import causal_lm  # noqa: F401  (registers the parts)
    from sllm_b200.parts.base import FEED_FORWARDS
    dev = cuda_or_skip()
    W = 256
    part = FEED_FORWARDS.build(PartSpec(kind, dict(params, hidden_size=W)), dtype=torch.bfloat16, device=dev)
    g = torch.Generator(device=dev).manual_seed(T)
    part.bind({s.name: torch.randn(*s.shape, device=dev, generator=g) / max(1, s.shape[-1]) ** 0.5 for s in part.tensor_specs()}.__getitem__)
    x = torch.randn(T, W, device=dev, generator=g).bfloat16()
    monkeypatch.setattr(ops, "moe_grouped_pays", lambda *a: False)
    want = part.forward(x, None)
    want = want.sum(0) if want.dim() == 3 else want
    monkeypatch.setattr(ops, "moe_grouped_pays", lambda *a: True)
    got = part.forward(x, None)
    stream = torch.randn(T, W, device=dev, generator=g)
    added = stream.clone()
    assert part.forward(x, None, residual=added) is None
    ops.check_tcgen05_status()
    assert float((got - want).norm() / want.norm()) < 1e-2
    torch.testing.assert_close(added, stream + got, rtol=1e-6, atol=1e-5)


def _in_float64(part, kind, params, tensors, x):
    """The mixture from the router's own choices and weights, expert by expert."""
    dense, idx, wts = part.route(x)
    t = {n: v.bfloat16().double() for n, v in tensors.items()}
    x, silu = x.double(), torch.nn.functional.silu

    def expert(n):
        if kind == "routed_experts":
            return torch.nn.functional.gelu(x @ t[f"{n}.up"].T) @ t[f"{n}.down"].T
        gate, up = x @ t[f"{n}.gate"].T, x @ t[f"{n}.up"].T
        if params.get("activation") == "silu":
            return (silu(gate) * up) @ t[f"{n}.down"].T
        gate, up = gate.clamp(max=params["limit"]), up.clamp(-params["limit"], params["limit"])
        return (gate * torch.sigmoid(1.702 * gate) * (up + 1)) @ t[f"{n}.down"].T
    out = sum(((idx == e) * wts).double().sum(-1, keepdim=True) * expert(f"e{e}") for e in range(params["experts"]))
    if params.get("shared_ff"):
        out = out + expert("shared") * (torch.sigmoid(x @ t["shared.sg"].T) if kind == "gated_experts" else 1.0)
    return out


@pytest.mark.parametrize("kind,params", CASES)
@pytest.mark.parametrize("sort", [False, True])
def test_a_mixture_in_float64(monkeypatch, kind, params, sort):
    import sllm_b200.ops as ops
    from sllm_b200.config.plan import PartSpec
    from sllm_b200.models import causal_lm  # noqa: F401  (registers the parts)
    from sllm_b200.parts.base import FEED_FORWARDS
    dev = cuda_or_skip()
    part = FEED_FORWARDS.build(PartSpec(kind, dict(params, hidden_size=256)), dtype=torch.bfloat16, device=dev)
    g = torch.Generator(device=dev).manual_seed(7)
    tensors = {s.name: torch.randn(*s.shape, device=dev, generator=g) / max(1, s.shape[-1]) ** 0.5 for s in part.tensor_specs()}
    part.bind(tensors.__getitem__)
    x = torch.randn(530, 256, device=dev, generator=g).bfloat16()
    monkeypatch.setattr(ops, "moe_grouped_pays", lambda *a: sort)
    y = part.forward(x, None)
    ops.check_tcgen05_status()
    y = (y.sum(0) if y.dim() == 3 else y).double()
    want = _in_float64(part, kind, params, tensors, x)
    assert float((y - want).norm() / want.norm()) < 1e-2
    worst = (y - want).norm(dim=1) / want.norm(dim=1).clamp(min=0.1 * float(want.norm(dim=1).mean()))
    assert float(worst.max()) < 3e-2                         # no token with another expert's rows or weights


@pytest.mark.parametrize("shared_ff", [100, 96])
def test_a_shared_expert_of_any_size_beside_experts_of_whole_tiles(shared_ff):
    """Long portions by the dispatch's own choice: no size that the product over all experts takes is refused."""
    import sllm_b200.ops as ops
    from sllm_b200.config.plan import PartSpec
    from sllm_b200.models import causal_lm  # noqa: F401  (registers the parts)
    from sllm_b200.parts.base import FEED_FORWARDS
    dev = cuda_or_skip()
    part = FEED_FORWARDS.build(PartSpec("gated_experts", {"hidden_size": 1024, "experts": 8, "top": 2, "expert_ff": 1024, "activation": "silu",
                                                           "shared_ff": shared_ff}), dtype=torch.bfloat16, device=dev)
    g = torch.Generator(device=dev).manual_seed(shared_ff)
    part.bind({s.name: torch.randn(*s.shape, device=dev, generator=g) / s.shape[-1] ** 0.5 for s in part.tensor_specs()}.__getitem__)
    x = torch.randn(4000, 1024, device=dev, generator=g).bfloat16()
    y = part.forward(x, None)
    ops.check_tcgen05_status()
    y = y.sum(0) if y.dim() == 3 else y
    one = part.forward(x[-100:].contiguous(), None)
    one = one.sum(0) if one.dim() == 3 else one
    assert float((y[-100:] - one).norm() / one.norm()) < 1e-2


@pytest.mark.parametrize("kind,params", CASES)
def test_no_room_for_the_sorted_rows(monkeypatch, kind, params):
    """Where the sorted form's buffers cannot be had, the mixture runs as it does for short portions, and a stream that it adds to has been added to once."""
    import sllm_b200.ops as ops
    from sllm_b200.config.plan import PartSpec
    from sllm_b200.models import causal_lm  # noqa: F401  (registers the parts)
    from sllm_b200.parts.base import FEED_FORWARDS
    dev = cuda_or_skip()
    part = FEED_FORWARDS.build(PartSpec(kind, dict(params, hidden_size=256)), dtype=torch.bfloat16, device=dev)
    g = torch.Generator(device=dev).manual_seed(5)
    part.bind({s.name: torch.randn(*s.shape, device=dev, generator=g) / max(1, s.shape[-1]) ** 0.5 for s in part.tensor_specs()}.__getitem__)
    x = torch.randn(300, 256, device=dev, generator=g).bfloat16()
    stream = torch.randn(300, 256, device=dev, generator=g)
    want, got = stream.clone(), stream.clone()
    monkeypatch.setattr(ops, "moe_grouped_pays", lambda *a: False)
    term = part.forward(x, None, residual=want)

    def full(*a, **kw):
        raise torch.OutOfMemoryError("no room (raised by the test)")
    for at in ("moe_gather", "moe_combine"):
        got.copy_(stream)
        with monkeypatch.context() as m:
            m.setattr(ops, "moe_grouped_pays", lambda *a: True)
            m.setattr(ops, at, full)
            same = part.forward(x, None, residual=got)
        assert torch.equal(got, want) and (same is None) == (term is None) and (term is None or torch.equal(same, term))


def test_tables_of_another_type_are_refused():
    """The kernels read them as 32-bit numbers: wider ones would be other experts, and other rows."""
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    idx = torch.zeros(300, 2, dtype=torch.int32, device=dev)
    place, tile_expert, row_token = ops.moe_assign(idx, 4)
    x, w = torch.zeros(300, 64, device=dev).bfloat16(), torch.zeros(64, 256, device=dev).bfloat16()
    rows = ops.moe_gather(x, row_token)
    y = ops.gemm_pair_grouped(rows, w, tile_expert, 64, 64, 0, 64, torch.float32)
    wts, stream = torch.zeros(300, 2, device=dev), torch.zeros(300, 64, device=dev)
    assert ops.moe_combine(y, place, wts, residual=stream) is None
    for bad in (lambda: ops.moe_assign(idx.long(), 4), lambda: ops.moe_assign(idx.float(), 4), lambda: ops.moe_assign(idx.reshape(-1), 4),
                lambda: ops.moe_gather(x, row_token.long()), lambda: ops.gemm_pair_grouped(rows, w, tile_expert.long(), 64, 64, 0, 64, torch.float32),
                lambda: ops.moe_combine(y, place.long(), wts), lambda: ops.moe_combine(y, place, wts.double()), lambda: ops.moe_combine(y, place, wts[:, :1].contiguous()),
                lambda: ops.moe_combine(y, place, wts, shared=stream[:, :32].contiguous()), lambda: ops.moe_combine(y, place, wts, residual=stream.bfloat16())):
        with pytest.raises(ops.KernelError):
            bad()
