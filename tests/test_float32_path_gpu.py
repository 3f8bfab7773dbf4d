"""The float32 products and attention at the sizes where their forms and splits change: rows around 1, 2, 4, 8, 16, 32, 64 and 128 (skinny form, 32,
64 and 128-row tiles), reductions cut into 1 to 8 segments, lengths that are no multiple of 4 (scalar copies) or of 32 (a ragged last
step).  The bound of a product: K rounded multiply-adds in at least two chains, so the error stays under sqrt(K) 2^-24 of the terms' root sum of
squares (about 1 here) times a small factor: 1e-5."""

import pytest
import torch

from tests.conftest import cuda_or_skip

pytestmark = pytest.mark.gpu
ROWS = [1, 2, 3, 5, 8, 9, 16, 17, 32, 33, 64, 65, 128, 129, 300]


@pytest.mark.parametrize("N,K", [(896, 896), (1152, 900), (20000, 96), (9728, 256), (31, 4864), (130, 333), (33, 70), (40, 2)])
def test_products_of_every_form_agree_in_every_bit(N, K):
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    g = torch.Generator(device=dev).manual_seed(N + K)
    x = torch.randn(max(ROWS), K, device=dev, generator=g)
    w = torch.randn(N, K, device=dev, generator=g) / K ** 0.5
    b = torch.randn(N, device=dev, generator=g)
    full = ops.linear(x, w, b, torch.float32)
    want = x.double() @ w.double().t() + b.double()
    torch.testing.assert_close(full.double(), want, rtol=1e-5, atol=1e-5)
    for m in ROWS:
        assert torch.equal(ops.linear(x[-m:].contiguous(), w, b, torch.float32), full[-m:]), m
    # operands off the 16-byte boundary take the scalar copies
    flat = torch.empty(x.numel() + 1, device=dev)
    flat[1:] = x.reshape(-1)
    off = flat[1:].view_as(x)
    assert torch.equal(ops.linear(off, w, b, torch.float32), full)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("hd,ps", [(64, 16), (128, 8), (40, 4), (17, 16), (256, 16), (320, 16)])
@pytest.mark.parametrize("window", [None, 45])
def test_attention_around_blocks_of_32_keys(dtype, hd, ps, window):
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    g = torch.Generator(device=dev).manual_seed(hd + ps)
    nq, nkv, ctx = 6, 2, [1, 31, 32, 33, 64, 257, 300]
    pages = sum(-(-c // ps) for c in ctx)
    kc, vc = (torch.randn(pages, nkv, ps, hd, device=dev, generator=g).to(dtype) for _ in range(2))
    order, at = torch.randperm(pages, device=dev, generator=g).int(), 0
    bt = torch.full((len(ctx), -(-max(ctx) // ps)), -1, dtype=torch.int32, device=dev)
    for i, c in enumerate(ctx):
        n = -(-c // ps)
        bt[i, :n] = order[at:at + n]
        at += n
    pos = torch.tensor([c - 1 for c in ctx], dtype=torch.int32, device=dev)
    seq = torch.arange(len(ctx), dtype=torch.int32, device=dev)
    q = torch.randn(len(ctx), nq * hd, device=dev, generator=g).to(dtype)
    got = ops.attention_simt(q, kc, vc, bt, pos, seq, nq, nkv, hd, hd ** -0.5, window).double().reshape(len(ctx), nq, hd)
    for i, c in enumerate(ctx):
        lo = max(0, c - window) if window else 0
        rows = [(int(bt[i, j // ps]), j % ps) for j in range(lo, c)]
        k, v = (torch.stack([x[p, :, o] for p, o in rows]).double().repeat_interleave(nq // nkv, 1) for x in (kc, vc))
        s = torch.einsum("hd,jhd->hj", q[i].double().reshape(nq, hd), k) * hd ** -0.5
        want = torch.einsum("hj,jhd->hd", torch.softmax(s, -1), v)
        tol = 2e-5 if dtype == torch.float32 else 1e-2
        torch.testing.assert_close(got[i], want, rtol=tol, atol=tol)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("hd,nkv", [(64, 2), (100, 2), (128, 2), (132, 2), (255, 2), (300, 1), (576, 1), (640, 1)])
@pytest.mark.parametrize("window,softcap", [(None, 0.0), (90, 5.0), (150, 0.0)])
def test_attention_four_keys_a_warp(dtype, hd, nkv, window, softcap):
    """Wide heads and, of narrow ones, contexts and windows on both sides of the line between the two ways through the keys, with all that a score and a
    head pass, pages before the window given back: against the same in float32."""
    import sllm_b200.ops as ops
    from tests import torch_ops as ref
    dev = cuda_or_skip()
    g = torch.Generator(device=dev).manual_seed(hd)
    nq, ps, ctx = 4, 8, [1, 3, 4, 5, 95, 96, 97, 98, 159, 160, 161, 162, 290]
    per = -(-max(ctx) // ps)
    kc, vc = (torch.randn(len(ctx) * per, nkv, ps, hd, device=dev, generator=g).to(dtype) for _ in range(2))
    bt = torch.randperm(len(ctx) * per, device=dev, generator=g).int().reshape(len(ctx), per).contiguous()
    for i, c in enumerate(ctx):
        if window:
            bt[i, :max(0, c - window) // ps] = -1
    pos = torch.tensor([c - 1 for c in ctx], dtype=torch.int32, device=dev)
    seq = torch.arange(len(ctx), dtype=torch.int32, device=dev)
    q = torch.randn(len(ctx), nq * hd, device=dev, generator=g).to(dtype)
    sink = torch.randn(nq, device=dev, generator=g)
    gate = (torch.randn(len(ctx), nq + 3, device=dev, generator=g), 3)
    args = (bt, pos, seq, nq, nkv, hd, hd ** -0.5, window, None, sink, softcap, gate)
    got = ops.attention_simt(q, kc, vc, *args).float()
    want = ref.attention_simt(q.float(), kc.float(), vc.float(), *args)
    tol = 2e-5 if dtype == torch.float32 else 1e-2           # (bfloat16: the result's own rounding, 2^-8)
    torch.testing.assert_close(got, want, rtol=tol, atol=tol)


@pytest.mark.parametrize("N,K", [(64, 64), (512, 512), (2304, 768), (896, 1792), (257, 1001), (3000, 130), (4100, 36)])
def test_every_number_of_rows_takes_a_form_of_the_same_bits(N, K):
    """Rows from one tile to many waves of them: tiles of all sizes, segments over a cluster and one after the other."""
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    g = torch.Generator(device=dev).manual_seed(N + K)
    x = torch.randn(4133, K, device=dev, generator=g)
    w = torch.randn(N, K, device=dev, generator=g) / K ** 0.5
    b = torch.randn(N, device=dev, generator=g)
    few = torch.cat([ops.linear(x[i:i + 16].contiguous(), w, b, torch.float32) for i in range(0, 64, 16)])
    torch.testing.assert_close(few.double(), x[:64].double() @ w.double().t() + b.double(), rtol=1e-5, atol=1e-5)
    last = ops.linear(x[-9:].contiguous(), w, b, torch.float32)
    for m in (17, 31, 64, 100, 129, 257, 543, 1025, 2050, 4133):
        y = ops.linear(x[-m:].contiguous() if m > 64 else x[:m].contiguous(), w, b, torch.float32)
        if m > 64:
            assert torch.equal(y[-9:], last), m
            torch.testing.assert_close(y[:7].double(), x[-m:][:7].double() @ w.double().t() + b.double(), rtol=1e-5, atol=1e-5)
        else:
            assert torch.equal(y, few[:m]), m
