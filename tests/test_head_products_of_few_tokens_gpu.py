"""Per-head products of at most 32 tokens (latent.cu) at token counts around its tiles of 8, outputs that end inside a warp's 16 and reductions beside its 128
columns, with both kinds of gate, against float64.  The bound: the bfloat16 rounding of the result and of a float32 input's elements, 2^-9 each
of the terms' magnitudes at worst."""

import pytest
import torch

from tests.conftest import cuda_or_skip

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 7, 8, 9, 16, 17, 32, 33])
@pytest.mark.parametrize("H,din,dout", [(16, 128, 128), (3, 32, 24), (5, 96, 40), (2, 256, 130), (1, 160, 16)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("gate", [None, "head", "element"])
def test_few_tokens(T, H, din, dout, dtype, gate):
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    g = torch.Generator(device=dev).manual_seed(T + din)
    off, stride, ostride = 8, din + 8, dout + 3
    x = torch.randn(T, off + H * stride, device=dev, generator=g).to(dtype)
    w = (torch.randn(H, dout, din, device=dev, generator=g) / din ** 0.5).bfloat16()
    logits = torch.randn(T, 4 + H * dout, device=dev, generator=g)
    got = ops.head_linear(x, off, w, torch.bfloat16, gate=None if gate is None else logits, goff=4 if gate else 0, gate_elem=gate == "element",
                          xstride=stride, ostride=ostride)
    xs = x[:, off:].double().reshape(T, H, stride)[..., :din]
    want, size = torch.einsum("thi,hoi->tho", xs, w.double()), torch.einsum("thi,hoi->tho", xs.abs(), w.double().abs())
    if gate:
        s = torch.sigmoid((logits[:, 4:4 + H, None] if gate == "head" else logits[:, 4:].reshape(T, H, dout)).double())
        want, size = want * s, size * s
    heads = torch.stack([got[:, h * ostride:h * ostride + dout] for h in range(H)], 1).double()
    assert bool(((heads - want).abs() <= 2.0 ** -8 * size + 1e-6).all())
