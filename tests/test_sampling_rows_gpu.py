"""Rows that eight blocks share and rows of one block, around the sizes where that changes: the greedy choice, top-k with and without top-p on flat
rows and on peaked ones (the k-th largest logit far below the largest), ties at the cut, logits that are minus infinity or not a number.  The
choice is exact: against the same steps in float64, at uniforms that lie no closer than 1e-6 to a step of the cumulative probability."""

import numpy as np
import pytest
import torch

from tests.conftest import ROOT, cuda_or_skip

pytestmark = pytest.mark.gpu


def _choose(row, t, k, p, u):
    """(the id, the distance of u to the nearest step) in float64: top-k by value then index, top-p over it, the inverse CDF in index order."""
    order = np.lexsort((np.arange(len(row)), -row))[:k]
    q = np.exp((row[order] - row[order[0]]) / t)
    if p >= 0:
        cum = np.cumsum(q / q.sum())
        n = int(np.searchsorted(cum, p)) + 1
        order, q = order[:n], q[:n]
        edge = np.abs(cum - p).min()
    else:
        edge = 1.0
    by_index = np.argsort(order)
    cum = np.cumsum(q[by_index]) / q.sum()
    at = min(int(np.searchsorted(cum, u)), len(cum) - 1)
    return int(order[by_index][at]), min(edge, float(np.abs(cum - u).min()))


@pytest.mark.parametrize("V", [300, 16383, 16384, 16387, 151936])
@pytest.mark.parametrize("k", [1, 2, 20, 255, 256])
@pytest.mark.parametrize("peak", [0.0, 60.0])
def test_top_k_of_long_and_short_rows(V, k, peak):
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    g = torch.Generator(device=dev).manual_seed(V + k)
    R = 6
    logits = torch.randn(R, V, device=dev, generator=g) * 3
    logits[:, V // 3] += peak
    logits[1, ::7] = -float("inf")
    logits[2, 5] = float("nan")
    logits[3] = (logits[3] * 2).round() / 2                  # many ties
    logits[4, 10:] = -float("inf")
    logits[5] = -float("inf")                                # no choice at all: any id of the row
    rng = np.random.default_rng(V + k)
    top_p = torch.tensor([-1.0, 0.8, 0.95, -1.0, 0.5, 0.99], device=dev)
    for _ in range(3):
        u = rng.random(R)
        got = ops.sample_rows(logits, torch.full((R,), 0.7, device=dev), torch.tensor(u, device=dev),
                              torch.full((R,), k, dtype=torch.int32, device=dev), top_p).tolist()
        assert 0 <= got[5] < V
        for i, row in enumerate(logits[:5].double().cpu().numpy()):
            row = np.where(np.isnan(row), -np.inf, row)
            want, far = _choose(row, float(np.float32(0.7)), k, float(top_p[i]), u[i])
            assert got[i] == want or far < 1e-6, (i, got[i], want, far)


@pytest.mark.parametrize("V", [1, 5, 16383, 16384, 16390, 151936])
def test_greedy_of_long_and_short_rows(V):
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    g = torch.Generator(device=dev).manual_seed(V)
    logits = torch.randn(9, V, device=dev, generator=g).round()          # the first of many equal maxima
    logits[1] = -float("inf")
    logits[2] = float("nan")
    logits[3, V - 1] = 50
    logits[4, 0] = 50
    clean = torch.nan_to_num(logits, nan=-float("inf"), neginf=-float("inf"), posinf=float("inf"))
    want = [int((row == row.max()).nonzero()[0]) for row in clean]
    assert ops.sample_rows(logits).tolist() == want


@pytest.mark.parametrize("V", [49151, 49152, 65537, 151936])
@pytest.mark.parametrize("R", [1, 14, 15, 16, 33, 34, 74, 75, 149])
def test_few_rows_are_shared_by_blocks_and_many_are_not(V, R):
    """All of a launch's blocks fit the GPU at once wherever a row has several (a block fills an SM), and a row's choice is the same however many blocks it
    has: greedy, temperature alone, top-k with and without top-p, a top-k beyond the short form, top-p alone."""
    import sllm_b200.ops as ops
    dev = cuda_or_skip()
    blocks = ops.lib().sllm_sample_rows_blocks(R, V)
    assert blocks in (1, 2, 4, 8) and (blocks == 1 or (R * blocks <= ops.num_sms() and V >= 49152))
    g = torch.Generator(device=dev).manual_seed(V + R)
    logits = torch.randn(R, V, device=dev, generator=g) * 3
    i = torch.arange(R, device=dev) % 6
    t = torch.where(i == 0, 0.0, 0.7)
    k = torch.tensor([0, 0, 20, 200, 700, 0], dtype=torch.int32, device=dev)[i]
    p = torch.tensor([-1.0, -1.0, 0.8, -1.0, 0.9, 0.95], device=dev)[i]
    u = torch.rand(R, device=dev, generator=g, dtype=torch.float64)
    got = ops.sample_rows(logits, t, u, k, p)
    few = range(0, R, max(1, R // 12))
    alone = [int(ops.sample_rows(logits[r:r + 1], t[r:r + 1], u[r:r + 1], k[r:r + 1], p[r:r + 1])) for r in few]
    assert [int(got[r]) for r in few] == alone


def test_blocks_a_row_asked_before_the_first_launch():
    """The answer is kept for the process, so it must not depend on whether a row has been sampled yet."""
    import subprocess
    import sys
    cuda_or_skip()
    code = "import torch, sllm_b200.ops as ops; torch.zeros(1, device='cuda'); print(ops.lib().sllm_sample_rows_blocks(1, 151936))"
    done = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300, cwd=ROOT)
    assert done.returncode == 0, done.stderr
    assert int(done.stdout.split()[-1]) == 8
