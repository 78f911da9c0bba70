"""The coarse space's blocked inverse where its register-held pivot blocks can
go wrong: one pivot, a full and a ragged last block, rows that have to change
places inside a block at every step, and equal pivot candidates.

Tolerance: |A X - I| <= 1e-12 for matrices of condition below 1e3 (n eps
times the condition, n <= 129).
"""
import numpy as np
import pytest

from tests.meshes import make_ctx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [129, 1, 2, 32, 64, 65, 95])
@pytest.mark.parametrize("kind", ["swaps", "ties"])
def test_pivot_blocks(n, kind):
    import torch
    ctx = make_ctx("amr2_free", device=0)
    rng = np.random.default_rng(n)
    A = 0.01 * rng.standard_normal((n, n))
    for k in range(0, n, 32):  # a permutation inside each pivot block: no diagonal entry is the pivot
        m = min(32, n - k)
        p = np.roll(np.arange(m), 1)
        A[k + p, k + np.arange(m)] += 1.0 + (0.0 if kind == "ties" else 1.0) * rng.random(m)
    if kind == "ties":  # equal magnitudes in the pivot columns
        A = np.round(A)
    a = torch.tensor(A, device="cuda")
    assert not ctx.dense_inverse(a)
    assert np.linalg.cond(A) < 1e3
    assert np.abs(A @ a.cpu().numpy() - np.eye(n)).max() <= 1e-12
