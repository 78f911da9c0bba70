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


def _hadamard(m):
    """+-1 entries, orthogonal columns: powers of two along the diagonal."""
    H = np.zeros((m, m))
    at = 0
    while at < m:
        k = 1 << (int(m - at).bit_length() - 1)
        h = np.ones((1, 1))
        while len(h) < k:
            h = np.block([[h, h], [h, -h]])
        H[at:at + k, at:at + k] = h
        at += k
    return H


def _tied_pivots(A):
    """Pivot columns of Gaussian elimination with partial pivoting whose
    largest entry occurs more than once."""
    A = A.copy()
    ties = 0
    for j in range(len(A)):
        c = np.abs(A[j:, j])
        ties += np.sum(c == c.max()) > 1
        p = j + int(np.argmax(c))
        A[[j, p]] = A[[p, j]]
        A[j + 1:] -= np.outer(A[j + 1:, j] / A[j, j], A[j])
    return ties


@pytest.mark.parametrize("n", [129, 1, 2, 32, 64, 65, 95])
@pytest.mark.parametrize("kind", ["swaps", "ties"])
def test_pivot_blocks(n, kind):
    import torch
    ctx = make_ctx("amr2_free", device=0)
    rng = np.random.default_rng(n)
    A = 0.01 * rng.standard_normal((n, n))
    for k in range(0, n, 32):
        m = min(32, n - k)
        if kind == "swaps":  # a permutation inside each pivot block: no diagonal entry is the pivot
            p = np.roll(np.arange(m), 1)
            A[k + p, k + np.arange(m)] += 1.0 + rng.random(m)
        else:  # equal candidates in most pivot columns of a block, rows in any order
            # (nothing below the block, whose update would part them)
            A[k:k + m, k:k + m] = _hadamard(m)[rng.permutation(m)]
            A[k + m:, k:k + m] = 0.0
            assert _tied_pivots(A[k:k + m, k:k + m]) >= m // 2
    a = torch.tensor(A, device="cuda")
    assert not ctx.dense_inverse(a)
    assert np.linalg.cond(A) < 1e3
    assert np.abs(A @ a.cpu().numpy() - np.eye(n)).max() <= 1e-12
