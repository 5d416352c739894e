"""Batched LU of a matrix with an infinity or a NaN right of a 64-column block: in its column the rows
of U above it, and in the block's rows every other column, are the clean matrix's.  The
matrices are diagonally dominant, so that rows stay in place; the bound, 100 n eps, allows for
another order of the sums."""
import numpy as np
import pytest
import torch

from util import EPS, fro

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [np.inf, np.nan])
@pytest.mark.parametrize("n,r,c", [(65, 20, 64), (100, 31, 90), (100, 40, 70), (200, 63, 64),
                                   (200, 1, 199), (300, 33, 257)])
def test_batched_lu_rows_above(gpu, rng, bad, n, r, c):
    A = rng.uniform(-1, 1, (n, n)) + n * np.eye(n)
    B = A.copy()
    B[r, c] = bad
    a = [gpu.to_device(A), gpu.to_device(B)]
    piv = [torch.zeros(n, dtype=torch.int64, device="cuda") for _ in a]
    gpu.BatchPlan(gpu.BATCH_LU, [n, n]).run(a, None, piv)
    clean, out = (x.cpu().numpy() for x in a)
    assert piv[1][:64].tolist() == list(range(64))
    assert not np.isfinite(out[r, c])
    keep = np.ones((64, n), bool)
    keep[r:, c] = False
    assert np.isfinite(out[:64][keep]).all()
    assert fro((out[:64] - clean[:64])[keep]) <= 100 * n * EPS * fro(clean)


def test_batched_lu_spoilt_row_at_the_end_of_a_block(gpu, rng):
    # two rows become NaN as a whole and are interchanged to the end: row 63, the last of the
    # first block, is one of them, and the rows above it stay clean
    n = 65
    A = rng.uniform(-1, 1, (n, n)) + n * np.eye(n)
    A[10, 3] = A[43, 21] = np.nan
    a, piv = [gpu.to_device(A)], [torch.zeros(n, dtype=torch.int64, device="cuda")]
    gpu.BatchPlan(gpu.BATCH_LU, [n]).run(a, None, piv)
    out = a[0].cpu().numpy()
    assert np.isfinite(out[:63]).all() and not np.isfinite(out[63, 64])


@pytest.mark.parametrize("n", [16, 32, 48, 64, 128])
def test_batched_cholesky_zero_last_pivot(gpu, n):
    # semidefinite, the zero in the last column: the root of zero is zero, as in the reference
    # (only a pivot whose root is NaN is refused, chol.go:33-36)
    A = np.diag(np.arange(1.0, n + 1))
    A[n - 1, n - 1] = 0.0
    a = [gpu.to_device(A)]
    assert gpu.BatchPlan(gpu.BATCH_CHOL, [n]).run(a).tolist() == [0]
    out = a[0].cpu().numpy()
    assert fro(out - np.sqrt(A)) <= n * EPS * fro(A) and out[n - 1, n - 1] == 0.0
