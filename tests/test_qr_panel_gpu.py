"""DecomposeQRT around the sizes where the panel changes its number of CTAs, its rows per thread and
its kernel (256 rows per CTA and thread row, 16 CTAs, 8192 rows) and at ragged widths: A = Q R
with Q = I - Y T Y^T, Q orthogonal, and R's sign convention of LAPACK, within the bound of the
factorization's parity tests, 8 max(m, n) eps ||A||."""
import numpy as np
import pytest

from util import EPS, fro

pytestmark = pytest.mark.gpu


def _check(gpu, A0):
    m, n = A0.shape
    k = min(m, n)
    A, T = gpu.to_device(A0), gpu.matrix(k, k, fill=0.0)
    assert gpu.DecomposeQRT(A, T, None, 0)[1] is None
    out, T = A.cpu().numpy(), T.cpu().numpy()
    Y = np.tril(out[:, :k], -1) + np.eye(m, k)
    R = np.vstack([np.triu(out[:k]), np.zeros((m - k, n))])
    QR = R - Y @ (T @ (Y.T @ R))
    bound = 8 * max(m, n) * EPS
    assert fro(QR - A0) <= bound * fro(A0)
    # Q^T Q = I: T^-1 + T^-T = Y^T Y on the nonzero tau, checked as T^T (Y^T Y) T = T + T^T
    assert fro(T.T @ (Y.T @ Y) @ T - T - T.T) <= bound * np.sqrt(k) * max(1.0, fro(T))
    return out, T


@pytest.mark.parametrize("m,n", [(1, 1), (2, 2), (5, 40), (31, 33), (32, 32), (33, 31), (64, 100), (255, 32),
                                 (256, 31), (257, 65), (512, 33), (513, 130), (1025, 40), (4096, 32),
                                 (4097, 33), (8192, 20), (8193, 34)])
def test_panel_shapes(gpu, rng, m, n):
    _check(gpu, rng.uniform(-1, 1, (m, n)))


def test_zero_columns_and_scaling(gpu, rng):
    A = rng.uniform(-1, 1, (300, 50))
    A[:, 7] = 0.0           # tau = 0: T's column is zero
    A[1:, 0] = 0.0          # nothing below the diagonal at once
    out, T = _check(gpu, A)
    assert T[0, 0] == 0.0 and out[0, 0] == A[0, 0]
    _check(gpu, rng.uniform(-1, 1, (700, 40)) * 1e150)


def test_nan_stays_right_of_finished_columns(gpu, rng):
    A = rng.uniform(-1, 1, (600, 40))
    clean, _ = _check(gpu, A)
    B = A.copy()
    B[400, 20] = np.nan
    D, T = gpu.to_device(B), gpu.matrix(40, 40, fill=0.0)
    assert gpu.DecomposeQRT(D, T, None, 0)[1] is None
    out = D.cpu().numpy()
    # the first 20 columns are factored before the NaN's column is reached
    assert np.array_equal(out[:, :20], clean[:, :20])
    assert np.isnan(out[20:, 20]).any()
