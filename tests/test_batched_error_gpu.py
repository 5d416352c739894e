"""The error of the batched Cholesky factor is no larger than that of a right-looking factorization by
32 columns in FP64 (numpy and scipy), both against the factor in extended precision, on
diagonally dominant matrices and at a condition of 1e6: the ratio of the errors, geometric
mean over the matrices.  It is about 0.75 and 0.95; a C that is rounded by every product gives 1.5
and 1.5 to 1.9.  The scatter of the mean is 0.02 and 0.1, so the bound is 1.2."""
import numpy as np
import pytest
from scipy.linalg import solve_triangular

from util import colmajor

pytestmark = pytest.mark.gpu


def _extended(A):
    L = np.tril(A).astype(np.longdouble)
    for k in range(L.shape[0]):
        L[k, k] = np.sqrt(L[k, k])
        L[k + 1:, k] /= L[k, k]
        L[k + 1:, k + 1:] -= np.tril(np.outer(L[k + 1:, k], L[k + 1:, k]))
    return L


def _right_looking(A, nb=32):
    L = A.copy()
    for j in range(0, A.shape[0], nb):
        e = j + nb
        L[j:e, j:e] = np.linalg.cholesky(L[j:e, j:e])
        L[e:, j:e] = solve_triangular(L[j:e, j:e], L[e:, j:e].T, lower=True).T
        L[e:, e:] -= L[e:, j:e] @ L[e:, j:e].T
    return np.tril(L)


@pytest.mark.parametrize("cond", [None, 1e6])
@pytest.mark.parametrize("n,count", [(256, 10), (400, 6)])
def test_error_of_batched_cholesky(gpu, rng, n, count, cond):
    mats = []
    for _ in range(count):
        G = rng.standard_normal((n, n))
        if cond is None:
            A = G @ G.T / n + np.eye(n)
        else:
            Q = np.linalg.qr(G)[0]
            A = (Q * np.geomspace(1.0, 1.0 / cond, n)) @ Q.T
        mats.append(np.tril(A) + np.tril(A, -1).T)
    dev = [gpu.to_device(colmajor(A)) for A in mats]
    assert gpu.BatchPlan(gpu.BATCH_CHOL, [n] * count).run(dev).tolist() == [0] * count
    ratio = []
    for A, d in zip(mats, dev):
        ref = _extended(A)
        here = np.linalg.norm((np.tril(d.cpu().numpy()) - ref).astype(float))
        ratio.append(here / np.linalg.norm((_right_looking(A) - ref).astype(float)))
    assert np.exp(np.mean(np.log(ratio))) <= 1.2, ratio
