"""Unit lower triangles with few right-hand sides: the error of SolveTrm is that of a substitution by
64-row blocks with explicit inverses of the diagonal blocks, not that of larger blocks, whose
inverses grow (a partially pivoted L has entries up to 1).  Both errors are taken against the
substitution in extended precision and averaged (geometric mean) over ten matrices; with
128-row blocks the ratio is 1.3 to 1.45, the scatter of the mean is 5 to 8 %, so the bound is
1.2."""
import numpy as np
import pytest
import torch

from util import colmajor

pytestmark = pytest.mark.gpu

LO, UNIT, LEFT = 0x4, 0x40, 0x10


def _extended(L, B):
    L, X = L.astype(np.longdouble), B.astype(np.longdouble)
    for k in range(L.shape[0]):
        X[k + 1:] -= np.outer(L[k + 1:, k], X[k])
    return X


def _blocked(L, B, nb=64):
    X = B.copy()
    for j in range(0, L.shape[0], nb):
        e = min(j + nb, L.shape[0])
        X[j:e] = np.linalg.inv(L[j:e, j:e]) @ X[j:e]
        X[e:] -= L[e:, j:e] @ X[j:e]
    return X


@pytest.mark.parametrize("n,nrhs", [(500, 1), (1001, 3)])
def test_error_of_unit_lower(gpu, rng, n, nrhs):
    ratio = []
    for _ in range(10):
        LU, _ = torch.linalg.lu_factor(torch.from_numpy(rng.standard_normal((n, n))))
        L = np.tril(LU.numpy(), -1) + np.eye(n)
        B = rng.uniform(-1, 1, (n, nrhs))
        ref = _extended(L, B)
        Bg = gpu.to_device(B)
        assert gpu.SolveTrm(Bg, gpu.to_device(colmajor(L)), 1.0, LO | UNIT | LEFT) is None
        here = np.linalg.norm((Bg.cpu().numpy() - ref).astype(float))
        ratio.append(here / np.linalg.norm((_blocked(L, B) - ref).astype(float)))
    assert np.exp(np.mean(np.log(ratio))) <= 1.2, ratio


@pytest.mark.parametrize("flags", [LO, LO | 0x1, 0x8, 0x8 | 0x1])
@pytest.mark.parametrize("side", [0x10, 0x20])
@pytest.mark.parametrize("n,nrhs", [(129, 1), (191, 2), (193, 5), (300, 64), (2049, 3)])
def test_unit_forms(gpu, rng, n, nrhs, side, flags):
    # every storage and side, and last blocks that end inside their first 64 rows: the residual,
    # within 10 n eps ||A|| ||X|| (entries of 1/sqrt(n): the triangle is well conditioned)
    A = np.triu(rng.uniform(-1, 1, (n, n)) / np.sqrt(n), 1)
    A = (A if flags & 0x8 else A.T) + np.diag(rng.uniform(3, 9, n))  # the diagonal is not read
    T = A - np.diag(np.diag(A)) + np.eye(n)
    op = T.T if flags & 0x1 else T
    B = rng.uniform(-1, 1, (n, nrhs) if side == 0x10 else (nrhs, n))
    Bg = gpu.to_device(B)
    assert gpu.SolveTrm(Bg, gpu.to_device(A), 2.0, flags | side | UNIT) is None
    X = Bg.cpu().numpy()
    R = (op @ X if side == 0x10 else X @ op) - 2.0 * B
    assert np.linalg.norm(R) <= 10 * n * np.finfo(float).eps * np.linalg.norm(T) * np.linalg.norm(X)
