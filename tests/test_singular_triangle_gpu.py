"""A zero on the diagonal of a triangle spoils the unknowns from its row on (in the order of the
substitution) and no others: those before it equal the ones of the regular system.  The same
for an off-diagonal infinity, and for the rows of an inverse above a zero pivot.

Bound of the finite part: the regular system's solution from the same kernels differs by rounding
only, and the triangle's condition number is below 10 in every case, so 100 n eps."""
import numpy as np
import pytest

from util import EPS, fro

pytestmark = pytest.mark.gpu

LO, UP, TA, LEFT, RIGHT = 0x4, 0x8, 0x1, 0x10, 0x20


def _tri(rng, n):
    a = np.tril(rng.uniform(-0.5, 0.5, (n, n)) / np.sqrt(n), -1)
    return a + np.diag(rng.uniform(1.0, 2.0, n))


@pytest.mark.parametrize("n", [5, 16, 20, 64, 100, 128])
@pytest.mark.parametrize("nrhs", [1, 70])
@pytest.mark.parametrize("side", [LEFT, RIGHT])
@pytest.mark.parametrize("upper", [False, True])
def test_backward_solve_before_a_zero_pivot(gpu, rng, n, nrhs, side, upper):
    # op(A) is upper triangular from the left (lower from the right): the last unknowns first
    for p in sorted({0, n // 3, n - 2}):
        L = _tri(rng, n)
        B = rng.uniform(-1, 1, (n, nrhs))
        X = np.linalg.solve(L.T, B)
        L[p, p] = 0.0
        flags = UP if upper else LO | TA
        A = L.T if upper else L
        if side == RIGHT:
            flags, A = (UP | TA, L.T) if upper else (LO, L)
        Bg = gpu.to_device(B if side == LEFT else B.T)
        assert gpu.SolveTrm(Bg, gpu.to_device(A), 1.0, flags | side) is None
        out = Bg.cpu().numpy() if side == LEFT else Bg.cpu().numpy().T
        assert not np.isfinite(out[p]).any()
        assert fro(out[p + 1:] - X[p + 1:]) <= 100 * n * EPS * fro(X)


@pytest.mark.parametrize("n", [5, 33, 130])
def test_inverse_with_a_zero_pivot(gpu, rng, n):
    p = n // 2
    L = _tri(rng, n)
    X = np.linalg.inv(L)
    L[p, p] = 0.0
    A = gpu.to_device(L)
    assert gpu.InverseTrm(A, LO, 0)[1] is None
    out = np.tril(A.cpu().numpy())
    ok = np.tril(np.ones((n, n), bool))
    ok[p:, :p + 1] = False   # everything that passes through the pivot
    assert np.isfinite(out[ok]).all() and fro((out - X)[ok]) <= 100 * n * EPS * fro(X)
    assert not np.isfinite(out[p, p])


@pytest.mark.parametrize("n", [20, 32])
def test_infinite_entry(gpu, rng, n):
    # L(r, q) infinite: L^T x = b gives the unknowns after q by the other equations
    r, q = 13, 6
    L = _tri(rng, n)
    B = rng.uniform(-1, 1, (n, 2))
    X = np.linalg.solve(L.T, B)
    L[r, q] = np.inf
    Bg = gpu.to_device(B)
    assert gpu.SolveTrm(Bg, gpu.to_device(L), 1.0, LO | TA | LEFT) is None
    out = Bg.cpu().numpy()
    assert fro(out[r + 1:] - X[r + 1:]) <= 100 * n * EPS * fro(X)
    assert not np.isfinite(out[q]).any()
