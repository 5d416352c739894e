"""DecomposeLU around the sizes where the panel changes its number of CTAs, its rows per thread
and its kernel (256 rows per CTA and thread row, 16 CTAs, 16384 rows), against the oracle:
pivots identical, ||A - A_ref|| <= 10 n eps ||A|| (the bound of the factorization's parity
tests), and the rules for zeros, ties and NaN of the pivot search (pivot.go:98-107)."""
import numpy as np
import pytest

from util import EPS, colmajor, fro

pytestmark = pytest.mark.gpu


def _run(gpu, oracle, A, nb=0):
    import torch
    Ad = gpu.to_device(A)
    k = min(A.shape)
    piv = torch.full((k,), -7, dtype=torch.int64, device="cuda")
    assert gpu.DecomposeLU(Ad, piv, nb)[1] is None
    Ar, pr = colmajor(A, A.shape[0] + A.shape[0] % 2), np.zeros(k, dtype=np.int64)
    assert oracle.DecomposeLU(Ar, pr, nb) == 0
    return Ad.cpu().numpy(), piv.cpu().numpy(), Ar, pr


@pytest.mark.parametrize("m,n", [(16, 16), (17, 15), (33, 20), (128, 128), (129, 200), (255, 144),
                                 (256, 47), (257, 257), (512, 33), (513, 130), (1025, 129),
                                 (2049, 17), (4096, 31), (4097, 140), (8193, 35), (16384, 20),
                                 (16385, 18)])
def test_panel_shapes(gpu, oracle, rng, m, n):
    A = rng.standard_normal((m, n))
    X, p, Xr, pr = _run(gpu, oracle, A)
    assert np.array_equal(p, pr)
    assert fro(X - Xr) <= 10 * max(m, n) * EPS * fro(A)


@pytest.mark.parametrize("m", [60, 300, 700])
def test_pivot_rules(gpu, oracle, rng, m):
    n = 40
    A = rng.integers(-2, 3, (m, n)).astype(float)  # many ties: the first row wins
    A[:, 5] = A[:, 3]                              # a column that becomes zero
    X, p, Xr, pr = _run(gpu, oracle, A)
    # past the zero pivot the columns hold infinities and NaN, and what the later pivots
    # do to the order of the rows is not defined: the first five rows are final by then
    assert np.array_equal(p[:5], pr[:5])
    assert fro(X[:5] - Xr[:5]) <= 10 * m * EPS * fro(A)
    # a NaN below the diagonal never wins, one on the diagonal stays; columns left of it agree
    B = rng.standard_normal((m, n))
    B[m - 1, 0] = np.nan
    X, p, Xr, pr = _run(gpu, oracle, B)
    assert p[0] == pr[0] and p[0] != m - 1
    B = rng.standard_normal((m, n))
    B[0, 0] = np.nan
    X, p, Xr, pr = _run(gpu, oracle, B)
    assert p[0] == pr[0] == 0
