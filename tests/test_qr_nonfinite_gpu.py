"""DecomposeQRT of a matrix with a NaN or an infinity: the columns of A left of it, and of the block
reflectors of T, are the ones of the clean matrix (bound: 8 max(m, n) eps, the factorization's
own), and a last column without rows below its diagonal has tau = 0, a zero column of T."""
import numpy as np
import pytest

from util import EPS, fro

pytestmark = pytest.mark.gpu


def _run(gpu, A0):
    m, n = A0.shape
    k = min(m, n)
    A, T = gpu.to_device(A0), gpu.matrix(k, k, fill=0.0)
    assert gpu.DecomposeQRT(A, T, None, 0)[1] is None
    return A.cpu().numpy(), T.cpu().numpy()


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("m,n,q", [(300, 60, 50), (600, 200, 100), (600, 200, 190), (3000, 100, 50),
                                   (700, 128, 127)])
def test_columns_left_of_it(gpu, rng, bad, m, n, q):
    A = rng.uniform(-1, 1, (m, n))
    clean, T = _run(gpu, A)
    A[m // 2, q] = bad
    out, Tb = _run(gpu, A)
    bound = 8 * max(m, n) * EPS
    assert fro(out[:, :q] - clean[:, :q]) <= bound * fro(clean)
    # (T's rows above the 128-column block of column q come from products over that whole block,
    # with the NaN in them: there only the columns of the blocks before it are clean)
    kb = q // 128 * 128
    assert fro(Tb[:, :kb] - T[:, :kb]) <= bound * fro(T)
    assert fro(Tb[kb:, kb:q] - T[kb:, kb:q]) <= bound * fro(T)
    assert not np.isfinite(Tb[:q + 1, q]).all()


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("m,n", [(5, 5), (30, 60), (256, 256)])
def test_last_column_of_a_square_block(gpu, rng, bad, m, n):
    A = rng.uniform(-1, 1, (m, n))
    A[m // 2, m // 4] = bad
    _, T = _run(gpu, A)
    if m <= 32:                      # one panel: T's last column is tau = 0's
        assert not T[:, m - 1].any()
    assert T[m - 1, m - 1] == 0.0
