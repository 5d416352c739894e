"""The 128 x 128 diagonal block (factor and inverse by 16 x 16 sub-blocks) at the sizes where its
sub-blocks, padding and neighbours change: DecomposeCHOL against ||A - L L^T|| <= 10 n eps ||A||,
its failing column, and SolveTrm, which uses the block inverses, against 100 n eps relative."""
import numpy as np
import pytest

from util import EPS, fro, spd

pytestmark = pytest.mark.gpu

LO, UP, LEFT, TA, UNIT = 0x4, 0x8, 0x10, 0x1, 0x40
SIZES = [1, 2, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 65, 80, 111, 112, 113, 127, 128, 129, 144, 255, 257]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("flags", [LO, UP])
def test_factor(gpu, rng, n, flags):
    A = spd(rng, n)
    D = gpu.to_device(A)
    assert gpu.DecomposeCHOL(D, flags, 0)[1] is None
    out = D.cpu().numpy()
    L = np.tril(out) if flags == LO else np.triu(out).T
    assert fro(A - L @ L.T) <= 10 * n * EPS * fro(A)
    other = np.triu(out, 1) - np.triu(A, 1) if flags == LO else np.tril(out, -1) - np.tril(A, -1)
    assert not other.any()


@pytest.mark.parametrize("n,at", [(1, 0), (16, 15), (40, 16), (128, 0), (128, 77), (128, 127), (200, 128),
                                  (300, 290)])
def test_failing_column(gpu, n, at):
    A = np.eye(n)
    A[at, at] = -2.0
    with pytest.raises(gpu.MatopsPanic, match=f"illegal value at {at}: -2.0"):
        gpu.DecomposeCHOL(gpu.to_device(A), LO, 0)


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("flags", [LO, UP, LO | TA, UP | TA, LO | UNIT, UP | TA | UNIT])
def test_block_inverse(gpu, rng, n, flags):
    T = rng.uniform(-1, 1, (n, n)) / max(n, 1) + 2.0 * np.eye(n)
    M = np.tril(T) if flags & LO else np.triu(T)
    if flags & UNIT:
        np.fill_diagonal(M, 1.0)
    B = rng.uniform(-1, 1, (n, 70))  # more than 64 columns: the sweep with block inverses
    Bd = gpu.to_device(B)
    assert gpu.SolveTrm(Bd, gpu.to_device(T), 1.0, LEFT | flags) is None
    ref = np.linalg.solve(M.T if flags & TA else M, B)
    assert fro(Bd.cpu().numpy() - ref) <= 100 * n * EPS * fro(ref)
