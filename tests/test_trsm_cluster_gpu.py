"""SolveTrm with few right-hand sides: up to order 2048 one thread-block cluster per 4 of them
(128 rows per CTA), above by blocks of 512, 1024 or 2048; at the edges of the blocks and cluster
sizes, all sides, triangles and transpositions, with odd leading dimensions; bound 100 n eps
relative, as in the parity tests of SolveTrm."""
import numpy as np
import pytest

from util import EPS, fro

pytestmark = pytest.mark.gpu

TA, LO, UP, LEFT, RIGHT, UNIT = 0x1, 0x4, 0x8, 0x10, 0x20, 0x40


def _solve(gpu, rng, n, nrhs, flags, pad=0, alpha=1.0):
    T = rng.uniform(-1, 1, (n, n)) / n + 2.0 * np.eye(n)
    M = np.tril(T) if flags & LO else np.triu(T)
    if flags & UNIT:
        np.fill_diagonal(M, 1.0)
    op = M.T if flags & TA else M
    B = rng.uniform(-1, 1, (nrhs, n) if flags & RIGHT else (n, nrhs))
    Ad, Bd = gpu.matrix(n + pad, n, fill=9.0)[:n], gpu.matrix(B.shape[0] + pad, B.shape[1], fill=9.0)
    import torch
    Ad.copy_(torch.from_numpy(T))
    Bv = Bd[: B.shape[0]]
    Bv.copy_(torch.from_numpy(B))
    assert gpu.SolveTrm(Bv, Ad, alpha, flags) is None
    assert gpu.Sync() == 0
    ref = alpha * (np.linalg.solve(op.T, B.T).T if flags & RIGHT else np.linalg.solve(op, B))
    assert fro(Bv.cpu().numpy() - ref) <= 100 * n * EPS * fro(ref)
    assert bool((Bd[B.shape[0]:] == 9.0).all())


@pytest.mark.parametrize("n", [129, 255, 256, 257, 511, 600, 1025, 2047, 2048, 2049])
@pytest.mark.parametrize("flags", [LO, UP, LO | TA, UP | TA])
@pytest.mark.parametrize("nrhs", [1, 3])
def test_sizes(gpu, rng, n, flags, nrhs):
    _solve(gpu, rng, n, nrhs, LEFT | flags, pad=1 + (n & 1))


@pytest.mark.parametrize("nrhs", [1, 2, 4, 5, 16, 31, 64])
@pytest.mark.parametrize("side", [LEFT, RIGHT])
@pytest.mark.parametrize("flags", [LO | UNIT, UP | TA])
def test_right_hand_sides(gpu, rng, nrhs, side, flags):
    _solve(gpu, rng, 300, nrhs, side | flags, alpha=-1.5)
    _solve(gpu, rng, 1300, nrhs, side | flags)


@pytest.mark.parametrize("n", [128, 129, 700, 2049])
@pytest.mark.parametrize("flags", [LO, UP])
@pytest.mark.parametrize("nrhs", [1, 5, 65])
def test_cholesky_sweeps_are_the_two_solves(gpu, rng, n, flags, nrhs):
    # SolveCHOL forms the block inverses once for both sweeps: the same operations, bit for bit
    A = gpu.matrix(n, n)
    import torch
    A.copy_(torch.from_numpy(rng.uniform(-1, 1, (n, n)) / n + 2.0 * np.eye(n)))
    B, C = gpu.matrix(n, nrhs), gpu.matrix(n, nrhs)
    B.copy_(torch.from_numpy(rng.uniform(-1, 1, (n, nrhs))))
    C.copy_(B)
    gpu.SolveCHOL(B, A, flags)
    for f in ((flags, flags | TA) if flags == LO else (flags | TA, flags)):
        assert gpu.SolveTrm(C, A, 1.0, LEFT | f) is None
    assert gpu.Sync() == 0
    assert torch.equal(B, C)


@pytest.mark.parametrize("n,nrhs", [(1025, 17), (2048, 64), (2177, 33), (4097, 1), (4200, 20),
                                    (513, 49)])
@pytest.mark.parametrize("side", [LEFT, RIGHT])
@pytest.mark.parametrize("flags", [LO, UP | UNIT, LO | TA, UP | TA])
def test_blocks(gpu, rng, n, nrhs, side, flags):
    # cluster-sized diagonal blocks with a product for the rest of B between them
    _solve(gpu, rng, n, nrhs, side | flags, pad=n & 1, alpha=0.75)
