"""Mult's tile edges: the engine's 128 x 64 and 64 x 128 tiles with operands by TMA (even leading
dimensions) and by cp.async (odd ones), the 32 x 32 tiles and strips of products up to 2^27
multiply-adds, k-slabs of 16, and in-place products, against numpy.
Bound: 4 k eps (|alpha| ||A|| ||B|| + |beta| ||C||), as in the parity tests of Mult."""
import numpy as np
import pytest

from util import fro, gemm_bound

pytestmark = pytest.mark.gpu

TA, TB, LO, UP = 0x1, 0x2, 0x4, 0x8


def _dev(gpu, a, ld):
    import torch
    t = gpu.matrix(ld, a.shape[1], fill=7.0)
    t[: a.shape[0]].copy_(torch.from_numpy(a))
    return t[: a.shape[0]], t


@pytest.mark.parametrize("odd", [0, 1])
@pytest.mark.parametrize("flags", [0, TA, TB, TA | TB])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (63, 129, 15), (64, 65, 16), (65, 64, 17), (64, 128, 33),
                                   (127, 63, 31), (128, 64, 48), (129, 65, 64), (257, 191, 79),
                                   (33, 400, 130), (31, 33, 4096), (32, 65, 4097),
                                   (2300, 456, 129), (640, 1088, 208), (2049, 65, 1040),
                                   (2560, 2432, 40)])
def test_tile_edges(gpu, rng, m, n, k, flags, odd):
    A = rng.uniform(-1, 1, (k, m) if flags & TA else (m, k))
    B = rng.uniform(-1, 1, (n, k) if flags & TB else (k, n))
    C = rng.uniform(-1, 1, (m, n))

    def ld(r):  # an odd or an even leading dimension, larger than the view
        return r + 1 + ((r + 1 + odd) & 1)
    (Ad, _), (Bd, _), (Cd, Cbuf) = _dev(gpu, A, ld(A.shape[0])), _dev(gpu, B, ld(B.shape[0])), \
        _dev(gpu, C, ld(m))
    assert gpu.Mult(Cd, Ad, Bd, 1.5, -0.5, flags) is None
    ref = 1.5 * (A.T if flags & TA else A) @ (B.T if flags & TB else B) - 0.5 * C
    assert fro(Cd.cpu().numpy() - ref) <= gemm_bound(k, 1.5, -0.5, A, B, C)
    assert bool((Cbuf[m:] == 7.0).all())  # nothing written below the view
    # beta = 0 does not read C
    Cd.fill_(float("nan"))
    assert gpu.Mult(Cd, Ad, Bd, -1.0, 0.0, flags) is None
    ref = -(A.T if flags & TA else A) @ (B.T if flags & TB else B)
    assert fro(Cd.cpu().numpy() - ref) <= gemm_bound(k, 1.0, 0.0, A, B, C)


@pytest.mark.parametrize("flags", [LO, UP, LO | TA, UP | TA])
@pytest.mark.parametrize("n,k", [(1, 1), (64, 16), (65, 33), (129, 40), (193, 17), (700, 64)])
def test_triangle_tiles(gpu, rng, n, k, flags):
    A = rng.uniform(-1, 1, (k, n) if flags & TA else (n, k))
    C = rng.uniform(-1, 1, (n, n))
    Cd, _ = _dev(gpu, C, n)
    # beta = 1: the same with the reference's diagonal-block beta and with BLAS semantics
    assert gpu.RankUpdateSym(Cd, _dev(gpu, A, A.shape[0])[0], -1.0, 1.0, flags) is None
    full = C - (A.T @ A if flags & TA else A @ A.T)
    tri = np.tril if flags & LO else np.triu
    other = np.triu(C, 1) if flags & LO else np.tril(C, -1)
    assert fro(Cd.cpu().numpy() - (tri(full) + other)) <= gemm_bound(k, 1.0, 1.0, A, A, C)


@pytest.mark.parametrize("side", [0x10, 0x20])
@pytest.mark.parametrize("n,nrhs", [(100, 200), (128, 130), (129, 65), (300, 257), (31, 97),
                                    (160, 9001)])
def test_in_place_products(gpu, rng, n, nrhs, side):
    """SolveTrm above 64 right-hand sides multiplies by block inverses in place, from the left
    (C = op(B)) and from the right (C = op(A)); odd orders take the cp.async producer.  Bound:
    100 n eps relative, as in the parity tests of SolveTrm."""
    A = np.tril(rng.uniform(-1, 1, (n, n))) / n + 2.0 * np.eye(n)
    B = rng.uniform(-1, 1, (n, nrhs) if side == 0x10 else (nrhs, n))
    Bd, _ = _dev(gpu, B, B.shape[0])
    assert gpu.SolveTrm(Bd, _dev(gpu, A, n)[0], 1.0, side | LO) is None
    ref = np.linalg.solve(A, B) if side == 0x10 else np.linalg.solve(A.T, B.T).T
    assert fro(Bd.cpu().numpy() - ref) <= 100 * n * np.finfo(float).eps * fro(ref)
