"""Mult and RankUpdateSym on both sides of the rules that pick a product's kernel: a few 32 x 32 tiles
of C with a very long K (split along K up to 2^31 multiply-adds for at most 16 tiles, 2^29
otherwise), and many tiles with a short K and A transposed (with B not, the engine past 1500 tiles
and one slab of 16), against numpy.  Bound: 4 k eps (|alpha| ||A|| ||B|| + |beta| ||C||), as in the
other tests of Mult."""
import numpy as np
import pytest

from util import colmajor, fro, gemm_bound

pytestmark = pytest.mark.gpu

TA, TB, LO = 0x1, 0x2, 0x4


def _mult(gpu, rng, m, n, k, flags, odd):
    import torch
    A = rng.uniform(-1, 1, (k, m) if flags & TA else (m, k))
    B = rng.uniform(-1, 1, (n, k) if flags & TB else (k, n))
    C = rng.uniform(-1, 1, (m, n))

    def dev(a):
        t = gpu.matrix(a.shape[0] + odd, a.shape[1])[:a.shape[0]]
        t.copy_(torch.from_numpy(a))
        return t
    Cd = dev(C)
    assert gpu.Mult(Cd, dev(A), dev(B), -1.0, 0.5, flags) is None
    ref = 0.5 * C - (A.T if flags & TA else A) @ (B.T if flags & TB else B)
    assert fro(Cd.cpu().numpy() - ref) <= gemm_bound(k, 1.0, 0.5, A, B, C)


@pytest.mark.parametrize("odd", [0, 1])
@pytest.mark.parametrize("flags", [0, TA, TB])
@pytest.mark.parametrize("m,n,k", [(128, 128, 40001), (100, 97, 70000), (1, 64, 200000),
                                   (129, 128, 40001), (64, 64, 600000)])
def test_few_tiles_long_k(gpu, rng, m, n, k, flags, odd):
    _mult(gpu, rng, m, n, k, flags, odd)


@pytest.mark.parametrize("odd", [0, 1])
@pytest.mark.parametrize("m,n", [(1216, 1216), (1249, 1217), (48000, 31), (31, 48100)])
@pytest.mark.parametrize("k", [16, 17, 47])
def test_transposed_short_k(gpu, rng, m, n, k, odd):
    for flags in (TA, TA | TB):
        _mult(gpu, rng, m, n, k, flags, odd)


@pytest.mark.parametrize("n", [1700, 1800])
@pytest.mark.parametrize("k", [16, 33])
def test_transposed_rank_update(gpu, rng, n, k):
    A, C = rng.uniform(-1, 1, (k, n)), rng.uniform(-1, 1, (n, n))
    Cd = gpu.to_device(colmajor(C))
    assert gpu.RankUpdateSym(Cd, gpu.to_device(A), 1.0, 1.0, LO | TA) is None
    ref = np.tril(C + A.T @ A) + np.triu(C, 1)
    assert fro(Cd.cpu().numpy() - ref) <= gemm_bound(k, 1.0, 1.0, A, A, C)
