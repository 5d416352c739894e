"""DecomposeQRT gives the same bits every time, at the sizes whose panels run in one CTA (at most
256 rows left) and in a cluster: a warp that ran ahead into the next column and replaced its
sums before the others had read them would change some runs.  The bound is equality: the
panel adds its sums in a fixed order."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(32, 32), (200, 32), (256, 32), (255, 130), (256, 256), (700, 690)])
def test_repeated_factorization_same_bits(gpu, rng, m, n):
    import torch
    A0 = gpu.to_device(rng.uniform(-1, 1, (m, n)))
    first = None
    for _ in range(150):
        A, T = gpu.matrix(m, n), gpu.matrix(n, n, fill=0.0)
        A.copy_(A0)
        assert gpu.DecomposeQRT(A, T, None, 0)[1] is None
        if first is None:
            first = (A, T)
        else:
            assert torch.equal(A, first[0]) and torch.equal(T, first[1])
