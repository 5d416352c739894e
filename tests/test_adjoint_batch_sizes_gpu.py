"""DecomposeCHOLAdjointBatched on both sides of the rule that picks its kernel (the largest order up
to 96; up to 320 with at most one matrix per SM), with odd orders and smaller matrices beside:
the closed form sym(L^-T Phi(L^T Lbar) L^-1), within the 1e-10 of the adjoint's other tests."""
import numpy as np
import pytest
import torch

from util import fro

pytestmark = pytest.mark.gpu

LO = 0x4


@pytest.mark.parametrize("n", [1, 31, 96, 97, 320, 321])
@pytest.mark.parametrize("many", [False, True])
def test_closed_form(gpu, rng, n, many):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    sizes = [n] * (sms if many else 2) + [max(1, n // 3)]
    Ls, Gs, refs = [], [], []
    for k, m in enumerate(sizes):
        if 3 < k < len(sizes) - 3:   # a few different matrices are enough
            A0, Lbar = refs[k % 4][1:3]
        else:
            g = rng.standard_normal((m, m))
            A0, Lbar = g @ g.T / m + np.eye(m), np.tril(rng.standard_normal((m, m)))
        L = np.linalg.cholesky(A0)
        Li = np.linalg.inv(L)
        P = np.tril(L.T @ Lbar)
        P[np.diag_indices(m)] *= 0.5
        S = Li.T @ P @ Li
        refs.append((0.5 * (S + S.T), A0, Lbar))
        Ls.append(gpu.to_device(np.tril(L) + np.triu(A0, 1)))
        Gs.append(gpu.to_device(Lbar + np.triu(np.full((m, m), 7.0), 1)))
    assert gpu.DecomposeCHOLAdjointBatched(Ls, Gs, LO) is None
    for G, (ref, _, _) in zip(Gs, refs):
        out = G.cpu().numpy()
        assert fro(out - ref) <= 1e-10 * fro(ref) and np.array_equal(out, out.T)
