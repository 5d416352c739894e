"""Batched factor + solve at the edges of its tiles, blocks and kernels (16 and 32 columns, 64-row
LU blocks, 128 and 256 threads per matrix) in both configurations, with views whose leading
dimension is odd, and the pivot rules: ties to the lowest row, a NaN never chosen.  Bounds as
in the batched parity tests: residuals 10 n eps, pivots identical to the oracle's."""
import numpy as np
import pytest
import torch

from util import EPS, colmajor, fro

pytestmark = pytest.mark.gpu

SIZES = [1, 3, 8, 15, 16, 17, 31, 32, 33, 48, 63, 64, 65, 80, 95, 96, 97, 127, 128, 129, 160, 191,
         193, 255, 256, 257, 321, 400, 511, 512]


def _views(gpu, mats, pad):
    out = []
    for a in mats:
        n = a.shape[0]
        v = gpu.matrix(n + pad, a.shape[1], fill=7.0)[:n]
        v.copy_(torch.as_tensor(a))
        out.append(v)
    return out


@pytest.mark.parametrize("cfg", [0, 1])
@pytest.mark.parametrize("nrhs,pad", [(1, 0), (2, 1)])
def test_both_configurations(gpu, oracle, rng, cfg, nrhs, pad):
    for kind in (gpu.BATCH_CHOL, gpu.BATCH_LU):
        As, Bs = [], [rng.standard_normal((n, nrhs)) for n in SIZES]
        for n in SIZES:
            G = rng.standard_normal((n, n))
            As.append(G @ G.T / n + np.eye(n) if kind == gpu.BATCH_CHOL else G)
        dA, dB = _views(gpu, As, pad), _views(gpu, Bs, pad)
        pivs = [torch.zeros(n, dtype=torch.int64, device="cuda") for n in SIZES]
        plan = gpu.BatchPlan(kind, SIZES, nrhs)
        plan.schedule([cfg] * 4)
        info = plan.run(dA, dB, pivs if kind == gpu.BATCH_LU else None)
        assert info.cpu().numpy().tolist() == [0] * len(SIZES)
        for n, A, B, a, b, p in zip(SIZES, As, Bs, dA, dB, pivs):
            out, X = a.cpu().numpy(), b.cpu().numpy()
            if kind == gpu.BATCH_CHOL:
                L = np.tril(out)
                assert fro(A - L @ L.T) <= 10 * n * EPS * fro(A)
                assert np.array_equal(np.triu(out, 1), np.triu(A, 1))
            else:
                pr = np.zeros(n, np.int64)
                assert oracle.DecomposeLU(colmajor(A, n + n % 2), pr, 64) == 0
                assert np.array_equal(p.cpu().numpy(), pr), n
                PA = A.copy()
                for k in range(n):
                    PA[[k, pr[k]]] = PA[[pr[k], k]]
                assert fro(PA - (np.tril(out, -1) + np.eye(n)) @ np.triu(out)) <= 10 * n * EPS * fro(A)
            assert fro(A @ X - B) <= 10 * n * EPS * (fro(A) * fro(X) + fro(B))


@pytest.mark.parametrize("cfg", [0, 1])
def test_lu_pivot_rules(gpu, rng, cfg):
    sizes = [20, 70, 200, 300]
    ties, nans, tiny = [], [], []
    for n in sizes:
        T = rng.integers(-2, 3, (n, n)).astype(float)
        T[:, 0] = 0.0
        T[n // 2:, 0] = -2.0  # the largest magnitude, first at row n // 2
        ties.append(T)
        N = rng.standard_normal((n, n))
        N[0, 0] = N[n - 1, 0] = np.nan
        nans.append(N)
        D = np.eye(n)
        D[n - 1, n - 1] = 1e-310  # 1 / pivot overflows, b / pivot does not
        tiny.append(D)
    plan = gpu.BatchPlan(gpu.BATCH_LU, sizes, 1)
    plan.schedule([cfg] * 4)

    def run(mats, rhs):
        pivs = [torch.zeros(n, dtype=torch.int64, device="cuda") for n in sizes]
        dB = _views(gpu, rhs, 0)
        info = plan.run(_views(gpu, mats, 0), dB, pivs).cpu().numpy()
        return [p.cpu().numpy() for p in pivs], [b.cpu().numpy() for b in dB], info
    ones = [np.ones((n, 1)) for n in sizes]
    p, _, _ = run(ties, ones)
    assert [int(q[0]) for q in p] == [n // 2 for n in sizes]
    p, _, _ = run(nans, ones)
    for q, N, n in zip(p, nans, sizes):
        assert q[0] == 1 + int(np.argmax(np.abs(N[1:n - 1, 0])))
    small = [np.full((n, 1), 1e-10) for n in sizes]
    p, X, info = run(tiny, small)
    assert info.tolist() == [0] * 4
    for x in X:
        assert np.allclose(x[:-1], 1e-10, rtol=1e-15) and abs(x[-1, 0] / 1e300 - 1) <= 1e-12


@pytest.mark.parametrize("cfg", [0, 1])
@pytest.mark.parametrize("n,at", [(16, 0), (40, 15), (40, 16), (100, 33), (300, 299), (512, 255)])
def test_cholesky_failure_column(gpu, rng, n, at, cfg):
    A = np.eye(n)
    A[at, at] = -1.0
    good = np.eye(n) * 4.0
    dA, dB = _views(gpu, [A, good], 0), _views(gpu, [np.ones((n, 1)), np.ones((n, 1))], 0)
    plan = gpu.BatchPlan(gpu.BATCH_CHOL, [n, n], 1)
    plan.schedule([cfg] * 4)
    assert plan.run(dA, dB).cpu().numpy().tolist() == [at + 1, 0]
    assert np.array_equal(dB[0].cpu().numpy(), np.ones((n, 1)))  # not touched
    assert np.array_equal(dB[1].cpu().numpy(), np.full((n, 1), 0.25))
