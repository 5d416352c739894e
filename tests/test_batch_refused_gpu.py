"""A BatchPlan.run that is refused leaves nothing behind: the next call works on the matrices it
is given, and on no others."""
import numpy as np
import pytest
import torch

from util import EPS, fro

pytestmark = pytest.mark.gpu

SIZES = [5, 40, 33]


def _systems(gpu, rng):
    mats = [rng.uniform(-1, 1, (n, n)) for n in SIZES]
    mats = [a @ a.T + n * np.eye(n) for a, n in zip(mats, SIZES)]
    return mats, [gpu.to_device(a) for a in mats]


@pytest.mark.parametrize("kind", ["chol", "lu"])
@pytest.mark.parametrize("wrong", ["rows", "layout", "pivots"])
def test_refused_run_then_a_good_one(gpu, rng, kind, wrong):
    if wrong == "pivots" and kind == "chol":
        pytest.skip("no pivots")
    lu = kind == "lu"
    m1, a1 = _systems(gpu, rng)
    m2, a2 = _systems(gpu, rng)
    B = [rng.uniform(-1, 1, (n, 2)) for n in SIZES]
    b = [gpu.to_device(x) for x in B]
    piv = [torch.zeros(n, dtype=torch.int64, device="cuda") for n in SIZES] if lu else None
    plan = gpu.BatchPlan(gpu.BATCH_LU if lu else gpu.BATCH_CHOL, SIZES, 2)
    assert plan.run(a1, b, piv).tolist() == [0] * len(SIZES)
    done = [a.clone() for a in a1]
    for t, x in zip(b, B):
        t.copy_(torch.as_tensor(x))
    bad, badp = list(b), piv
    if wrong == "rows":
        bad[-1] = gpu.matrix(SIZES[-1] + 1, 2)
    elif wrong == "layout":
        bad[-1] = torch.zeros(SIZES[-1], 2, dtype=torch.float64, device="cuda")
    else:
        badp = piv[:-1] + [None]
    with pytest.raises((ValueError, TypeError)):
        plan.run(a2, bad, badp)
    assert plan.run(a2, b, piv).tolist() == [0] * len(SIZES)
    for A, x, t, n in zip(m2, B, b, SIZES):
        assert fro(A @ t.cpu().numpy() - x) <= 10 * n * EPS * fro(A) * fro(t.cpu().numpy())
    for x, y in zip(a1, done):
        assert torch.equal(x, y)
    for A, a in zip(m2, a2):
        assert not np.array_equal(np.tril(a.cpu().numpy()), np.tril(A))
