"""GPU: mo_set_spin_limit in each form of the triangular solve with few right-hand sides -- one
thread-block cluster (order up to 2048), cluster-sized blocks with products between them, and the
step-flag kernel (few columns above order 12288).  With no polls allowed a wait gives up at
once: the timeout is recorded, and in the cluster the rows of every block that had to wait stay
as they were.  The context stays usable: the next call, with the default limit, solves.

Every wait ends by itself; nothing is faulted or hung.  The bound of the solve: ||op(A) X - B|| <=
10 n eps ||A|| ||X|| (the triangles are diagonally dominant)."""
import pytest
import torch

from util import EPS

pytestmark = pytest.mark.gpu

LO, TA, LEFT = 0x4, 0x1, 0x10
MO_EDEVTIMEOUT = -21


def _system(gpu, n, nrhs):
    g = torch.Generator(device="cuda").manual_seed(n + nrhs)
    A, B = gpu.matrix(n, n), gpu.matrix(n, nrhs)
    A.uniform_(-0.5, 0.5, generator=g)
    A.mul_(n ** -0.5)
    A.tril_()
    A.diagonal().add_(1.5)
    B.normal_(generator=g)
    return A, B


@pytest.mark.parametrize("flags", [LO, LO | TA])
@pytest.mark.parametrize("n,nrhs", [(200, 1), (2000, 2), (2048, 16), (4096, 16), (6000, 64), (12416, 4)])
def test_gives_up_and_recovers(gpu, n, nrhs, flags):
    A, B0 = _system(gpu, n, nrhs)
    assert gpu.Sync() == 0
    old = gpu.SetSpinLimit(0)
    try:
        B = gpu.matrix(n, nrhs)
        B.copy_(B0)
        assert gpu.SolveTrm(B, A, 1.0, LEFT | flags) is None  # enqueued
        assert gpu.Sync() == MO_EDEVTIMEOUT
        assert gpu.Sync() == 0  # the status word was cleared by the first read
        if n <= 2048:
            rest = slice(128, n) if flags == LO else slice(0, (n - 1) // 128 * 128)
            assert torch.equal(B[rest], B0[rest])
    finally:
        assert gpu.SetSpinLimit(old) == 0
    B.copy_(B0)
    assert gpu.SolveTrm(B, A, 1.0, LEFT | flags) is None
    assert gpu.Sync() == 0
    R = (A.t() if flags & TA else A) @ B - B0
    assert float(R.norm()) <= 10 * n * EPS * float(A.norm()) * float(B.norm())
