"""DecomposeCHOLAdjointBatched under stream capture is refused: its table of matrices is uploaded from
the call's own host memory, which a replay would read after it is gone.  (Nothing is replayed
here.)  Outside a capture the same call works as before."""
import pytest
import torch

pytestmark = pytest.mark.gpu

LO = 0x4


def test_refused_while_capturing(gpu):
    n = 20
    L, G = gpu.matrix(n, n, fill=0.0), gpu.matrix(n, n, fill=0.0)
    L.fill_diagonal_(2.0)
    G.fill_diagonal_(1.0)
    assert gpu.DecomposeCHOLAdjointBatched([L], [G], LO) is None
    torch.cuda.synchronize()
    want = G.clone()
    G.zero_()
    G.fill_diagonal_(1.0)
    keep = G.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        with pytest.raises(RuntimeError):
            gpu.DecomposeCHOLAdjointBatched([L], [G], LO)
    del graph
    torch.cuda.synchronize()
    assert torch.equal(G, keep)
    assert gpu.DecomposeCHOLAdjointBatched([L], [G], LO) is None
    assert torch.equal(G, want) and float(G[3, 3]) == 0.25
