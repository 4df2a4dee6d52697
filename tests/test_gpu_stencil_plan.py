"""FP32 Jacobi at the edges of its plan: strips of 128 columns less the halo, segments of 8 rows and
up, one to six sweeps a pass -- bit-exact against the oracle."""
import numpy as np
import pytest

import oracle
from gpu_util import dev, host, torch_cuda

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    return torch_cuda()


@pytest.mark.parametrize("order", [0, 1, 2])
@pytest.mark.parametrize("M,N,iters", [(8, 116, 6), (9, 117, 11), (7, 232, 12), (65, 118, 5), (31, 349, 13),
                                       (512, 129, 3), (700, 715, 24), (2, 1500, 18), (1500, 1, 7)])
def test_stencil_f32_plan_edges(torch, order, M, N, iters):
    import gbblas
    A = np.full((M + 2, N + 2), 1.0, dtype=np.float32)
    A[1:M + 1, 1:N + 1] = oracle.fill(M, N, 23, kind=1, dtype=np.float32)
    A[0, :], A[-1, :], A[:, 0], A[:, -1] = -2.0, 3.0, 0.5, -0.25     # a boundary that tells its sides apart
    a, b = A.copy(), A.copy()
    oracle.stencil(M, N, a, b, iters, order)
    dA, dB = dev(A), dev(A)
    gbblas.stencil2d(M, N, dA, dB, iters, order, 32)
    res, want = (host(dB), b) if iters % 2 else (host(dA), a)
    assert res.tobytes() == want.tobytes()


def test_stencil_f32_captured_equals_eager(torch):
    """a captured call replays to the same bits as an eager one"""
    import gbblas
    M, N, iters = 300, 400, 14
    A = torch.rand((M + 2, N + 2), dtype=torch.float32, device="cuda:0")
    eager, eb = A.clone(), A.clone()
    gbblas.stencil2d(M, N, eager, eb, iters, 0, 32)
    cap, cb = A.clone(), A.clone()
    g = torch.cuda.CUDAGraph()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(g, stream=s):
        gbblas.stencil2d(M, N, cap, cb, iters, 0, 32, stream=s)
    cap.copy_(A)
    cb.copy_(A)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(eager, cap)
