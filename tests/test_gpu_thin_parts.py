"""Skinny products whose stages are shared out in equal parts: exact on small integers where parts begin and end at
tile edges, inside one tile, and after whole waves; every layout of the large operand."""
import pytest

from gpu_util import torch_cuda

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    return torch_cuda()


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("mode,side", [("NN", "B"), ("TT", "B"), ("NT", "A"), ("TN", "A")])
@pytest.mark.parametrize("rows,n,K,pad", [(1, 9, 64, 0), (130, 33, 5000, 1), (1024, 16, 1030, 0), (19456, 12, 130, 0),
                                          (19457, 20, 514, 3), (60001, 40, 70, 0), (5000, 64, 700, 2)])
def test_equal_parts_exact(torch, bits, mode, side, rows, n, K, pad):
    import gbblas
    dt = torch.float64 if bits == 64 else torch.float32
    M, N = (rows, n) if side == "B" else (n, rows)
    g = torch.Generator(device="cuda:0").manual_seed(rows + n)
    mk = lambda r, c: torch.randint(-9, 10, (r, c + pad), generator=g, device="cuda:0").to(dt)  # noqa: E731
    A = mk(K, M) if mode[0] == "T" else mk(M, K)
    B = mk(N, K) if mode[1] == "T" else mk(K, N)
    C = mk(M, N)
    opA = (A[:, :M].t() if mode[0] == "T" else A[:, :K]).double()
    opB = (B[:, :K].t() if mode[1] == "T" else B[:, :N]).double()
    want = C.double().clone()
    want[:, :N] = 2.0 * (opA @ opB) - 3.0 * want[:, :N]
    for _ in range(2):
        D = C.clone()
        gbblas.gemm(mode[0], mode[1], M, N, K, 2.0, A, A.shape[1], B, B.shape[1], -3.0, D, N + pad, bits,
                    algo=gbblas.ALGO_SKINNY)
    torch.cuda.synchronize()
    assert torch.equal(D.double(), want)
