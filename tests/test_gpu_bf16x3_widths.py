"""BF16X3 / FP16X3 in 64-, 128- and 256-column tiles, aligned and unaligned operands: exact on integers that the
pieces hold, in every mode, at the edges of tiles, k-blocks and waves."""
import numpy as np
import pytest

from gpu_util import dev, host, op_shape, torch_cuda

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    return torch_cuda()


@pytest.mark.parametrize("algo", ["bf16x3", "fp16x3"])
@pytest.mark.parametrize("mode", ["NN", "NT", "TN", "TT"])
@pytest.mark.parametrize("M,N,K,pad", [(513, 511, 515, 0), (128, 64, 64, 0), (130, 66, 97, 1), (1280, 1280, 96, 0),
                                       (1, 300, 70, 3), (700, 3000, 65, 2), (2100, 2500, 64, 1), (4000, 300, 40, 0)])
def test_widths_exact(torch, algo, mode, M, N, K, pad):
    import gbblas
    g = torch.Generator(device="cuda:0").manual_seed(M + N + K)
    sa, sb = op_shape(mode[0], M, K), op_shape(mode[1], K, N)
    A = torch.full((sa[0], sa[1] + pad), float("nan"), device="cuda:0")
    B = torch.full((sb[0], sb[1] + pad), float("nan"), device="cuda:0")
    A[:, :sa[1]] = torch.randint(-40, 41, sa, generator=g, device="cuda:0").float()
    B[:, :sb[1]] = torch.randint(-40, 41, sb, generator=g, device="cuda:0").float()
    C = torch.randint(-9, 10, (M, N + pad), generator=g, device="cuda:0").float()
    opA = (A[:, :sa[1]].t() if mode[0] == "T" else A[:, :sa[1]]).double()
    opB = (B[:, :sb[1]].t() if mode[1] == "T" else B[:, :sb[1]]).double()
    want = C.double()
    want[:, :N] = opA @ opB - 2.0 * want[:, :N]
    for _ in range(2):     # the second call's split overlaps the first call's GEMM
        D = C.clone()
        gbblas.sgemm(mode[0], mode[1], M, N, K, 1.0, A, sa[1] + pad, B, sb[1] + pad, -2.0, D, N + pad,
                     algo=gbblas.ALGO_BF16X3 if algo == "bf16x3" else gbblas.ALGO_FP16X3)
    torch.cuda.synchronize()
    assert torch.equal(D.double(), want)
