"""Ozaki digits cut four at a time, even accumulator chunks and both tile forms: exact on integers that the slices
hold, for every slice count, sign and scale, at the edges of blocks, chunks and tiles."""
import numpy as np
import pytest

from gpu_util import op_shape, torch_cuda

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    return torch_cuda()


def _run(torch, mode, opA, opB, C, slices, pad, alpha=1.0, beta=-2.0):
    import gbblas
    M, K = opA.shape
    N = opB.shape[1]
    sa, sb = op_shape(mode[0], M, K), op_shape(mode[1], K, N)
    A = torch.full((sa[0], sa[1] + pad), float("nan"), dtype=torch.float64, device="cuda:0")
    B = torch.full((sb[0], sb[1] + pad), float("nan"), dtype=torch.float64, device="cuda:0")
    A[:, :sa[1]] = opA.t() if mode[0] == "T" else opA
    B[:, :sb[1]] = opB.t() if mode[1] == "T" else opB
    D = C.clone()
    gbblas.dgemm(mode[0], mode[1], M, N, K, alpha, A, sa[1] + pad, B, sb[1] + pad, beta, D, N, algo=gbblas.ALGO_OZAKI,
                 ozaki_slices=slices)
    torch.cuda.synchronize()
    return D


@pytest.mark.parametrize("mode", ["NN", "NT", "TN", "TT"])
@pytest.mark.parametrize("slices", [2, 5, 7, 8, 9])
@pytest.mark.parametrize("M,N,K,pad", [(1, 1, 1, 0), (130, 257, 65, 1), (300, 100, 1100, 0), (129, 1300, 2111, 3)])
def test_ozaki_exact_integers(torch, mode, slices, M, N, K, pad):
    """entries of at most 13 bits are cut without loss into two slices or more; K past one accumulator chunk"""
    g = torch.Generator(device="cuda:0").manual_seed(M + N + slices)
    mk = lambda r, c: torch.randint(-4095, 4096, (r, c), generator=g, device="cuda:0").double()  # noqa: E731
    opA, opB, C = mk(M, K), mk(K, N), mk(M, N)
    opA[:, 0] = 4095.0        # a line's largest
    want = (opA @ opB) - 2.0 * C
    if slices == 2:           # the cross products of the second digits are dropped: keep them zero
        opB = (opB / 64).round()
        want = (opA @ opB) - 2.0 * C
        assert float((_run(torch, mode, opA, opB, C, slices, pad) - want).abs().max()) <= 2.0 ** 12 * K
        return
    assert torch.equal(_run(torch, mode, opA, opB, C, slices, pad), want)


@pytest.mark.parametrize("M,N,K", [(64, 300, 200), (200, 64, 1025)])
def test_ozaki_extreme_lines(torch, M, N, K):
    """powers of two at the ends of a line's range, zero lines, subnormals, results that leave the normal range"""
    g = torch.Generator(device="cuda:0").manual_seed(K)
    opA = torch.randint(-3, 4, (M, K), generator=g, device="cuda:0").double()
    opB = torch.randint(-3, 4, (K, N), generator=g, device="cuda:0").double()
    ra = np.random.default_rng(K).choice([-1070, -600, -60, 0, 3, 500], M)
    # exact powers of two, in two factors (torch.pow's are off by one place for some)
    scale = torch.from_numpy(np.ldexp(1.0, np.maximum(ra, -1000))).to("cuda:0").unsqueeze(1)
    low = torch.from_numpy(np.ldexp(1.0, np.minimum(ra + 1000, 0))).to("cuda:0").unsqueeze(1)
    want = opA @ opB
    opA[3] = 0.0
    want[3] = 0.0
    A = opA * scale * low
    got = _run(torch, "NN", A, opB, torch.zeros((M, N), dtype=torch.float64, device="cuda:0"), 8, 0, 1.0, 0.0)
    assert torch.equal(got, want * scale * low)
