"""The grouped kernel's tiles (FP64 16 x 16 and 32 x 32, FP32 64 x 64) at their edges: exact on small integers for
batches of mixed shapes, modes, types and semantics, few and many, K from 0 on."""
import numpy as np
import pytest

from gpu_util import torch_cuda

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    return torch_cuda()


@pytest.mark.parametrize("count,lo,hi", [(1, 1, 2), (7, 1, 70), (40, 15, 67), (12, 250, 400), (60, 120, 300)])
@pytest.mark.parametrize("bits", [0, 32, 64])
def test_grouped_exact(torch, count, lo, hi, bits):
    import gbblas
    rng = np.random.default_rng(count + hi + bits)
    g = torch.Generator(device="cuda:0").manual_seed(count)
    keep, descs, wants = [], [], []
    for i in range(count):
        b = bits or int(rng.choice([32, 64]))
        dt = torch.float64 if b == 64 else torch.float32
        ta, tb, sem = rng.choice(["N", "T"]), rng.choice(["N", "T"]), int(rng.integers(0, 3))
        M, N, K = (int(x) for x in rng.integers(lo, hi, 3))
        if i % 9 == 4:
            K = int(rng.choice([0, 1, 15, 16, 17]))
        pad = int(rng.integers(0, 3))
        mk = lambda r, c: torch.randint(-9, 10, (max(r, 1), max(c, 1) + pad), generator=g, device="cuda:0").to(dt)  # noqa: E731
        A, B, C = (mk(K, M) if ta == "T" else mk(M, K)), (mk(N, K) if tb == "T" else mk(K, N)), mk(M, N)
        opA = (A[:K, :M].t() if ta == "T" else A[:M, :K]).double()
        opB = (B[:N, :K].t() if tb == "T" else B[:K, :N]).double()
        want = C.double().clone()
        P = 2.0 * (opA @ opB) if K else torch.zeros((M, N), dtype=torch.float64, device="cuda:0")
        want[:, :N] = P - 3.0 * want[:, :N] if sem == 0 else P - 3.0 if sem == 1 else want[:, :N] + P - 3.0
        descs.append(gbblas.gemm_desc(str(ta), str(tb), M, N, K, 2.0, A, A.shape[1], B, B.shape[1], -3.0, C, C.shape[1],
                                      b, sem))
        keep.append((A, B, C))
        wants.append(want)
    gbblas.gemm_batch(descs)
    torch.cuda.synchronize()
    for (A, B, C), want in zip(keep, wants):
        assert torch.equal(C.double(), want)
