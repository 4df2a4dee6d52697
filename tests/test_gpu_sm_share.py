"""Requests that the server plans for a share of the SMs (long_sm_percent), down to one SM: every form's
plan launches and gives exact results on integers, as without a cap."""
import numpy as np
import pytest

from gpu_util import dev, host, op_shape, torch_cuda

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    return torch_cuda()


def _serve(req, percent):
    import gbblas
    with gbblas.Server(streams=2, short_streams=1, short_us=1.0, long_sm_percent=percent, use_graphs=0,
                       use_grouped=0) as s:
        s.submit(req)
        s.drain(60.0)
        st = s.stats()
    assert st["failed"] == 0 and st["completed"] == 1 and st["urgent_launches"] == 0


@pytest.mark.parametrize("percent", [1, 2, 50])
@pytest.mark.parametrize("bits,algo,M,N,K,fold", [
    (32, "BF16X3", 300, 520, 1100, 32),    # folding form: more than a wave of 256 columns, K past 1024
    (32, "BF16X3", 300, 520, 1100, 0), (32, "BF16X3", 129, 70, 2500, 0), (32, "FP16X3", 300, 520, 300, 0),
    (32, "BF16X6", 200, 300, 300, 0), (32, "SIMT", 130, 200, 70, 0), (32, "ORDERED", 100, 70, 600, 0),
    (32, "SKINNY", 3000, 33, 1500, 0), (32, "SKINNY", 1500, 12, 800, 0), (64, "OZAKI", 300, 520, 200, 0),
    (64, "OZAKI", 100, 130, 1500, 0), (64, "SKINNY", 2000, 20, 1500, 0), (64, "ORDERED", 100, 70, 100, 0)])
def test_capped_gemm(torch, monkeypatch, bits, algo, M, N, K, fold, percent):
    import gbblas
    if fold:
        monkeypatch.setenv("GB_BF16X3_FOLD", str(fold))
    rng = np.random.default_rng(M + K)
    dt = np.float64 if bits == 64 else np.float32
    A = rng.integers(-8, 9, op_shape("T", M, K)).astype(dt)
    B = rng.integers(-8, 9, (K, N)).astype(dt)
    C = rng.integers(-8, 9, (M, N)).astype(dt)
    want = A.T.astype(np.float64) @ B.astype(np.float64) - 2.0 * C
    dA, dB, dC = dev(A), dev(B), dev(C)
    torch.cuda.synchronize()
    _serve(gbblas.request(gbblas.OP_GEMM, bits, M, N, K, A=dA, lda=M, B=dB, ldb=N, C=dC, ldc=N, ta="T", beta=-2.0,
                          algo=getattr(gbblas, "ALGO_" + algo)), percent)
    assert np.array_equal(host(dC).astype(np.float64), want)


@pytest.mark.parametrize("percent", [1, 2])
def test_capped_jacobi(torch, percent):
    import gbblas
    rng = np.random.default_rng(5)
    G = rng.random((302, 402), dtype=np.float32)
    a, b, c, d = dev(G), dev(G), dev(G), dev(G)
    gbblas.stencil2d(300, 400, c, d, 13, bits=32)
    torch.cuda.synchronize()
    _serve(gbblas.request(gbblas.OP_STENCIL, 32, 300, 400, A=a, C=b, iters=13), percent)
    assert np.array_equal(host(b), host(d))
