"""Plain FP32 SGEMM in small tiles with K split over thread groups and clusters: exact on small integers, and
within 2 K u of the compensated oracle, at the edges of tiles, slices and parts."""
import numpy as np
import pytest

import oracle
from gpu_util import dev, host, op_shape, torch_cuda, u_bound

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    return torch_cuda()


SHAPES = [(1, 1, 1), (32, 32, 64), (33, 31, 65), (64, 64, 4096), (100, 700, 900), (129, 65, 17), (256, 256, 256),
          (384, 380, 390), (512, 512, 513), (5, 1000, 63), (1024, 1024, 33)]


@pytest.mark.parametrize("mode", ["NN", "NT", "TN", "TT"])
@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("semantics", [0, 1, 2])
def test_simt_small_exact_on_integers(torch, mode, M, N, K, semantics):
    import gbblas
    rng = np.random.default_rng(M + N + K)
    pad = (M + K) % 5
    opA = rng.integers(-9, 10, (M, K)).astype(np.float32)
    opB = rng.integers(-9, 10, (K, N)).astype(np.float32)
    A = np.full((op_shape(mode[0], M, K)[0], op_shape(mode[0], M, K)[1] + pad), np.nan, np.float32)
    B = np.full((op_shape(mode[1], K, N)[0], op_shape(mode[1], K, N)[1] + pad), np.nan, np.float32)
    A[:, :A.shape[1] - pad] = opA.T if mode[0] == "T" else opA
    B[:, :B.shape[1] - pad] = opB.T if mode[1] == "T" else opB
    C = rng.integers(-50, 51, (M, N + pad)).astype(np.float32)
    P = 2.0 * (opA.astype(np.float64) @ opB.astype(np.float64))
    want = C.copy()
    want[:, :N] = P - 3.0 * C[:, :N] if semantics == 0 else P - 3.0 if semantics == 1 else C[:, :N] + P - 3.0
    dC = dev(C)
    gbblas.sgemm(mode[0], mode[1], M, N, K, 2.0, dev(A), A.shape[1], dev(B), B.shape[1], -3.0, dC, N + pad,
                 algo=gbblas.ALGO_SIMT, semantics=semantics)
    assert host(dC).tobytes() == want.tobytes()


@pytest.mark.parametrize("M,N,K", [(64, 64, 4096), (300, 280, 777), (512, 512, 512)])
def test_simt_small_normwise(torch, M, N, K):
    import gbblas
    A = oracle.fill(M, K, 5, dtype=np.float32)
    B = oracle.fill(K, N, 6, dtype=np.float32)
    C = oracle.fill(M, N, 7, dtype=np.float32)
    dC = dev(C)
    gbblas.sgemm("N", "N", M, N, K, 1.5, dev(A), K, dev(B), N, -0.5, dC, N, algo=gbblas.ALGO_SIMT)
    err, _ = oracle.normwise_error(host(dC), "N", "N", M, N, K, 1.5, A, K, B, N, -0.5, C, N)
    assert err <= 2 * K * u_bound(np.float32)
