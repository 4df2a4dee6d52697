"""The ordered FP32 GEMM off the FP64 pipe: bit-exact where rounding to 53 bits and then to 24 differs
from one rounding, where ties are the rule, at the ends of FP32's range, and at the edges of its tiles."""
import numpy as np
import pytest

import oracle
from gpu_util import dev, host, op_shape, torch_cuda

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    return torch_cuda()


def _twice_rounded(rng, M, N, K):
    """Sums where rounding to 53 bits lands on the midpoint of two floats and the sum does not: in the first block
    of 512 a 24-bit t and a product 2^-30 .. 2^-46 of half a spacing away from it, in the second a product that is
    a midpoint and a t of 2^-31."""
    A = np.zeros((M, K), np.float32)
    B = np.zeros((K, N), np.float32)
    A[:, 0] = rng.integers(2 ** 23, 2 ** 24, M).astype(np.float32)
    B[0, :] = 1.0
    A[:, 1] = (1.0 + 2.0 ** -rng.integers(15, 19, M).astype(float)) * rng.choice([0.5, -0.5], M)
    B[1, :] = 1.0 - 2.0 ** -rng.integers(15, 19, N).astype(float)
    if K > 514:
        A[:, 512] = 2.0 ** -16 * rng.choice([1.0, -1.0, 0.0], M)
        B[512, :] = 2.0 ** -15
        A[:, 513] = 2 * rng.integers(2049, 2850, M) + 1
        B[513, :] = 2 * rng.integers(2049, 2850, N) + 1
        A[:, :2] *= rng.choice([0.0, 1.0], M)[:, None]     # rows that show one block's sum alone
    return A, B


def _cases(rng, kind, M, N, K):
    if kind == "twice":
        return _twice_rounded(rng, M, N, K)
    if kind == "ties":            # integers whose sums pass 2^24
        return (rng.integers(-4000, 4000, (M, K)).astype(np.float32),
                rng.integers(-4000, 4000, (K, N)).astype(np.float32))
    A = rng.uniform(-1, 1, (M, K)).astype(np.float32)
    B = rng.uniform(-1, 1, (K, N)).astype(np.float32)
    if kind == "spread":          # products 2^-40 .. 2^40 apart, zeros among them
        A = (A * 2.0 ** rng.integers(-20, 20, A.shape)).astype(np.float32)
        B = (B * 2.0 ** rng.integers(-20, 20, B.shape)).astype(np.float32)
        A[rng.random(A.shape) < 0.2] = 0.0
    elif kind == "range":         # subnormals, overflow, Inf and NaN in some slices of some chains
        A[:, K // 3] *= np.float32(2.0 ** -130)
        A[M // 2, K // 2] = np.inf
        B[K // 4, N // 3] = np.nan
        A[0, :] = (A[0, :] * 2.0 ** 100).astype(np.float32)
        B[:, 0] = (B[:, 0] * 2.0 ** 100).astype(np.float32)
        A[M - 1, :] = (A[M - 1, :] * 2.0 ** -80).astype(np.float32)
        B[:, N - 1] = (B[:, N - 1] * 2.0 ** -60).astype(np.float32)
    return A, B


@pytest.mark.parametrize("mode", ["NN", "NT", "TN", "TT"])
@pytest.mark.parametrize("kind", ["twice", "ties", "spread", "range"])
@pytest.mark.parametrize("M,N,K", [(33, 65, 517), (300, 500, 90), (700, 640, 40)])
def test_ordered_f32_bit_exact(torch, mode, kind, M, N, K):
    import gbblas
    rng = np.random.default_rng(M + 7 * K + len(kind))
    opA, opB = _cases(rng, kind, M, N, K)
    A = np.ascontiguousarray(opA.T if mode[0] == "T" else opA)
    B = np.ascontiguousarray(opB.T if mode[1] == "T" else opB)
    assert A.shape == op_shape(mode[0], M, K) and B.shape == op_shape(mode[1], K, N)
    want = np.zeros((M, N), np.float32)
    with np.errstate(all="ignore"):
        oracle.sgemm_ref(mode[0], mode[1], M, N, K, 1.0, A, A.shape[1], B, B.shape[1], 0.0, want, N)
    dC = dev(np.full((M, N), 7.0, np.float32))
    gbblas.sgemm(mode[0], mode[1], M, N, K, 1.0, dev(A), A.shape[1], dev(B), B.shape[1], 0.0, dC, N,
                 algo=gbblas.ALGO_ORDERED, semantics=gbblas.SEM_SCALAR_BETA)
    got = host(dC)
    bad = ~((got.view(np.uint32) == want.view(np.uint32)) | (np.isnan(got) & np.isnan(want)))
    assert not bad.any(), (int(bad.sum()), got[bad][:3], want[bad][:3])


@pytest.mark.parametrize("mode", ["NN", "TT"])
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (17, 15, 16), (512, 512, 33), (600, 601, 31)])
def test_ordered_f64_tiles_bit_exact(torch, mode, M, N, K):
    import gbblas
    rng = np.random.default_rng(M)
    A = rng.uniform(-1, 1, op_shape(mode[0], M, K))
    B = rng.uniform(-1, 1, op_shape(mode[1], K, N))
    C = rng.uniform(-1, 1, (M, N))
    want = C.copy()
    oracle.dgemm_ref(mode[0], mode[1], M, N, K, A, A.shape[1], B, B.shape[1], want, N)
    dC = dev(C)
    gbblas.dgemm(mode[0], mode[1], M, N, K, 1.0, dev(A), A.shape[1], dev(B), B.shape[1], 1.0, dC, N,
                 algo=gbblas.ALGO_ORDERED)
    assert host(dC).tobytes() == want.tobytes()
