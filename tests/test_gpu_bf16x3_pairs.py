"""BF16X3 on 256 x 256 tiles of two CTAs, plain and folding: odd numbers of 128-row
blocks (the second CTA out of range), ragged rows and columns, K off every stage,
each operand order and beta form, against FP64; and C's padding left alone."""
import pytest
import torch

import gbblas

pytestmark = pytest.mark.gpu


# 8192 columns and more: long waves of wide tiles, which go to pairs
@pytest.mark.parametrize("M,N,K,ta,tb,beta,accum_k", [
    (4096, 8192, 64, "N", "N", 0.0, 0), (8065, 8190, 333, "N", "T", -0.5, 0), (4097, 8195, 1000, "T", "N", 1.0, 0),
    (3967, 6145, 2049, "T", "T", 0.5, 0), (2500, 2561, 1111, "N", "N", -0.5, 512), (4225, 1793, 2050, "T", "N", 1.0, 1024)])
def test_pair_tiles(M, N, K, ta, tb, beta, accum_k):
    g = torch.Generator(device="cuda").manual_seed(M + K)
    A = torch.rand(*((K, M) if ta == "T" else (M, K)), generator=g, device="cuda") * 2 - 1
    B = torch.rand(*((N, K) if tb == "T" else (K, N)), generator=g, device="cuda") * 2 - 1
    C = torch.rand(M, N + 3, generator=g, device="cuda") * 2 - 1
    C0 = C.clone()
    gbblas.gemm(ta, tb, M, N, K, 1.25, A, A.shape[1], B, B.shape[1], beta, C, N + 3, 32,
                algo=gbblas.ALGO_BF16X3, accum_k=accum_k)
    gbblas.sync()
    opA, opB = (A.t() if ta == "T" else A).double(), (B.t() if tb == "T" else B).double()
    want = 1.25 * (opA @ opB) + beta * C0[:, :N].double()
    mag = 1.25 * (opA.abs() @ opB.abs()) + abs(beta) * C0[:, :N].double().abs()
    # two pieces carry 16 bits: 2^-16 a product; the accumulator one unit in the last place per MMA
    # (three products a 16-long step), truncating, of a sum within mag
    tol = (3 * 2.0 ** -16 + 3 * (min(K, accum_k or K) // 16 + 2) * 2.0 ** -23 + 4 * 2.0 ** -24) * mag
    assert ((C[:, :N].double() - want).abs() <= tol).all()
    assert torch.equal(C[:, N:], C0[:, N:])
