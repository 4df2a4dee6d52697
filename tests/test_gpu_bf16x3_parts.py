"""BF16X3 with a tile's k-blocks shared by several CTAs: few tiles and a long K, ragged
sizes and leading dimensions, each operand order and each of the epilogue's forms,
against FP64; calls back to back on one stream reuse the workspace halves."""
import pytest
import torch

import gbblas

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sem", [gbblas.SEM_BLAS, gbblas.SEM_SCALAR_BETA, gbblas.SEM_ACCUM_SCALAR_BETA])
@pytest.mark.parametrize("M,N,K,ta,tb,beta", [
    (256, 256, 4096, "N", "N", 0.0), (300, 401, 4001, "N", "T", -0.5), (512, 511, 4096, "T", "N", 1.0),
    (1, 64, 2500, "T", "T", 0.5), (129, 65, 8000, "N", "N", -0.5), (800, 800, 3000, "T", "N", 2.0)])
def test_shared_tiles(M, N, K, ta, tb, beta, sem):
    g = torch.Generator(device="cuda").manual_seed(M + K)
    A = torch.rand(*((K, M) if ta == "T" else (M, K)), generator=g, device="cuda") * 2 - 1
    B = torch.rand(*((N, K) if tb == "T" else (K, N)), generator=g, device="cuda") * 2 - 1
    C0 = torch.rand(M, N + 3, generator=g, device="cuda") * 2 - 1
    opA, opB = (A.t() if ta == "T" else A).double(), (B.t() if tb == "T" else B).double()
    x, c = 1.25 * (opA @ opB), C0[:, :N].double()
    want = x + beta * c if sem == gbblas.SEM_BLAS else x + beta if sem == gbblas.SEM_SCALAR_BETA else c + x + beta
    mag = 1.25 * (opA.abs() @ opB.abs()) + abs(beta) + (1 + abs(beta)) * c.abs()
    # two pieces carry 16 bits: 2^-16 a product; the accumulator one unit in the last place per MMA
    # (three products a 16-long step), truncating, of a sum within mag
    tol = (3 * 2.0 ** -16 + 3 * (K // 16 + 2) * 2.0 ** -23 + 20 * 2.0 ** -24) * mag
    outs = [C0.clone() for _ in range(3)]
    for C in outs:
        gbblas.gemm(ta, tb, M, N, K, 1.25, A, A.shape[1], B, B.shape[1], beta, C, N + 3, 32,
                    algo=gbblas.ALGO_BF16X3, semantics=sem)
    gbblas.sync()
    assert ((outs[0][:, :N].double() - want).abs() <= tol).all()
    assert torch.equal(outs[0][:, N:], C0[:, N:])
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
