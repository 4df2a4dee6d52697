"""FP32 skinny products on the tensor cores that read C, in the forms of their store: equal parts, whole tiles and
K ranges, C by rows and by columns, n off sixteen, each semantics; exact on integers."""
import pytest
import torch

import gbblas

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sem", [gbblas.SEM_BLAS, gbblas.SEM_ACCUM_SCALAR_BETA, gbblas.SEM_SCALAR_BETA])
@pytest.mark.parametrize("side", "AB")
@pytest.mark.parametrize("rows,n,K", [
    (24300, 61, 1100), (24321, 33, 1500), (24300, 17, 1027),    # equal parts: 16 stages and more, under four waves
    (30011, 64, 700), (30011, 47, 961), (5003, 9, 130),         # whole tiles: under 16 stages
    (2000, 50, 2000), (77900, 20, 70)])                         # K ranges; four waves of tiles and more
def test_store_reads_c(rows, n, K, side, sem):
    g = torch.Generator(device="cuda").manual_seed(rows + n)
    ints = lambda r, c: torch.randint(-7, 8, (r, c), generator=g, device="cuda").float()
    M, N = (rows, n) if side == "B" else (n, rows)
    A, B, C = ints(M, K), ints(K, N), ints(M, N + 3)
    P, C0 = A.double() @ B.double(), C[:, :N].double()
    want = P - 2.0 * C0 if sem == gbblas.SEM_BLAS else P - 2.0 if sem == gbblas.SEM_SCALAR_BETA else C0 + P - 2.0
    pad = C[:, N:].clone()
    if side == "A":     # the large operand K-contiguous
        B = B.t().contiguous()
    gbblas.sgemm("N", "T" if side == "A" else "N", M, N, K, 1.0, A, K, B, B.shape[1], -2.0, C, N + 3, semantics=sem,
                 algo=gbblas.ALGO_SKINNY)
    gbblas.sync()
    assert torch.equal(C[:, :N].double(), want) and torch.equal(C[:, N:], pad)
