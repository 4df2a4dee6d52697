"""Transpose: each tile and access form that csrc/transpose.cu chooses between, at
its edges (partial tiles, odd leading dimensions, streams beyond the L2, more rows
than 32-row blocks can number).  B = A^T and B += A^T are exact against torch."""
import pytest
import torch

import gbblas

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("M,N,pa,pb", [(1, 1, 0, 0), (31, 33, 1, 0), (65, 127, 0, 3), (700, 900, 2, 2),
                                       (1153, 1217, 0, 1), (1216, 1280, 0, 0), (2200001, 2, 0, 0),
                                       (4001, 2003, 1, 1), (6001, 3001, 0, 0), (3, 70001, 0, 1)])
def test_transpose_tiles(bits, M, N, pa, pb):
    dt = torch.float64 if bits == 64 else torch.float32
    g = torch.Generator(device="cuda").manual_seed(M + N)
    A = torch.rand(M, N + pa, generator=g, device="cuda", dtype=dt)
    B0 = torch.rand(N, M + pb, generator=g, device="cuda", dtype=dt)
    for op, want in ((gbblas.transpose, A[:, :N].t()), (gbblas.transpose_add, B0[:, :M] + A[:, :N].t())):
        B = B0.clone()
        op(M, N, A, N + pa, B, M + pb, bits)
        gbblas.sync()
        assert torch.equal(B[:, :M], want)
        assert torch.equal(B[:, M:], B0[:, M:])
