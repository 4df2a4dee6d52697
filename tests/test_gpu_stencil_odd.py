"""FP32 Jacobi with an odd number of sweeps: the result in B and the sweep left in A (that
of an even spread over an odd number of passes of at most eight), against single sweeps."""
import pytest
import torch

import gbblas

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [gbblas.STENCIL_HOST, gbblas.STENCIL_SCALAR, gbblas.STENCIL_VECTOR])
@pytest.mark.parametrize("M,N,iters", [(1, 1, 1), (5, 300, 3), (40, 113, 7), (300, 115, 9), (129, 230, 23), (64, 500, 55),
                                       (700, 900, 19), (33, 33, 127)])
def test_odd_sweeps(M, N, iters, order):
    g = torch.Generator(device="cuda").manual_seed(M + iters)
    A = torch.rand(M + 2, N + 2, generator=g, device="cuda")
    B = A.clone()
    a, b = A.clone(), A.clone()
    passes = -(-iters // 8)
    last = iters // (passes + 1 - passes % 2)
    states = [a.clone()]
    for _ in range(iters):
        gbblas.stencil2d(M, N, a, b, 1, bits=32, order=order)
        a, b = b, a
        states.append(a.clone())
    gbblas.stencil2d(M, N, A, B, iters, bits=32, order=order)
    gbblas.sync()
    assert torch.equal(B, states[iters])
    assert torch.equal(A, states[iters - last])
