"""Ozaki DGEMM captured with less scratch than its shared tiles take: it runs with one CTA per tile, gives the same
bits, and leaves no error status behind."""
import pytest
import torch

import gbblas

pytestmark = pytest.mark.gpu


def test_capture_without_room_for_shared_tiles():
    M, N, K, s = 600, 600, 4000, 8
    g = torch.Generator(device="cuda").manual_seed(1)
    A = torch.rand(M, K, generator=g, dtype=torch.float64, device="cuda") - 0.5
    B = torch.rand(K, N, generator=g, dtype=torch.float64, device="cuda") - 0.5
    want = torch.zeros(M, N, dtype=torch.float64, device="cuda")
    gbblas.dgemm("N", "N", M, N, K, 1.0, A, K, B, N, 0.0, want, N, algo=gbblas.ALGO_OZAKI, ozaki_slices=s)
    torch.cuda.synchronize()
    st = torch.cuda.Stream()
    mp = (M + 127) // 128 * 128
    kp = (K + 63) // 64 * 64
    # the digit slices, exponents and line maxima, without the parts' sums
    gbblas.workspace_reserve(2 * s * mp * kp * 2 + 2 * mp * 12 + 256 + 4096, st)
    assert gbblas.workspace_query(64, "N", "N", M, N, K, K, N, algo=gbblas.ALGO_OZAKI, ozaki_slices=s) > \
        2 * s * mp * kp * 2 + 2 * mp * 12 + 256 + 4096
    C = torch.full((M, N), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    gbblas.lib().gb_clear_last_status()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=st):
        gbblas.dgemm("N", "N", M, N, K, 1.0, A, K, B, N, 0.0, C, N, algo=gbblas.ALGO_OZAKI, ozaki_slices=s, stream=st)
    assert gbblas.lib().gb_get_last_status() == gbblas.OK, gbblas.lib().gb_last_error()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(C, want)
