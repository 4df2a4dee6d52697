"""Ozaki DGEMM with a tile's digit pairs shared by several CTAs: the same bits as one CTA
per tile, from one tile to as many as are shared, one and several accumulator chunks,
few and many slices, ragged edges, each operand order, beta form and a non-finite row."""
import os

import pytest
import torch

import gbblas

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,ta,tb,beta,s", [
    (1, 1, 64, "N", "N", 0.0, 8), (128, 128, 5000, "N", "T", -0.5, 8), (100, 130, 16000, "T", "N", 1.0, 7),
    (300, 300, 1025, "T", "T", 0.5, 9), (513, 640, 700, "N", "N", 2.0, 2), (1000, 1000, 1000, "N", "T", 1.0, 8),
    (900, 1100, 2100, "T", "N", 0.0, 5), (128, 1200, 333, "N", "N", -1.0, 8), (70, 40, 20000, "N", "N", 0.0, 8)])
def test_split_matches_whole(M, N, K, ta, tb, beta, s):
    g = torch.Generator(device="cuda").manual_seed(M + K)

    def rnd(r, c):
        x = torch.rand(r, c, generator=g, device="cuda", dtype=torch.float64) - 0.5
        return x * torch.exp2(torch.randint(-30, 30, (r, 1), generator=g, device="cuda").double())

    A = rnd(*((K, M) if ta == "T" else (M, K)))
    B = rnd(*((N, K) if tb == "T" else (K, N)))
    A[-1, -1] = float("inf")
    C0 = rnd(M, N)
    got = []
    for split in ("1", "0"):
        os.environ["GB_OZAKI_SPLIT"] = split
        try:
            C = C0.clone()
            gbblas.gemm(ta, tb, M, N, K, 1.25, A, A.shape[1], B, B.shape[1], beta, C, N, 64,
                        algo=gbblas.ALGO_OZAKI, ozaki_slices=s)
            gbblas.sync()
            got.append(C)
        finally:
            os.environ.pop("GB_OZAKI_SPLIT", None)
    assert torch.equal(got[0].view(torch.int64), got[1].view(torch.int64))
    assert torch.isfinite(got[0]).all(dim=1).sum() >= M - 1
