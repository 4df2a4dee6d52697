"""Ozaki DGEMM on 256 x 256 tiles of CTA pairs: the same bits as on 128 x 128 tiles, at
odd numbers of 128-row blocks (a pair's second half out of range), ragged columns,
one and several accumulator chunks, each operand order and beta form."""
import os

import pytest
import torch

import gbblas

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,ta,tb,beta", [
    (9000, 300, 4200, "N", "N", 0.0), (4097, 1280, 2500, "N", "T", -0.5), (4096, 1024, 2048, "T", "N", 1.0),
    (2432, 2561, 2113, "T", "T", 0.5), (4000, 1270, 4449, "N", "N", 2.0), (257, 18000, 2200, "N", "N", 0.0)])
def test_pair_tiles_match_narrow(M, N, K, ta, tb, beta):
    g = torch.Generator(device="cuda").manual_seed(M + K)

    def rnd(r, c):
        x = torch.rand(r, c, generator=g, device="cuda", dtype=torch.float64) - 0.5
        return x * torch.exp2(torch.randint(-30, 30, (r, 1), generator=g, device="cuda").double())

    A = rnd(*((K, M) if ta == "T" else (M, K)))
    B = rnd(*((N, K) if tb == "T" else (K, N)))
    C0 = rnd(M, N)
    got = []
    for wide in ("1", "0"):
        os.environ["GB_OZAKI_WIDE"] = wide
        try:
            C = C0.clone()
            gbblas.gemm(ta, tb, M, N, K, 1.25, A, A.shape[1], B, B.shape[1], beta, C, N, 64,
                        algo=gbblas.ALGO_OZAKI, ozaki_slices=8)
            gbblas.sync()
            got.append(C)
        finally:
            os.environ.pop("GB_OZAKI_WIDE", None)
    assert torch.equal(got[0], got[1])
