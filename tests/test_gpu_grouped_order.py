"""Grouped launches whose list is reordered: many GEMMs of mixed types and K, empty ones and K = 0 among them, and
thin outputs of a short K, whose time is their store; exact on integers, padding left alone."""
import random

import pytest
import torch

import gbblas

pytestmark = pytest.mark.gpu


def _run(items, sem, alpha, beta):
    """items: (bits, ta, tb, M, N, K)"""
    g = torch.Generator(device="cuda").manual_seed(len(items))
    flat = {b: torch.randint(-6, 7, (1 << 20,), generator=g, device="cuda").to(t)
            for b, t in ((32, torch.float32), (64, torch.float64))}
    rng, descs, outs = random.Random(len(items)), [], []
    for b, ta, tb, M, N, K in items:
        take = lambda r, c: flat[b][(o := rng.randrange(1 << 18)):o + r * c].view(r, c)
        A, B = take(*((K, M) if ta == "T" else (M, K))), take(*((N, K) if tb == "T" else (K, N)))
        C = take(M, N + 2).clone()
        want = C.double().clone()
        P = (A.t() if ta == "T" else A).double() @ (B.t() if tb == "T" else B).double()
        c0 = want[:, :N]
        want[:, :N] = (alpha * P + beta * c0 if sem == gbblas.SEM_BLAS else alpha * P + beta if sem == gbblas.SEM_SCALAR_BETA
                       else c0 + alpha * P + beta)
        outs.append((C, want))
        descs.append(gbblas.gemm_desc(ta, tb, M, N, K, alpha, A, max(1, A.shape[1]), B, max(1, B.shape[1]), beta, C,
                                      N + 2, b, semantics=sem))
    gbblas.gemm_batch(descs)
    gbblas.sync()
    for i, (C, want) in enumerate(outs):
        assert torch.equal(C.double(), want), items[i]


@pytest.mark.parametrize("n", [2, 33, 700, 4096])
def test_mixed_list(n):
    rng = random.Random(n)
    _run([(rng.choice((32, 64)), rng.choice("NT"), rng.choice("NT"), rng.randint(0, 20), rng.randint(1, 20),
           rng.choice((0, 1, 2, 7, 8, 9, 15, 16, 17, 31, 64, 200))) for _ in range(n)], gbblas.SEM_BLAS, 2.0, -1.0)


@pytest.mark.parametrize("sem", [gbblas.SEM_BLAS, gbblas.SEM_SCALAR_BETA, gbblas.SEM_ACCUM_SCALAR_BETA])
def test_thin_outputs_of_a_short_k(sem):
    _run([(b, ta, tb, M, N, K) for b in (32, 64) for ta in "NT" for tb in "NT"
          for M, N, K in ((180, 9, 11), (9, 180, 1), (1, 1, 3), (65, 3, 16), (3, 65, 17), (64, 64, 5))], sem, 1.0, -2.0)
