"""FP64 skinny products of a long K, where several CTAs share a column of W in the exponent scan: exact on
integers with a column's largest value at the start, the end and on either side of a part's edge."""
import pytest
import torch

import gbblas

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tw", ["N", "T"])
@pytest.mark.parametrize("K", [32768, 32769, 65537, 131072, 131075, 262145, 300001])
def test_column_maximum_in_any_part(K, tw):
    M, n = 70, 6
    g = torch.Generator(device="cuda").manual_seed(K)
    X = torch.randint(-3, 4, (M, K), generator=g, device="cuda").double()
    W = torch.randint(-3, 4, (K, n), generator=g, device="cuda").double()
    # 2^20 times the rest: digits cut relative to a smaller maximum would overflow
    for j, k in enumerate((0, K - 1, K // 2 - 1, K // 2, (K + 7) // 8, K - (K + 7) // 8)):
        W[k, j] = 3.0 * 2 ** 20
    W[:, 5] = 0.0
    stored = W.t().contiguous() if tw == "T" else W
    C = torch.full((M, n), float("nan"), dtype=torch.float64, device="cuda")
    gbblas.dgemm("N", tw, M, n, K, 1.0, X, K, stored, stored.shape[1], 0.0, C, n, algo=gbblas.ALGO_SKINNY)
    gbblas.sync()
    assert torch.equal(C, X @ W)


@pytest.mark.parametrize("rows", [2358, 1976, 4850, 2300])    # 19, 16 and 38 row tiles: ranges in a row; 18: by ranges
@pytest.mark.parametrize("split", [0, 1, 5])
def test_order_of_units_in_pieces(rows, split):
    """K-major X of an odd leading dimension, in either order of its units."""
    K, n, ld = 2700, 7, rows + (rows + 1) % 2
    g = torch.Generator(device="cuda").manual_seed(rows)
    X = torch.randint(-9, 10, (K, ld), generator=g, device="cuda").double()
    W = torch.randint(-9, 10, (K, n), generator=g, device="cuda").double()
    C = torch.randint(-9, 10, (rows, n), generator=g, device="cuda").double()
    want = X[:, :rows].t() @ W - 2.0 * C
    gbblas.dgemm("T", "N", rows, n, K, 1.0, X, ld, W, n, -2.0, C, n, algo=gbblas.ALGO_SKINNY, split_k=split)
    gbblas.sync()
    assert torch.equal(C, want)
