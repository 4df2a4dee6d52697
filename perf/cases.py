"""The library's measured workloads: GEMM in its forms, transpose, Jacobi and grouped batches.

Sizes are those the tests, the benchmark and the serving mix of this repository use: regular
GEMMs of 64 to 8192 a side, skinny products with one side of 4 to 64 and the others up to
262144 x 4096, transposes up to 30000 x 17000, Jacobi grids of 512 to 8192 a side.  Entries are
U[-1, 1] (Jacobi: U[0, 1] inside a boundary of 1).  Every case is one call (or one batch) through
the Python binding on device-resident operands, as a program that keeps its data on the GPU makes
it; C operands are updated in place with |beta| <= 1, so a pass can follow a pass.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "blas-for-multi-core-dsp_gb300"))
import gbblas  # noqa: E402

ALGOS = {"auto": gbblas.ALGO_AUTO, "fp16x3": gbblas.ALGO_FP16X3}
KINDS = ("gemm", "named", "skinny", "transpose", "jacobi", "batch")


def _gemm(name, bits, mode, M, N, K, alpha, beta, algo="auto", pad=0):
    return {"name": name, "kind": "gemm", "bits": bits, "mode": mode, "M": M, "N": N, "K": K, "alpha": alpha,
            "beta": beta, "algo": algo, "pad": pad}


def listed():
    return [
        # the smallest regular product of the serving mix: one short launch
        _gemm("sgemm_256_nn", 32, "NN", 256, 256, 256, 1.0, 0.0),
        # an ordinary FP32 product of ragged sizes with the default algorithm
        _gemm("sgemm_1111x937x1500_tn", 32, "TN", 1111, 937, 1500, 1.5, -0.5),
        # the benchmark's SGEMM: padded leading dimensions, the form with FP32-level error
        _gemm("sgemm_fp16x3_4096_nt", 32, "NT", 4096, 4096, 4096, 1.5, -0.5, "fp16x3", 16),
        # a host program of the reference, calling its SGEMM by name (bit-exact summation order)
        {"name": "named_sgemm_768x1000x1536_nt", "kind": "named", "bits": 32, "mode": "NT", "M": 768, "N": 1000,
         "K": 1536},
        # the plain DGEMM configuration, C += A B^T
        _gemm("dgemm_512_nt", 64, "NT", 512, 512, 512, 1.0, 1.0),
        # an ordinary FP64 product of ragged sizes, odd leading dimensions
        _gemm("dgemm_1500x1300x1100_tn", 64, "TN", 1500, 1300, 1100, 1.0, -0.5, "auto", 3),
        # the largest: the precision study's size
        _gemm("dgemm_8192_nn", 64, "NN", 8192, 8192, 8192, 1.0, 1.0),
        # a skinny FP32 product of the serving mix: ragged, N off every tile
        {"name": "thinb_f32_20011x6007x33_nt", "kind": "skinny", "bits": 32, "side": "B", "mode": "NT",
         "rows": 20011, "n": 33, "K": 6007, "alpha": 1.25, "beta": 0.75},
        # the skinny FP64 configuration with a short A, at full size
        {"name": "shorta_f64_16x262144x4096_nn", "kind": "skinny", "bits": 64, "side": "A", "mode": "NN",
         "rows": 262144, "n": 16, "K": 4096, "alpha": 1.0, "beta": 0.0},
        # a large transpose of arbitrary shape
        {"name": "transpose_f64_12345x6789", "kind": "transpose", "bits": 64, "M": 12345, "N": 6789, "pad": 0},
        # Jacobi sweeps on a grid of the serving mix
        {"name": "jacobi_f32_1000x1500x60", "kind": "jacobi", "bits": 32, "M": 1000, "N": 1500, "iters": 60},
        # a batch of small products of mixed shapes, modes and types in one grouped launch
        {"name": "batch_48_mixed", "kind": "batch", "count": 48, "lo": 64, "hi": 384, "shapes": 7},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(KINDS + ("gemm", "skinny"))
    bits = 64 if rng.random() < 0.3 else 32
    mode = rng.choice("NT") + rng.choice("NT")
    if kind == "gemm":
        if rng.random() < 0.5:
            M = N = K = _log(rng, 256, 4096)
        else:
            M, N, K = (_log(rng, 256, 4096) for _ in range(3))
        algo = "fp16x3" if bits == 32 and rng.random() < 0.25 else "auto"
        c = _gemm("", bits, mode, M, N, K, round(rng.uniform(-2, 2), 3), rng.choice((0.0, 1.0, -0.5)), algo,
                  rng.choice((0, 0, 3, 16)))
    elif kind == "named":
        c = {"kind": kind, "bits": bits, "mode": mode, "M": _log(rng, 96, 2048), "N": _log(rng, 96, 2048),
             "K": _log(rng, 96, 2048)}
    elif kind == "skinny":
        rows, K = _log(rng, 1024, 262144), _log(rng, 1024, 65536)
        K = max(1024, min(K, (1 << 30) // rows))
        c = {"kind": kind, "bits": bits, "side": rng.choice("AB"), "mode": mode, "rows": rows, "n": rng.randint(4, 64),
             "K": K, "alpha": round(rng.uniform(-2, 2), 3), "beta": rng.choice((0.0, 0.75, -0.5))}
    elif kind == "transpose":
        c = {"kind": kind, "bits": bits, "M": _log(rng, 512, 30000), "N": _log(rng, 512, 17000),
             "pad": rng.choice((0, 0, 1, 16))}
    elif kind == "jacobi":
        c = {"kind": kind, "bits": bits, "M": _log(rng, 512, 8192), "N": _log(rng, 512, 8192),
             "iters": _log(rng, 10, 200)}
    else:
        lo = _log(rng, 32, 128)
        c = {"kind": kind, "count": rng.randint(8, 48), "lo": lo, "hi": _log(rng, lo + 1, 512),
             "shapes": rng.randint(1, 1 << 20)}
    c.pop("name", None)
    return c


# ------------------------------------------------------------------ inputs
def _dtype(bits):
    return torch.float64 if bits == 64 else torch.float32


def _uniform(gen, rows, cols, bits, lo=-1.0):
    x = torch.empty((rows, cols), dtype=_dtype(bits), device="cuda")
    return x.uniform_(lo, 1.0, generator=gen)


def _stored(gen, trans, rows, cols, bits, pad=0):
    """op(X) is rows x cols: the buffer holds it, or its transpose, with `pad` more columns."""
    r, c = (cols, rows) if trans else (rows, cols)
    return _uniform(gen, r, c + pad, bits)


def _op(X, trans, rows, cols):
    """op(X) in 64 bits from its buffer."""
    r, c = (cols, rows) if trans else (rows, cols)
    X = X[:r, :c].double()
    return X.t() if trans else X


def _batch_shapes(case):
    """The batch's (bits, modes, M, N, K), the same for every seed of the inputs."""
    import random
    rng = random.Random(case["shapes"])
    out = []
    for _ in range(case["count"]):
        out.append((64 if rng.random() < 0.3 else 32, rng.choice("NT"), rng.choice("NT"),
                    _log(rng, case["lo"], case["hi"]), _log(rng, case["lo"], case["hi"]),
                    _log(rng, case["lo"], case["hi"])))
    return out


def _dims(case):
    """M, N, K of a GEMM-like case."""
    if case["kind"] == "skinny":
        r, n = case["rows"], case["n"]
        return (r, n, case["K"]) if case["side"] == "B" else (n, r, case["K"])
    return case["M"], case["N"], case["K"]


def _inputs(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    kind = case["kind"]
    if kind in ("gemm", "named", "skinny"):
        M, N, K = _dims(case)
        ta, tb = (m == "T" for m in case["mode"])
        pad, bits = case.get("pad", 0), case["bits"]
        return {"A": _stored(gen, ta, M, K, bits, pad), "B": _stored(gen, tb, K, N, bits, pad),
                "C": _uniform(gen, M, N + pad, bits)}
    if kind == "transpose":
        return {"A": _uniform(gen, case["M"], case["N"] + case["pad"], case["bits"])}
    if kind == "jacobi":
        A = torch.ones((case["M"] + 2, case["N"] + 2), dtype=_dtype(case["bits"]), device="cuda")
        A[1:-1, 1:-1].uniform_(0.0, 1.0, generator=gen)
        return {"A": A}
    return {"items": [(_stored(gen, ta == "T", M, K, b), _stored(gen, tb == "T", K, N, b), _uniform(gen, M, N, b))
                      for b, ta, tb, M, N, K in _batch_shapes(case)]}


def prepare(case, seed):
    st = dict(case, **_inputs(case, seed))
    kind = case["kind"]
    if kind == "transpose":
        st["B"] = torch.zeros((case["N"], case["M"] + case["pad"]), dtype=_dtype(case["bits"]), device="cuda")
    elif kind == "jacobi":
        st["B"] = torch.ones_like(st["A"])
    elif kind == "batch":
        st["descs"] = [gbblas.gemm_desc(ta, tb, M, N, K, 1.5, A, A.shape[1], B, B.shape[1], -0.5, C, C.shape[1], b)
                       for (b, ta, tb, M, N, K), (A, B, C) in zip(_batch_shapes(case), st["items"])]
    return st


def run(st):
    kind = st["kind"]
    if kind in ("gemm", "skinny"):
        A, B, C = st["A"], st["B"], st["C"]
        M, N, K = _dims(st)
        gbblas.gemm(st["mode"][0], st["mode"][1], M, N, K, st["alpha"], A, A.shape[1], B, B.shape[1], st["beta"], C,
                    C.shape[1], st["bits"], algo=ALGOS[st.get("algo", "auto")])
        return C
    if kind == "named":
        A, B, C, mode = st["A"], st["B"], st["C"], st["mode"]
        ids = (0, 1) if mode == "TN" else (0,)   # barrier ids
        if st["bits"] == 64:                      # C += op(A) op(B)
            gbblas.ref_call("dgemm_" + mode, A.shape[1], B.shape[1], C.shape[1], st["M"], st["N"], st["K"], *ids,
                            A, B, C)
        else:                                     # C = alpha op(A) op(B) + beta
            gbblas.ref_call("sgemm_" + mode + "_qxx", st["M"], st["N"], st["K"], *ids, A, B, C, 5.0, 3.0)
        return C
    if kind == "transpose":
        gbblas.transpose(st["M"], st["N"], st["A"], st["A"].shape[1], st["B"], st["B"].shape[1], st["bits"])
        return st["B"]
    if kind == "jacobi":
        gbblas.stencil2d(st["M"], st["N"], st["A"], st["B"], st["iters"], bits=st["bits"])
        return st["B"] if st["iters"] % 2 else st["A"]
    gbblas.gemm_batch(st["descs"])
    return [C for _, _, C in st["items"]]


def exact(case, seed):
    st = _inputs(case, seed)
    kind = case["kind"]
    if kind in ("gemm", "skinny", "named"):
        M, N, K = _dims(case)
        P = _op(st["A"], case["mode"][0] == "T", M, K) @ _op(st["B"], case["mode"][1] == "T", K, N)
        C = st["C"].double()
        if kind != "named":
            P, C0 = case["alpha"] * P, case["beta"] * C[:, :N]
        elif case["bits"] == 64:
            C0 = C[:, :N]
        else:
            P, C0 = 5.0 * P, 3.0
        C[:, :N] = P + C0
        return C
    if kind == "transpose":
        B = torch.zeros((case["N"], case["M"] + case["pad"]), dtype=torch.float64, device="cuda")
        B[:, :case["M"]] = st["A"][:, :case["N"]].t()
        return B
    if kind == "jacobi":
        a = st["A"].double()
        b = torch.ones_like(a)
        for _ in range(case["iters"]):
            b[1:-1, 1:-1] = (a[:-2, 1:-1] + a[1:-1, :-2] + a[1:-1, 2:] + a[2:, 1:-1] + a[1:-1, 1:-1]) * 0.2
            a, b = b, a
        return a
    return [1.5 * (_op(A, ta == "T", M, K) @ _op(B, tb == "T", K, N)) - 0.5 * C.double()
            for (_, ta, tb, M, N, K), (A, B, C) in zip(_batch_shapes(case), st["items"])]


def _product(bits, M, N, K, reads_c):
    return {"bytes": bits // 8 * (M * K + K * N + (2 if reads_c else 1) * M * N), "flops": 2.0 * M * N * K}


def work(case):
    kind = case["kind"]
    if kind in ("gemm", "skinny"):
        return _product(case["bits"], *_dims(case), case["beta"] != 0.0)
    if kind == "named":
        return _product(case["bits"], *_dims(case), case["bits"] == 64)
    if kind == "transpose":
        return {"bytes": 2 * case["bits"] // 8 * case["M"] * case["N"], "flops": 0}
    if kind == "jacobi":   # the grid once in and once out; four adds and a multiply a point and sweep
        return {"bytes": 2 * case["bits"] // 8 * case["M"] * case["N"],
                "flops": 5.0 * case["M"] * case["N"] * case["iters"]}
    each = [_product(b, M, N, K, True) for b, _, _, M, N, K in _batch_shapes(case)]
    return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
