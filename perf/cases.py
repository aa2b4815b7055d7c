"""Performance cases: what a user of this library has it do.

Each case is one call, or one short chain of calls, through a public entry
point: the six functions with MATLAB semantics on host arrays
(``mex_linear_algebra_b200.mela``), the packed device entry points
(``mex_linear_algebra_b200.device`` and the C ABI of include/mela.h) and the
batched rank + null-space plan.  ``listed()`` gives fixed cases, ``draw(rng)``
more of the same ranges, ``prepare`` what a program holds before the call,
``run`` one pass, ``work`` what a pass cannot do without, and ``exact`` the
result by plain numpy or torch arithmetic.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from mex_linear_algebra_b200 import _lib, device, mela

# Ones per row of a parity-check matrix (the batch configuration's value).
ROW_ONES = 6


def listed():
    return [
        # the smallest products: one call on arrays a user types in or reads
        # from a small code; latency and launches count
        dict(name="product-small", kind="product", fn="gf2", m=100, k=120, n=80, dtype="logical"),
        # the drop-in call of the first configuration: doubles 0/1 in, logical out
        dict(name="product-double", kind="product", fn="gf2", m=2048, k=2048, n=1024, dtype="double"),
        # an odd-sized product through the Four-Russians function
        dict(name="product-m4ri-odd", kind="product", fn="m4ri", m=3001, k=2500, n=1777, dtype="logical"),
        # null space of a small parity-check matrix
        dict(name="null-small", kind="null", fn="gf2", m=72, n=149, dtype="logical", matrix="parity"),
        # rank of a parity-check matrix of the batch configuration's largest size
        dict(name="rank-parity", kind="rank", fn="gf2", m=1000, n=2100, dtype="logical", matrix="parity"),
        # rank of dense doubles with dependent rows, Four-Russians function
        dict(name="rank-m4ri-double", kind="rank", fn="m4ri", m=1501, n=2900, dtype="double", matrix="dense"),
        # null space of a dense logical matrix, Four-Russians function
        dict(name="null-m4ri", kind="null", fn="m4ri", m=2048, n=4096, dtype="logical", matrix="dense"),
        # the large dense product on packed device matrices
        dict(name="packed-product-32768", kind="packed_product", m=32768, k=32768, n=32768),
        # MATLAB-layout arrays already on the GPU: pack, multiply, unpack
        dict(name="device-chain-odd", kind="chain", m=4001, k=3000, n=3510, dtype="logical"),
        # rank of a mid-size packed device matrix, as the mixed request stream has them
        dict(name="packed-rank", kind="packed_rank", m=3000, n=5000, rank=2200),
        # rank and null-space basis of the large dense rank-deficient matrix
        dict(name="packed-null-16384", kind="packed_null", m=16384, n=32768, rank=12000),
        # a batch of parity-check matrices of uneven shape from logical input
        dict(name="batch-parity", kind="batch", count=4000, lo=64, hi=1024),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["product", "product", "null", "rank", "rank", "packed_product", "chain", "packed_rank",
                       "packed_null", "batch"])
    if kind == "product":
        # host arrays up to a few thousand rows, either function and class
        return dict(kind=kind, fn=rng.choice(["gf2", "m4ri"]), m=_log_uniform(rng, 64, 3500),
                    k=_log_uniform(rng, 64, 3500), n=_log_uniform(rng, 64, 3500),
                    dtype=rng.choice(["logical", "double"]))
    if kind in ("null", "rank"):
        m = _log_uniform(rng, 48, 2500)
        matrix = rng.choice(["parity", "dense"])
        return dict(kind=kind, fn=rng.choice(["gf2", "m4ri"]), m=m,
                    n=int(m * rng.uniform(1.9 if matrix == "parity" else 1.0, 2.3)) + 1,
                    dtype=rng.choice(["logical", "double"]), matrix=matrix)
    if kind == "packed_product":
        return dict(kind=kind, m=_log_uniform(rng, 64, 32768), k=_log_uniform(rng, 64, 32768),
                    n=_log_uniform(rng, 64, 32768))
    if kind == "chain":
        return dict(kind=kind, m=_log_uniform(rng, 100, 8192), k=_log_uniform(rng, 100, 8192),
                    n=_log_uniform(rng, 100, 8192), dtype=rng.choice(["logical", "double"]))
    if kind == "packed_rank":
        # the mixed request stream's sizes, at most 8:1
        m = _log_uniform(rng, 64, 8192)
        n = min(max(_log_uniform(rng, 64, 8192), m // 8), m * 8)
        return dict(kind=kind, m=m, n=n, rank=max(1, int(min(m, n) * rng.uniform(0.4, 1.0))))
    if kind == "packed_null":
        m = _log_uniform(rng, 512, 16384)
        return dict(kind=kind, m=m, n=int(m * rng.uniform(1.0, 2.0)), rank=max(1, int(m * rng.uniform(0.4, 1.0))))
    hi = _log_uniform(rng, 128, 1024)
    return dict(kind=kind, count=_log_uniform(rng, 200, 4000), lo=min(64, hi // 2), hi=hi)


# ------------------------------------------------------------------ inputs
def _host_array(rng, m, n, dtype, matrix, dependent):
    """A MATLAB-layout (Fortran order) logical or double array, `dependent`
    of its rows replaced by the sum of two of the others."""
    if matrix == "parity":
        a = np.zeros((m, n), dtype=np.bool_, order="F")
        cols = rng.integers(0, n, size=(m, min(ROW_ONES, n)))
        a[np.arange(m)[:, None], cols] = True
    else:
        a = np.asfortranarray(rng.integers(0, 2, size=(m, n), dtype=np.uint8).astype(np.bool_))
    if dependent:
        order = rng.permutation(m)
        i, rest = order[:dependent], order[dependent:]
        a[i] = a[rng.choice(rest, dependent)] ^ a[rng.choice(rest, dependent)]
    return a if dtype == "logical" else np.asfortranarray(a.astype(np.float64))


def _host_inputs(case, seed):
    rng = np.random.default_rng(seed)
    if case["kind"] == "product":
        def one(r, c):
            a = np.asfortranarray(rng.integers(0, 2, size=(r, c), dtype=np.uint8).astype(np.bool_))
            return a if case["dtype"] == "logical" else np.asfortranarray(a.astype(np.float64))
        return one(case["m"], case["k"]), one(case["k"], case["n"])
    # ranks: up to a quarter of the rows dependent; null spaces: an eighth of
    # a dense matrix's rows, a parity-check matrix as it is
    m = case["m"]
    dependent = int(rng.integers(1, m // 4 + 1)) if case["kind"] == "rank" else m // 8 if case["matrix"] == "dense" else 0
    return (_host_array(rng, m, case["n"], case["dtype"], case["matrix"], dependent),)


def _low_rank(seed, m, n, r):
    """Packed m x n product of random m x r and r x n factors."""
    left = device.rand_dense(seed, 0, m, r)
    right = device.rand_dense(seed, 1, r, n)
    return device.matmul(left, right, m, r, n)


def _device_arrays(case, seed):
    """Column-major (flat) arrays of the chain case on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)

    def one(r, c):
        a = torch.randint(0, 2, (r * c,), generator=g, device="cuda", dtype=torch.uint8)
        return a if case["dtype"] == "logical" else a.to(torch.float64)
    return one(case["m"], case["k"]), one(case["k"], case["n"])


def _parity_batch(case, seed):
    """Shapes and logical column-major bytes of a batch of parity-check
    matrices: m uniform in [lo, hi], n = 2m +- up to m/4, 6 ones a row.  The
    shapes are the case's, the ones the seed's."""
    rng = np.random.default_rng(case["count"])
    m = rng.integers(case["lo"], case["hi"] + 1, size=case["count"])
    n = 2 * m + rng.integers(-(m // 4), m // 4 + 1)
    shapes = np.stack([m, n], axis=1).astype(np.int64)
    offs = np.concatenate([[0], np.cumsum(m * n)])
    total = int(offs[-1])
    mat = torch.from_numpy(np.repeat(np.arange(case["count"]), m)).cuda()
    row0 = np.concatenate([[0], np.cumsum(m)[:-1]])
    dm = torch.from_numpy(m).cuda()[mat]
    dn = torch.from_numpy(n).cuda()[mat]
    row = torch.arange(len(mat), device="cuda") - torch.from_numpy(row0).cuda()[mat]
    off = torch.from_numpy(offs[:-1]).cuda()[mat]
    g = torch.Generator(device="cuda").manual_seed(seed)
    u = torch.rand((len(mat), ROW_ONES), generator=g, device="cuda", dtype=torch.float64)
    cols = (u * dn[:, None]).to(torch.int64)
    buf = torch.zeros(total, dtype=torch.uint8, device="cuda")
    buf[(off[:, None] + cols * dm[:, None] + row[:, None]).reshape(-1)] = 1
    return shapes, buf


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("product", "null", "rank"):
        fn = getattr(mela, {"product": "mela_matmul_", "null": "mela_null_", "rank": "mela_rank_"}[kind] + case["fn"])
        return dict(kind=kind, fn=fn, args=_host_inputs(case, seed))
    m, n = case.get("m"), case.get("n")
    if kind == "packed_product":
        k = case["k"]
        return dict(kind=kind, m=m, k=k, n=n, A=device.rand_dense(seed, 0, m, k), B=device.rand_dense(seed, 1, k, n))
    if kind == "chain":
        A, B = _device_arrays(case, seed)
        return dict(kind=kind, m=m, k=case["k"], n=n, A=A, B=B)
    if kind in ("packed_rank", "packed_null"):
        A = _low_rank(seed, m, n, case["rank"])
        wsb = int(_lib.lib().mela_elim_workspace_size(m, n))
        mn = min(m, n)
        return dict(kind=kind, m=m, n=n, A=A, work=torch.empty_like(A),
                    ws=torch.empty(wsb, dtype=torch.uint8, device="cuda"),
                    rank=torch.zeros(1, dtype=torch.int64, device="cuda"),
                    piv=torch.zeros(mn, dtype=torch.int64, device="cuda"),
                    prow=torch.zeros(mn, dtype=torch.int64, device="cuda"))
    shapes, buf = _parity_batch(case, seed)
    plan = device.BatchPlan(shapes)
    ranks = torch.zeros(plan.count, dtype=torch.int64, device="cuda")
    zt = torch.zeros(plan.z_words, dtype=torch.int64, device="cuda")
    return dict(kind=kind, plan=plan, buf=buf, ranks=ranks, zt=zt)


# ------------------------------------------------------------------ one pass
def _eliminate(s, rref):
    """Rank or RREF of a copy of the matrix (the calls work in place)."""
    L = _lib.lib()
    s["work"].copy_(s["A"])
    fn = L.mela_dev_rref if rref else L.mela_dev_rank
    _lib.check(fn(_lib.ELIM_AUTO, s["work"].data_ptr(), s["work"].shape[1], s["m"], s["n"], s["rank"].data_ptr(),
                  s["piv"].data_ptr(), s["prow"].data_ptr(), s["ws"].data_ptr(), s["ws"].numel(),
                  torch.cuda.current_stream().cuda_stream))
    return int(s["rank"].item())


def run(state):
    s = state
    kind = s["kind"]
    if kind in ("product", "null", "rank"):
        return s["fn"](*s["args"])
    if kind == "packed_product":
        return device.matmul(s["A"], s["B"], s["m"], s["k"], s["n"])
    if kind == "chain":
        A = device.pack(s["A"], s["m"], s["k"])
        B = device.pack(s["B"], s["k"], s["n"])
        return device.unpack(device.matmul(A, B, s["m"], s["k"], s["n"]), s["m"], s["n"])
    if kind == "packed_rank":
        r = _eliminate(s, False)
        return r, s["piv"][:r]
    if kind == "packed_null":
        L = _lib.lib()
        r = _eliminate(s, True)
        n, f = s["n"], s["n"] - r
        zt = device.empty_packed(f, n)
        wsb = int(L.mela_null_workspace_size(n, r))
        ws = torch.empty(wsb, dtype=torch.uint8, device="cuda")
        _lib.check(L.mela_dev_null_basis(s["work"].data_ptr(), s["work"].shape[1], s["m"], n, r, s["piv"].data_ptr(),
                                         s["prow"].data_ptr(), zt.data_ptr(), zt.shape[1], ws.data_ptr(), wsb,
                                         torch.cuda.current_stream().cuda_stream))
        return r, s["piv"][:r], zt
    ranks, zt = s["plan"].run_logical(s["buf"], s["ranks"], s["zt"])
    return ranks, zt


# ------------------------------------------------------------------ work
def _elim_ops(m, n, r, rref):
    """Bit operations (AND + XOR) of an elimination with r pivots."""
    rows = m * r if rref else m * r - r * r / 2
    return 2.0 * rows * max(n - r / 2, 1)


def work(case):
    kind = case["kind"]
    m, n = case.get("m"), case.get("n")
    if kind in ("product", "chain"):
        esz = 8 if case["dtype"] == "double" else 1
        return dict(bytes=(m * case["k"] + case["k"] * n) * esz + m * n, flops=2.0 * m * n * case["k"])
    if kind == "packed_product":
        k = case["k"]
        return dict(bytes=(m * k + k * n + m * n) / 8, flops=2.0 * m * n * k)
    if kind in ("rank", "null"):
        esz = 8 if case["dtype"] == "double" else 1
        r = min(m, n)
        out = n * (n - r) if kind == "null" else 8
        return dict(bytes=m * n * esz + out, flops=_elim_ops(m, n, r, kind == "null"))
    if kind in ("packed_rank", "packed_null"):
        r = case["rank"]
        out = n * (n - r) / 8 if kind == "packed_null" else 8 * r
        return dict(bytes=m * n / 8 + out, flops=_elim_ops(m, n, r, kind == "packed_null"))
    lo, hi, c = case["lo"], case["hi"], case["count"]
    m2 = (hi ** 3 - lo ** 3) / (3.0 * max(hi - lo, 1))  # mean of m^2
    m3 = (hi ** 4 - lo ** 4) / (4.0 * max(hi - lo, 1))  # mean of m^3
    return dict(bytes=c * (2 * m2 + 2 * m2 / 8), flops=c * 3.0 * m3)


# ------------------------------------------------------------------ exact results
def _rref(bits):
    """Reduced row echelon form of a 0/1 matrix on the host: (rows, pivot columns)."""
    m, n = bits.shape
    P = np.packbits(bits.astype(np.uint8), axis=1, bitorder="little")
    pad = (-P.shape[1]) % 8
    P = np.ascontiguousarray(np.pad(P, ((0, 0), (0, pad)))).view(np.uint64)
    piv, r = [], 0
    for c in range(n):
        if r == m:
            break
        col = (P[:, c >> 6] >> np.uint64(c & 63)) & np.uint64(1)
        hit = np.flatnonzero(col[r:])
        if not len(hit):
            continue
        p = r + int(hit[0])
        if p != r:
            P[[r, p]] = P[[p, r]]
            col[p] = col[r]
        col[r] = 0
        P[np.flatnonzero(col)] ^= P[r]
        piv.append(c)
        r += 1
    rows = np.unpackbits(P[:r].view(np.uint8), axis=1, bitorder="little")[:, :n]
    return rows, np.array(piv, dtype=np.int64)


def _null(rows, piv, n):
    """n x nullity logical basis from an RREF."""
    free = np.setdiff1d(np.arange(n), piv)
    Z = np.zeros((n, len(free)), dtype=np.bool_, order="F")
    Z[free, np.arange(len(free))] = True
    Z[piv, :] = rows[:, free] != 0
    return Z


def _unpacked(P, n):
    return np.unpackbits(P.cpu().numpy().view(np.uint8), axis=1, bitorder="little")[:, :n]


def _packed(bits):
    """0/1 rows -> int64 words, as the packed device matrices hold them."""
    P = np.packbits(np.ascontiguousarray(bits, dtype=np.uint8), axis=1, bitorder="little")
    P = np.ascontiguousarray(np.pad(P, ((0, 0), (0, (-P.shape[1]) % 8))))
    return P.view(np.int64)


def _random_packed(seed, stream, m, n):
    """The words of device.rand_dense, on the host."""
    from mex_linear_algebra_b200 import gen
    return torch.from_numpy(gen.dense_packed(seed, stream, m, n).view(np.int64))


def _product(A, B):
    """A*B mod 2 of 0/1 host arrays by a 64-bit floating product."""
    return (A.astype(np.float64) @ B.astype(np.float64)).astype(np.int64) & 1


def exact(case, seed):
    kind = case["kind"]
    m, n = case.get("m"), case.get("n")
    if kind == "product":
        A, B = _host_inputs(case, seed)
        return np.asfortranarray(_product(A, B).astype(np.bool_))
    if kind in ("rank", "null"):
        (A,) = _host_inputs(case, seed)
        rows, piv = _rref(A != 0)
        return float(len(piv)) if kind == "rank" else _null(rows, piv, n)
    if kind == "packed_product" and m * case["k"] * n <= 1 << 36:
        A = _unpacked(_random_packed(seed, 0, m, case["k"]), case["k"])
        B = _unpacked(_random_packed(seed, 1, case["k"], n), n)
        return _packed(_product(A, B))
    if kind == "chain" and m * case["k"] * n <= 1 << 36:
        A, B = (x.cpu().numpy() for x in _device_arrays(case, seed))
        C = _product(A.reshape(case["k"], m).T, B.reshape(n, case["k"]).T)
        return C.T.astype(np.uint8).reshape(-1)
    if kind in ("packed_rank", "packed_null") and m <= 3000 and n <= 6000:
        r = case["rank"]
        A = _product(_unpacked(_random_packed(seed, 0, m, r), r), _unpacked(_random_packed(seed, 1, r, n), n))
        rows, piv = _rref(A)
        if kind == "packed_rank":
            return len(piv), piv
        return len(piv), piv, _packed(_null(rows, piv, n).T)
    return None  # the large sizes and the batch take too long on the host
