"""Products that programs using this library run, for timing and for checking.

A case is a matrix, a store precision, an op and a number of vectors; one pass
is one call of ``mul_vec`` (``uniform.mul_vec``, ``h2.mul_vec``), y += alpha op(M) X.
The matrices are those of the library's tests and benchmark: the 1D log kernel,
the 3D exponential covariance and the single-layer potential on a sphere mesh,
leaf 64, eta 2, accuracy 1e-6 where a case names none.  Point sets and vectors follow from the seed; the
sphere mesh is fixed, so only the vectors do there.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import hlr_b200 as hlr

ALPHA = 2.0
OPS = {"N": hlr.apply_normal, "T": hlr.apply_transposed, "C": hlr.apply_adjoint}
EXACT_MAX_BYTES = 5e9   # exact() walks the leaves in numpy: up to this much leaf data


def listed():
    return [
        # one product with a small matrix: the inner step of an iterative solver, bound by latency
        {"name": "log_8192_f64", "form": "h", "kernel": "log", "n": 8192, "store": "f64", "op": "N", "nrhs": 1},
        # the product of the headline benchmark: a large covariance matrix, one vector
        {"name": "exp_131072_f64", "form": "h", "kernel": "exp", "n": 131072, "store": "f64", "op": "N", "nrhs": 1},
        # block adjoint product (range finders, block Krylov methods), leaf clusters of uneven size
        {"name": "exp_50021_f64_adj_x16", "form": "h", "kernel": "exp", "n": 50021, "store": "f64", "op": "C",
         "nrhs": 16},
        # uniform-H matrix of a boundary integral operator: one vector in a solver, and a block of load cases
        {"name": "sphere_uniform_f64", "form": "uniform", "refine": 6, "eps": 1e-6, "store": "f64", "op": "N",
         "nrhs": 1},
        {"name": "sphere_uniform_f64_x32", "form": "uniform", "refine": 6, "eps": 1e-6, "store": "f64", "op": "N",
         "nrhs": 32},
        # the same operator with nested bases
        {"name": "sphere_h2_f64", "form": "h2", "refine": 6, "eps": 1e-6, "store": "f64", "op": "N", "nrhs": 1},
        # compressed stores with one vector: the inner operator of iterative refinement
        {"name": "exp_32768_mixed", "form": "h", "kernel": "exp", "n": 32768, "store": "mixed", "op": "N", "nrhs": 1},
        {"name": "exp_20011_bfp_adj", "form": "h", "kernel": "exp", "n": 20011, "store": "bfp", "op": "C", "nrhs": 1},
        # 16-bit stores with many vectors: sampling and stochastic trace estimates
        {"name": "exp_32768_f16_x64", "form": "h", "kernel": "exp", "n": 32768, "store": "f16", "op": "N", "nrhs": 64},
        {"name": "exp_20011_bf16_x40", "form": "h", "kernel": "exp", "n": 20011, "store": "bf16", "op": "N",
         "nrhs": 40},
        # many matrices of different sizes in one handle, 8 vectors each: the batched inner solver
        {"name": "batch_mixed_x8", "form": "batch", "members": 6, "n_min": 2048, "n_max": 16384, "store": "mixed",
         "op": "N", "nrhs": 8},
        # vectors in host memory: the drop-in call of an unchanged host program
        {"name": "log_100003_f64_host", "form": "host", "kernel": "log", "n": 100003, "store": "f64", "op": "N",
         "nrhs": 1},
    ]


def _log_n(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    form = rng.choice(["h", "h", "h", "uniform", "h2", "store", "store", "batch", "host"])
    one = rng.random() < 0.5
    if form in ("h", "host"):
        kernel = rng.choice(["log", "exp"])
        n = _log_n(rng, 2000, 200000) if kernel == "log" else _log_n(rng, 3000, 65536)
        nrhs = 1 if one or form == "host" else rng.randint(2, 32)
        return {"form": form, "kernel": kernel, "n": n, "store": "f64", "op": rng.choice(["N", "N", "T", "C"]),
                "nrhs": nrhs}
    if form in ("uniform", "h2"):
        return {"form": form, "refine": rng.choice([4, 5, 6]), "eps": float(f"{10 ** rng.uniform(-6.5, -4):.1e}"),
                "store": "f64", "op": rng.choice(["N", "N", "C"]), "nrhs": 1 if one else rng.randint(2, 32)}
    if form == "store":
        return {"form": "h", "kernel": "exp", "n": _log_n(rng, 3000, 32768),
                "store": rng.choice(["mixed", "bfp", "f16", "bf16", "f32"]), "op": rng.choice(["N", "N", "C"]),
                "nrhs": 1 if one else rng.randint(2, 64)}
    return {"form": "batch", "members": rng.randint(3, 10), "n_min": _log_n(rng, 1000, 2000),
            "n_max": _log_n(rng, 4000, 12000), "store": rng.choice(["mixed", "f64"]), "op": "N",
            "nrhs": rng.randint(1, 8)}


@functools.lru_cache(maxsize=3)
def _sphere(refine, eps):
    """The sphere operator with shared and with nested bases: one geometry, built once by a program."""
    return hlr.build(hlr.Problem.laplace_sphere(refine=refine, eps=eps, uniform=True, nested=True))


def _member_sizes(case):
    m, lo, hi = case["members"], case["n_min"], case["n_max"]
    return [int(lo * (hi / lo) ** ((i + 0.5) / m)) | 1 for i in range(m)]


def _build(case, seed):
    """The host descriptions of the case's matrices (a list: one, or the members of a batch)."""
    if "refine" in case:
        return [_sphere(case["refine"], case["eps"])]
    if case["form"] == "batch":
        r = np.random.default_rng(seed)
        return [hlr.build(hlr.Problem.exp3d(n, ell=float(r.uniform(0.05, 0.2)), seed=1000 * seed + i, on_device=True))
                for i, n in enumerate(_member_sizes(case))]
    make = hlr.Problem.log1d if case["kernel"] == "log" else hlr.Problem.exp3d
    return [hlr.build(make(case["n"], seed=seed + 1, on_device=True))]


def _pad(case):
    return max(_member_sizes(case)) + 63 & ~63


def _length(case):
    if "refine" in case:
        return 8 * 4 ** case["refine"]
    return _pad(case) * case["members"] if case["form"] == "batch" else case["n"]


def _vectors(case, seed):
    """X and the starting Y, (n,) or column-major (n, nrhs), on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n, k = _length(case), case["nrhs"]
    x, y = (torch.randn((k, n), dtype=torch.float64, device="cuda", generator=g) for _ in range(2))
    return (x[0], y[0]) if k == 1 else (x.T, y.T)


def prepare(case, seed):
    hms = _build(case, seed)
    kw = {"precision": case["store"], "max_nrhs": case["nrhs"]}
    if case["form"] == "batch":
        M = hlr.upload_batch(hms, pad_to=_pad(case), **kw)
    elif case["form"] == "h2":
        M = hlr.upload(hms[0], h2=True, **kw)
    else:
        M = hlr.upload(hms[0], uniform=case["form"] == "uniform", **kw)
    x, y = _vectors(case, seed)
    if case["form"] == "host":
        x, y = x.cpu().numpy(), y.cpu().numpy()
    mul = {"uniform": hlr.uniform.mul_vec, "h2": hlr.h2.mul_vec}.get(case["form"], hlr.mul_vec)
    return {"M": M, "x": x, "y": y, "op": OPS[case["op"]], "mul_vec": mul}


def run(state):
    state["mul_vec"](ALPHA, state["op"], state["M"], state["x"], state["y"])
    return state["y"]


def work(case):
    """Stored matrix data read once, X read, Y read and written; two flops per stored entry and vector."""
    hms = _build(case, 1)
    k, n = case["nrhs"], _length(case)
    if "refine" in case:
        stored = hlr.plan_info(hms[0], uniform=case["form"] == "uniform", h2=case["form"] == "h2")["matrix_bytes"]
        entries = stored / 8
    else:
        entries = sum(h.bytes for h in hms) / 8
        stored = (8 * entries if case["store"] == "f64" else
                  sum(hlr.plan_info(h, precision=case["store"])["matrix_bytes"] for h in hms))
    return {"bytes": stored + 24 * n * k, "flops": 2 * entries * k}


def _mat(ptr, rows, cols, ld):
    """A column-major rows x cols array at a descriptor's pointer."""
    if rows == 0 or cols == 0:
        return np.zeros((rows, cols))
    a = np.ctypeslib.as_array(ptr, shape=(ld * (cols - 1) + rows,))
    return np.lib.stride_tricks.as_strided(a, (rows, cols), (8, 8 * ld))


def _near(b, normal, x, y):
    D = _mat(b.D, b.nrows, b.ncols, b.ldd)
    r, c = slice(b.row0, b.row0 + b.nrows), slice(b.col0, b.col0 + b.ncols)
    if normal:
        y[r] += D @ x[c]
    else:
        y[c] += D.T @ x[r]


def _exact_h(d, normal, x, y):
    for i in range(d.nblocks):
        b = d.blocks[i]
        if b.kind == hlr.LEAF_DENSE:
            _near(b, normal, x, y)
        elif b.rank:
            U, V = _mat(b.U, b.nrows, b.rank, b.ldu), _mat(b.V, b.ncols, b.rank, b.ldv)
            r, c = slice(b.row0, b.row0 + b.nrows), slice(b.col0, b.col0 + b.ncols)
            if normal:
                y[r] += U @ (V.T @ x[c])
            else:
                y[c] += V @ (U.T @ x[r])


def _couplings(d, rows, cols, normal, x, y, ux, uy):
    """uy += S ux (S^T for the adjoint) over the admissible blocks, and the near field into y."""
    for i in range(d.nblocks):
        b = d.blocks[i]
        if b.kind == hlr.LEAF_DENSE:
            _near(b, normal, x, y)
            continue
        S = _mat(b.S, rows[b.row_basis].rank, cols[b.col_basis].rank, b.lds)
        if normal:
            uy[b.row_basis] += S @ ux[b.col_basis]
        else:
            uy[b.col_basis] += S.T @ ux[b.row_basis]


def _exact_uniform(d, normal, x, y):
    rows, cols = ([p[i] for i in range(k)] for p, k in ((d.row_bases, d.nrow_bases), (d.col_bases, d.ncol_bases)))
    src, dst = (cols, rows) if normal else (rows, cols)
    ux = [_mat(b.V, b.size, b.rank, b.ldv).T @ x[b.ofs:b.ofs + b.size] for b in src]
    uy = [np.zeros((b.rank, x.shape[1])) for b in dst]
    _couplings(d, rows, cols, normal, x, y, ux, uy)
    for b, u in zip(dst, uy):
        y[b.ofs:b.ofs + b.size] += _mat(b.V, b.size, b.rank, b.ldv) @ u


def _exact_h2(d, normal, x, y):
    rows, cols = ([p[i] for i in range(k)]
                  for p, k in ((d.row_clusters, d.nrow_clusters), (d.col_clusters, d.ncol_clusters)))
    src, dst = (cols, rows) if normal else (rows, cols)
    ux = [np.zeros((c.rank, x.shape[1])) for c in src]
    uy = [np.zeros((c.rank, x.shape[1])) for c in dst]

    def sons(cs, i):
        return [s for s in cs[i].son if s >= 0]

    def up(i):
        c = src[i]
        if not sons(src, i):
            ux[i] += _mat(c.V, c.size, c.rank, c.ldv).T @ x[c.ofs:c.ofs + c.size]
        for s in sons(src, i):
            up(s)
            ux[i] += _mat(src[s].E, src[s].rank, c.rank, src[s].lde).T @ ux[s]

    def down(i):
        c = dst[i]
        if not sons(dst, i):
            y[c.ofs:c.ofs + c.size] += _mat(c.V, c.size, c.rank, c.ldv) @ uy[i]
        for s in sons(dst, i):
            uy[s] += _mat(dst[s].E, dst[s].rank, c.rank, dst[s].lde) @ uy[i]
            down(s)

    up(0)
    _couplings(d, rows, cols, normal, x, y, ux, uy)
    down(0)


def exact(case, seed):
    """y + alpha op(M) X in 64 bits from the leaves, for every store (a store's rounding is its error)."""
    hms = _build(case, seed)
    if sum(h.bytes for h in hms) > EXACT_MAX_BYTES and "refine" not in case:
        return None
    normal = case["op"] == "N"
    x, y0 = (v.cpu().numpy().reshape(_length(case), -1) for v in _vectors(case, seed))
    z = np.zeros_like(y0)
    if case["form"] == "uniform":
        _exact_uniform(hms[0].uniform_desc(), normal, x, z)
    elif case["form"] == "h2":
        _exact_h2(hms[0].h2_desc(), normal, x, z)
    else:
        step = _pad(case) if case["form"] == "batch" else 0
        for i, h in enumerate(hms):
            part = slice(i * step, i * step + h.n)
            _exact_h(h.fetch().h_desc(), normal, x[part], z[part])
    y = y0 + ALPHA * z
    return y[:, 0] if case["nrhs"] == 1 else y
