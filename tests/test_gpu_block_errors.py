"""Products of several vectors are no less exact than the products they replace:
the error against long double (64 bits of mantissa) of a block of 16, 24 or 32
vectors is at most that of the 8-vector kernels, and the error of a block adjoint
of a uniform-H or H^2 matrix about that of one vector at a time.

Bounds.  Rounding errors of a sum of terms of one size add up as the square root of
the number of roundings at the size of the sum.  Blocks against 8 vectors: not more
roundings, and the norm over 2 x 8192 entries varies by some percent: 1.1.  Block
adjoints: a column's sum over a tile takes 8 roundings within groups of rows and 8
to 12 between them where the one-vector kernel takes about 6 to 8 (2 rows per lane,
then a tree over lanes): sqrt(20 / 14) = 1.2, and 1.3 with the variation."""
import numpy as np
import pytest

import hlr_b200 as hlr

from conftest import built

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

LD = np.longdouble


def _mat(ptr, rows, cols, ld):
    if rows == 0 or cols == 0:
        return np.zeros((rows, cols), dtype=LD)
    a = np.ctypeslib.as_array(ptr, shape=(ld * (cols - 1) + rows,))
    return np.lib.stride_tricks.as_strided(a, (rows, cols), (8, 8 * ld)).astype(LD)


def _rows_cols(b, normal):
    r, c = slice(b.row0, b.row0 + b.nrows), slice(b.col0, b.col0 + b.ncols)
    return (r, c) if normal else (c, r)


def _h(d, normal, x):
    y = np.zeros_like(x)
    for i in range(d.nblocks):
        b = d.blocks[i]
        out, src = _rows_cols(b, normal)
        if b.kind == hlr.LEAF_DENSE:
            D = _mat(b.D, b.nrows, b.ncols, b.ldd)
            y[out] += (D if normal else D.T) @ x[src]
        elif b.rank:
            U, V = _mat(b.U, b.nrows, b.rank, b.ldu), _mat(b.V, b.ncols, b.rank, b.ldv)
            y[out] += U @ (V.T @ x[src]) if normal else V @ (U.T @ x[src])
    return y


def _uniform(d, normal, x):
    rows, cols = ([p[i] for i in range(k)] for p, k in ((d.row_bases, d.nrow_bases), (d.col_bases, d.ncol_bases)))
    src, dst = (cols, rows) if normal else (rows, cols)
    ux = [_mat(b.V, b.size, b.rank, b.ldv).T @ x[b.ofs:b.ofs + b.size] for b in src]
    uy = [np.zeros((b.rank, x.shape[1]), dtype=LD) for b in dst]
    y = np.zeros_like(x)
    for i in range(d.nblocks):
        b = d.blocks[i]
        if b.kind == hlr.LEAF_DENSE:
            out, s = _rows_cols(b, normal)
            D = _mat(b.D, b.nrows, b.ncols, b.ldd)
            y[out] += (D if normal else D.T) @ x[s]
        else:
            S = _mat(b.S, rows[b.row_basis].rank, cols[b.col_basis].rank, b.lds)
            if normal:
                uy[b.row_basis] += S @ ux[b.col_basis]
            else:
                uy[b.col_basis] += S.T @ ux[b.row_basis]
    for b, u in zip(dst, uy):
        y[b.ofs:b.ofs + b.size] += _mat(b.V, b.size, b.rank, b.ldv) @ u
    return y


def _errors(hm, kind, op, counts, max_nrhs, loop=False):
    """{vectors: relative error of the first two columns of a product of that many}"""
    M = hlr.upload(hm, uniform=kind == "uniform", max_nrhs=max_nrhs)
    if loop:
        M.set_tuning(mr_min_nrhs=1_000_000)
    g = torch.Generator(device="cuda").manual_seed(9)
    X = torch.randn((max(counts), hm.n), dtype=torch.float64, device="cuda", generator=g).T
    x = X[:, :2].cpu().numpy().astype(LD)
    ref = _uniform(hm.uniform_desc(), op == 0, x) if kind == "uniform" else _h(hm.h_desc(), op == 0, x)
    out = {}
    for k in counts:
        Y = torch.zeros((k, hm.n), dtype=torch.float64, device="cuda").T
        hlr.mul_vec(1.0, op, M, X[:, :k], Y)
        d = (Y[:, :2].cpu().numpy().astype(LD) - ref).astype(np.float64)
        out[k] = float(np.linalg.norm(d) / np.linalg.norm(ref.astype(np.float64)))
    M.free()
    return out


@pytest.mark.parametrize("op", [0, 2])
def test_blocks_as_exact_as_eight_vectors(op):
    hm = built("c1", lambda: hlr.build(hlr.Problem.log1d(8192)))
    eight = _errors(hm, "h", op, (8,), 8)[8]
    for k, e in _errors(hm, "h", op, (16, 24, 32), 32).items():
        assert e <= 1.1 * eight, (k, e, eight)


def test_uniform_blocks_as_exact_as_eight_vectors():
    hm = built("c3_small", lambda: hlr.build(hlr.Problem.laplace_sphere(refine=4, uniform=True)))
    eight = _errors(hm, "uniform", 0, (8,), 8)[8]
    for k, e in _errors(hm, "uniform", 0, (16, 24, 32), 32).items():
        assert e <= 1.1 * eight, (k, e, eight)


def test_uniform_block_adjoint_about_as_exact_as_one_vector():
    hm = built("c3_small", lambda: hlr.build(hlr.Problem.laplace_sphere(refine=4, uniform=True)))
    one = _errors(hm, "uniform", 2, (2,), 2, loop=True)[2]
    for k, e in _errors(hm, "uniform", 2, (2, 8, 16, 24, 32), 32).items():
        assert e <= 1.3 * one, (k, e, one)
