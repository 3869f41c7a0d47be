"""FP64 products of up to 32 vectors per pass of the matrix (two to four
8-vector tiles, kernels_dw.cuh) against the oracle: vector counts at the
edges of tiles and passes, tiles of every height, ops N and C of H, uniform-H
and H^2 matrices (the transposed couplings are unit T-forms)."""
import numpy as np
import pytest

import hlr_b200 as hlr
import oracle

from conftest import built, relerr

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

TOL = 1e-13   # the FP64 parity bound: sums of at most a few thousand products of order one

CASES = {
    # 3000 points: leaf clusters of 46 and 47 rows; leaf 20 and 12: tiles of 1 and 2 row blocks of 16
    "h": ("h", lambda: hlr.build(hlr.Problem.exp3d(3000))),
    "h_leaf20": ("h", lambda: hlr.build(hlr.Problem.log1d(1700, leaf_size=20))),
    "h_leaf12": ("h", lambda: hlr.build(hlr.Problem.log1d(901, leaf_size=12))),
    "uniform": ("uniform", lambda: hlr.build(hlr.Problem.laplace_sphere(refine=4, uniform=True))),
    "h2": ("h2", lambda: hlr.build(hlr.Problem.laplace_sphere(refine=4, nested=True))),
}


def _oracle(hm, kind, alpha, op, x, y0):
    y = y0.copy()
    if kind == "h2":
        assert oracle.h2_mvm(hm.h2_desc(), alpha, op, x, y) == 0
    elif kind == "uniform":
        assert oracle.uniform_mvm(hm.uniform_desc(), alpha, op, x, y) == 0
    else:
        oracle.hmvm_seq(hm.h_desc(), alpha, op, x, y)
    return y


@pytest.mark.parametrize("op", [0, 2])
@pytest.mark.parametrize("name", sorted(CASES))
def test_block_products_match_the_oracle(name, op):
    kind, make = CASES[name]
    hm = built("dw_" + name, make)
    M = hlr.upload(hm, uniform=kind == "uniform", h2=kind == "h2", max_nrhs=32)
    W = hlr.Workspace(M, max_nrhs=16)
    rng = np.random.default_rng(7)
    kmax, pad = 41, 3
    X = rng.standard_normal((kmax, hm.n + pad))
    Y0 = rng.standard_normal((kmax, hm.n + pad))
    ref = np.stack([_oracle(hm, kind, -0.75, op, X[j, :hm.n].copy(), Y0[j, :hm.n].copy()) for j in range(kmax)])
    Xd = torch.from_numpy(X).cuda().T[:hm.n]          # column-major, ld = n + 3
    for nrhs in (2, 8, 9, 15, 16, 17, 23, 24, 25, 31, 32, 33, 41):
        for ws in (None, W):                          # the workspace holds two tiles: more passes
            Yd = torch.from_numpy(Y0.copy()).cuda()
            hlr.mul_vec(-0.75, op, M, Xd[:, :nrhs], Yd.T[:hm.n, :nrhs], workspace=ws)
            torch.cuda.synchronize()
            Y = Yd.cpu().numpy()
            for j in range(nrhs):
                assert relerr(Y[j, :hm.n] - Y0[j, :hm.n], ref[j] - Y0[j, :hm.n]) <= TOL, (nrhs, j)
            assert np.array_equal(Y[nrhs:], Y0[nrhs:]) and np.array_equal(Y[:, hm.n:], Y0[:, hm.n:])
    assert M.device_error() == 0
    W.free()
    M.free()
