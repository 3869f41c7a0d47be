"""Products of matrices with few, heavy tiles: a cluster of 2 or 4 CTAs sums
each output tile of the N-form (distributed shared memory), and 2 or 4 CTAs
share the columns of each input tile of the T-form.  Sizes around the
limits (148 and 296 tiles, ragged tiles, runs shorter than a CTA's share),
every store format, against the oracle (arith/mulvec.hh:158-312 restated);
direct launches, plain launches and graph replays give identical bits, and
explicit launch shapes (whole tiles) agree to rounding."""
import numpy as np
import pytest

import hlr_b200 as hlr
import oracle

from conftest import built, relerr

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

# storage rounding of each format (VALR at eps = 1e-6 for mixed and BFP)
TOL = {"f64": 1e-13, "f32": 1e-6, "mixed": 2e-6, "bfp": 2e-5, "f16": 2e-3, "bf16": 2e-2}


@pytest.mark.parametrize("n,prec", [(1500, "f64"), (3001, "f64"), (6007, "f64"), (9001, "f64"), (3001, "mixed"),
                                    (6007, "bfp"), (6007, "f32"), (9001, "bf16"), (3001, "f16")])
@pytest.mark.parametrize("op", [0, 1])
def test_few_heavy_tiles(n, prec, op):
    hm = built(f"exp_{n}", lambda: hlr.build(hlr.Problem.exp3d(n)))
    M = hlr.upload(hm, precision=prec)
    xh = np.random.default_rng(n).standard_normal(n)
    y0 = np.random.default_rng(n + 1).standard_normal(n)
    x = torch.from_numpy(xh).cuda()

    def run(graph=False):
        y = torch.from_numpy(y0.copy()).cuda()
        if not graph:
            hlr.mul_vec(1.5, op, M, x, y)
        else:
            hlr.mul_vec(1.5, op, M, x, y)
            torch.cuda.synchronize()
            y.copy_(torch.from_numpy(y0))
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g):
                hlr.mul_vec(1.5, op, M, x, y)
            g.replay()
            torch.cuda.synchronize()
            del g
        torch.cuda.synchronize()
        return y.cpu().numpy()

    y = run()
    assert np.array_equal(run(), y) and np.array_equal(run(graph=True), y)
    M.set_tuning(overlap=0)
    assert np.array_equal(run(), y)
    M.set_tuning(overlap=1, nform_warps=4, ttform_warps=4)
    whole = run()
    M.set_tuning(nform_warps=16, ttform_warps=16)
    assert relerr(run() - y0, whole - y0) <= 1e-14
    assert relerr(y - y0, whole - y0) <= 1e-14
    yo = np.zeros(n)
    oracle.hmvm_seq(hm.h_desc(), 1.5, op, xh, yo)
    assert relerr(y - y0, yo) <= TOL[prec]
    assert M.device_error() == 0
    M.free()


@pytest.mark.parametrize("n,prec,nrhs", [(3001, "f64", 5), (3001, "f64", 16), (6007, "f64", 23), (9001, "f64", 32),
                                         (3001, "mixed", 8), (6007, "bfp", 3), (6007, "f32", 8), (9001, "bf16", 7),
                                         (3001, "f16", 8), (6007, "mixed", 19)])
@pytest.mark.parametrize("op", [0, 1])
def test_few_heavy_tiles_several_vectors(n, prec, nrhs, op):
    hm = built(f"exp_{n}", lambda: hlr.build(hlr.Problem.exp3d(n)))
    M = hlr.upload(hm, precision=prec, max_nrhs=nrhs)
    rng = np.random.default_rng(n + nrhs)
    X, Y0 = rng.standard_normal((nrhs, n)), rng.standard_normal((nrhs, n))
    Xd = torch.from_numpy(X).cuda().T
    ys = []
    for _ in range(2):
        Yd = torch.from_numpy(Y0.copy()).cuda().T
        hlr.mul_vec(-0.75, op, M, Xd, Yd)
        torch.cuda.synchronize()
        ys.append(Yd.T.cpu().numpy() - Y0)
    assert np.array_equal(ys[0], ys[1])
    for j in range(0, nrhs, 4):
        yo = np.zeros(n)
        oracle.hmvm_seq(hm.h_desc(), -0.75, op, X[j], yo)
        assert relerr(ys[0][j], yo) <= TOL[prec], j
    assert M.device_error() == 0
    M.free()
