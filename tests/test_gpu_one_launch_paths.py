"""Which products run as one launch, by matrix and op: small FP64 products of the
log kernel, of small dense-leaf 3D matrices and of small spheres do; matrices whose
chain holds much in heavy tiles, tree sweeps and large ones do not (nor op T / C that
is a T-form and its finish only), nor do products of several vectors, of other stores, or under capture.  Where it is one launch the
bits are those of separate passes, of graph replays, of a caller's workspace on
another stream and of the no-alloc entry point, op T / C with D^T x in the side
queue included."""
import ctypes as C

import numpy as np
import pytest

import hlr_b200 as hlr
import oracle
from hlr_b200 import _capi

from conftest import built, relerr

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

ONE = {
    "log_4099": ("h", lambda: hlr.build(hlr.Problem.log1d(4099))),
    "log_9001": ("h", lambda: hlr.build(hlr.Problem.log1d(9001))),       # 256 tiles
    "exp_1100": ("h", lambda: hlr.build(hlr.Problem.exp3d(1100))),       # mostly dense leaves, ragged
    "sphere3_h": ("h", lambda: hlr.build(hlr.Problem.laplace_sphere(refine=3))),   # dense leaves only: op N only
    "c3_small": ("uniform", lambda: hlr.build(hlr.Problem.laplace_sphere(refine=4, uniform=True))),
}
MANY = {
    "c2_small": ("h", lambda: hlr.build(hlr.Problem.exp3d(4096))),       # heavy tiles: several CTAs a tile
    "exp_20011": ("h", lambda: hlr.build(hlr.Problem.exp3d(20011))),     # 512 tiles
    "sphere5_h2": ("h2", lambda: hlr.build(hlr.Problem.laplace_sphere(refine=5, nested=True))),   # tree sweeps
}


def _upload(hm, kind, **kw):
    return hlr.upload(hm, uniform=kind == "uniform", h2=kind == "h2", **kw)


def _ops(kind):
    return (0, 1, 2) if kind == "h" else (0, 2)


@pytest.mark.parametrize("name", sorted(ONE))
def test_one_launch_and_its_bits(name):
    kind, make = ONE[name]
    hm = built(name, make)
    M, L = _upload(hm, kind), _capi.lib()
    W, other = hlr.Workspace(M), torch.cuda.Stream()
    rng = np.random.default_rng(6)
    xh, y0 = rng.standard_normal(hm.n), rng.standard_normal(hm.n)
    x = torch.from_numpy(xh).cuda()
    for op in _ops(kind):
        def run(how):
            y = torch.from_numpy(y0.copy()).cuda()
            torch.cuda.synchronize()
            n0 = M.launch_count()
            if how == "noalloc":
                assert L.hlrc_mvm_noalloc(M.handle, 1.5, op, C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr()),
                                          C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
            elif how == "workspace":
                with torch.cuda.stream(other):
                    hlr.mul_vec(1.5, op, M, x, y, workspace=W)
            elif how == "graph":
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g):
                    hlr.mul_vec(1.5, op, M, x, y)
                g.replay()
                torch.cuda.synchronize()
                del g
            else:
                M.set_profiling(how == "separate")
                hlr.mul_vec(1.5, op, M, x, y)
                torch.cuda.synchronize()
                M.last_profile()
                M.set_profiling(False)
            torch.cuda.synchronize()
            return y.cpu().numpy(), M.launch_count() - n0

        flows = op == 0 or name != "sphere3_h"
        first, n = run("plain")
        assert n == (1 if flows else M.info["launches"][op]), op
        for how, one in (("separate", False), ("workspace", True), ("noalloc", True), ("graph", False)):
            y, n = run(how)
            assert np.array_equal(y, first), (op, how)
            assert n == (1 if one and flows else M.info["launches"][op]), (op, how)
        ref = np.zeros(hm.n)
        if kind == "uniform":
            assert oracle.uniform_mvm(hm.uniform_desc(), 1.5, op, xh, ref) == 0
        else:
            oracle.hmvm_seq(hm.h_desc(), 1.5, op, xh, ref)
        assert relerr(first - y0, ref) <= 1e-13, op
    assert M.device_error() == 0
    W.free()
    M.free()


@pytest.mark.parametrize("name", sorted(MANY))
def test_separate_launches(name):
    kind, make = MANY[name]
    hm = built(name, make)
    M = _upload(hm, kind)
    x = torch.ones(hm.n, dtype=torch.float64, device="cuda")
    y = torch.zeros_like(x)
    for op in _ops(kind):
        n0 = M.launch_count()
        hlr.mul_vec(1.0, op, M, x, y)
        assert M.launch_count() - n0 > 1, op
    M.free()


def test_other_stores_and_blocks_are_separate():
    hm = built("log_4099", ONE["log_4099"][1])
    for kw, k in ((dict(precision="mixed"), 1), (dict(precision="bfp"), 1), (dict(max_nrhs=4), 4)):
        M = hlr.upload(hm, **kw)
        X = torch.ones((k, hm.n), dtype=torch.float64, device="cuda").T
        Y = torch.zeros((k, hm.n), dtype=torch.float64, device="cuda").T
        n0 = M.launch_count()
        hlr.mul_vec(1.0, 0, M, X if k > 1 else X[:, 0], Y if k > 1 else Y[:, 0])
        assert M.launch_count() - n0 > 1
        M.free()
