"""Op T / C of one vector: the tile T-form of D^T x runs on the side stream (or
from the side queue of a one-launch product) into partial sums of its own, and
its finish adds to y after the pass before it (tbb/detail/arith.hh:95-124 adds
every block of a row into y).  The sums and their order on y do not depend on
where it runs: separate and one launch, graph replays, a caller's workspace on
another stream, a workspace made for a smaller matrix and the no-alloc entry
point give identical bits, and they match the oracle."""
import ctypes as C

import numpy as np
import pytest

import hlr_b200 as hlr
import oracle
from hlr_b200 import _capi

from conftest import built, relerr

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

CASES = {   # one launch when eager; 512 tiles and tree sweeps: a launch per pass
    "h": lambda: built("c2_small", lambda: hlr.build(hlr.Problem.exp3d(4096))),
    "h_ragged": lambda: built("exp_20011", lambda: hlr.build(hlr.Problem.exp3d(20011))),
    "uniform": lambda: built("c3_small", lambda: hlr.build(hlr.Problem.laplace_sphere(refine=4, uniform=True))),
    "h2": lambda: built("sphere5_h2", lambda: hlr.build(hlr.Problem.laplace_sphere(refine=5, nested=True))),
}


@pytest.mark.parametrize("kind,prec", [(k, "f64") for k in sorted(CASES)] + [("h", "mixed"), ("h_ragged", "bfp")])
def test_every_path_gives_the_same_bits(kind, prec):
    hm = CASES[kind]()
    M = hlr.upload(hm, precision=prec, uniform=(kind == "uniform"), h2=(kind == "h2"))
    op = 1 if kind.startswith("h") and kind != "h2" else 2
    x = torch.from_numpy(np.random.default_rng(5).standard_normal(hm.n)).cuda()
    alphas = [0.75 + k for k in range(6)]

    def chain(overlap=1, graph=False, workspace=None, stream=None, noalloc=False):
        M.set_tuning(overlap=overlap)
        y = torch.zeros_like(x)
        st = stream or torch.cuda.current_stream()
        st.wait_stream(torch.cuda.current_stream())

        def product(a):
            if noalloc:
                L = _capi.lib()
                assert L.hlrc_mvm_noalloc(M.handle, a, op, C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr()),
                                          C.c_void_p(st.cuda_stream)) == 0, L.hlrc_last_error().decode()
            else:
                hlr.mul_vec(a, op, M, x, y, workspace=workspace)

        with torch.cuda.stream(st):
            if graph:
                product(1.0)
                torch.cuda.synchronize()
                y.zero_()
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g):
                    for a in alphas:
                        product(a)
                g.replay()
                torch.cuda.synchronize()
                del g
            else:
                for a in alphas:
                    product(a)
        torch.cuda.synchronize()
        return y.cpu().numpy()

    first = chain()
    W, other = hlr.Workspace(M), torch.cuda.Stream()
    for kw in (dict(overlap=0), dict(graph=True), dict(overlap=0, graph=True), dict(workspace=W, stream=other),
               dict(workspace=W, stream=other, graph=True)):
        assert np.array_equal(chain(**kw), first), kw
    if M.info["scratch_bytes"] <= 8 << 20:
        assert np.array_equal(chain(noalloc=True), first)
    yo = np.zeros(hm.n)
    xh = x.cpu().numpy()
    if kind == "h2":
        assert oracle.h2_mvm(hm.h2_desc(), sum(alphas), op, xh, yo) == 0
    elif kind == "uniform":
        assert oracle.uniform_mvm(hm.uniform_desc(), sum(alphas), op, xh, yo) == 0
    else:
        oracle.hmvm_seq(hm.h_desc(), sum(alphas), op, xh, yo)
    assert relerr(first, yo) <= {"f64": 1e-13, "mixed": 2e-6, "bfp": 2e-5}[prec]
    assert M.device_error() == 0
    W.free()
    M.free()
