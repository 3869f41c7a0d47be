"""One-vector FP64 products run as one launch (kernels_flow.cuh) against the
same passes as separate launches (per-pass profiling keeps those) and the
oracle; a wait that runs out is reported and the next product is exact."""
import numpy as np
import pytest

import hlr_b200 as hlr
import oracle
from hlr_b200 import _capi

from conftest import built, relerr

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

CASES = {
    "h_one_tile": ("h", lambda: hlr.build(hlr.Problem.log1d(40))),          # one dense leaf: no chain to wait for
    "h_log": ("h", lambda: hlr.build(hlr.Problem.log1d(4099))),
    "h_exp": ("h", lambda: hlr.build(hlr.Problem.exp3d(3000, leaf_size=48))),
    "uniform": ("uniform", lambda: hlr.build(hlr.Problem.laplace_sphere(refine=4, uniform=True))),
    "h2": ("h2", lambda: hlr.build(hlr.Problem.log1d(300, nested=True))),   # too few clusters for tree sweeps
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


@pytest.mark.parametrize("near_field", [1, 2])
@pytest.mark.parametrize("name", sorted(CASES))
def test_one_launch_matches_separate_passes(name, near_field):
    kind, make = CASES[name]
    hm = built("flow_" + name, make)
    M = hlr.upload(hm, uniform=kind == "uniform", h2=kind == "h2", plan={"near_field": near_field})
    rng = np.random.default_rng(12)
    for op in (0, 2) if kind != "h" else (0, 1, 2):
        xh, y0 = rng.standard_normal(hm.n), rng.standard_normal(hm.n)
        x = torch.from_numpy(xh).cuda()
        ys = []
        for separate in (True, False):
            y = torch.from_numpy(y0.copy()).cuda()
            M.set_profiling(separate)
            n0 = M.launch_count()
            for alpha in (0.5, -1.75, 3.0):        # a chain of products on one workspace
                hlr.mul_vec(alpha, op, M, x, y)
            torch.cuda.synchronize()
            # heavy tiles keep separate launches, several CTAs a tile
            assert separate or name == "h_exp" or M.launch_count() - n0 == 3
            M.last_profile()
            ys.append(y.cpu().numpy() - y0)
        M.set_profiling(False)
        yo = _oracle(hm, kind, 1.75, op, xh, np.zeros(hm.n))
        assert np.array_equal(ys[1], ys[0]), op        # the same sums in the same order
        assert relerr(ys[1], yo) <= 1e-13, op
    assert M.device_error() == 0
    M.free()


def test_one_launch_wait_runs_out_and_recovers():
    hm = built("flow_h_log", CASES["h_log"][1])
    M = hlr.upload(hm)
    L = _capi.lib()
    x = torch.from_numpy(np.random.default_rng(1).standard_normal(hm.n)).cuda()
    ref = torch.zeros_like(x)
    hlr.mul_vec(1.0, 0, M, x, ref)
    assert L.hlrc_debug_waits(M.handle, 20_000_000, 1) == 0      # 20 ms; one item is never counted
    y = torch.zeros_like(x)
    hlr.mul_vec(1.0, 0, M, x, y)
    torch.cuda.synchronize()
    assert M.device_error() & 1
    assert L.hlrc_debug_waits(M.handle, 0, 0) == 0
    y.zero_()
    hlr.mul_vec(1.0, 0, M, x, y)
    torch.cuda.synchronize()
    assert M.device_error() == 0
    assert torch.equal(y, ref)
    M.free()
