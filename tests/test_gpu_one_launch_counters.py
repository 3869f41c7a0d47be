"""The counters of one-launch products (kernels_flow.cuh) carry the number of
the product that uses them, so the state an earlier product leaves there does
not matter: after products that gave up half way, the next ones on the same
handle, on the same workspace and on the static scratch of the no-alloc entry
point, which all handles share, equal the reference bits."""
import ctypes as C

import numpy as np
import pytest

import hlr_b200 as hlr
import oracle
from hlr_b200 import _capi

from conftest import built, relerr

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _noalloc(M, a, op, x, y):
    L = _capi.lib()
    assert L.hlrc_mvm_noalloc(M.handle, a, op, C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr()),
                              C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0


@pytest.mark.parametrize("entry", ["handle", "workspace", "noalloc"])
def test_products_after_one_that_gave_up(entry):
    hms = [built("log_4099", lambda: hlr.build(hlr.Problem.log1d(4099))),
           built("log_700", lambda: hlr.build(hlr.Problem.log1d(700))),
           built("c3_small", lambda: hlr.build(hlr.Problem.laplace_sphere(refine=4, uniform=True)))]
    Ms = [hlr.upload(hm, uniform=i == 2) for i, hm in enumerate(hms)]
    W = hlr.Workspace(Ms[2]) if entry == "workspace" else None
    rng = np.random.default_rng(2)
    xs = [torch.from_numpy(rng.standard_normal(hm.n)).cuda() for hm in hms]

    def product(i, op):
        y = torch.zeros_like(xs[i])
        if entry == "noalloc":
            _noalloc(Ms[i], 0.5, op, xs[i], y)
        elif entry == "workspace" and i == 2:
            hlr.mul_vec(0.5, op, Ms[i], xs[i], y, workspace=W)
        else:
            hlr.mul_vec(0.5, op, Ms[i], xs[i], y)
        torch.cuda.synchronize()
        return y

    ref = {(i, op): product(i, op) for i in range(3) for op in (0, 2)}
    for i, hm in enumerate(hms):                       # the reference bits are right
        for op in (0, 2):
            yo = np.zeros(hm.n)
            xh = xs[i].cpu().numpy()
            if i == 2:
                assert oracle.uniform_mvm(hm.uniform_desc(), 0.5, op, xh, yo) == 0
            else:
                oracle.hmvm_seq(hm.h_desc(), 0.5, op, xh, yo)
            assert relerr(ref[i, op].cpu().numpy(), yo) <= 1e-13
    L = _capi.lib()
    for bad in range(3):
        assert L.hlrc_debug_waits(Ms[bad].handle, 5_000_000, 1) == 0     # 5 ms; one item is never counted
        product(bad, 0)
        assert Ms[bad].device_error() & 1
        assert L.hlrc_debug_waits(Ms[bad].handle, 0, 0) == 0
        for (i, op), y in ref.items():
            assert torch.equal(product(i, op), y), (bad, i, op)
    assert all(M.device_error() == 0 for M in Ms)
    if W:
        W.free()
    for M in Ms:
        M.free()
