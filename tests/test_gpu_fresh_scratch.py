"""A handle or a workspace is complete when the call that makes it returns:
products may start at once on a non-blocking stream, which nothing orders after
work that the default stream still has queued.  (HLR's matrices and vectors are
host objects, usable as soon as their constructors return.)"""
import numpy as np
import pytest

import hlr_b200 as hlr
import oracle

from conftest import built, relerr

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

TOL = 1e-13   # the FP64 parity bound


@pytest.mark.parametrize("what", ["workspace", "handle"])
def test_usable_while_the_default_stream_is_busy(what):
    hm = built("log_4099", lambda: hlr.build(hlr.Problem.log1d(4099)))
    rng = np.random.default_rng(3)
    xh, yh = rng.standard_normal(hm.n), rng.standard_normal(hm.n)
    ref = {}
    for op in (0, 1):
        ref[op] = np.zeros(hm.n)
        oracle.hmvm_seq(hm.h_desc(), 1.5, op, xh, ref[op])
    M = hlr.upload(hm)
    st = torch.cuda.Stream()
    x = torch.from_numpy(xh).cuda()
    ys = [torch.from_numpy(yh).cuda() for _ in range(8)]
    torch.cuda.synchronize()
    with torch.cuda.stream(st):    # the first launch of a kernel loads it, which waits for the device
        for op in (0, 1):
            hlr.mul_vec(1.5, op, M, x, torch.zeros_like(x))
    a = torch.randn((4096, 4096), device="cuda")
    a @ a
    torch.cuda.synchronize()
    for _ in range(200):
        a @ a                      # ordinary work on the default stream, some 400 ms
    busy = torch.cuda.Event()
    busy.record()
    made = []
    for k, y in enumerate(ys):
        with torch.cuda.stream(st):
            if what == "workspace":
                made.append(hlr.Workspace(M))
                hlr.mul_vec(1.5, k % 2, M, x, y, workspace=made[-1])
            else:                  # the upload's copies wait for the default stream themselves
                made.append(hlr.upload(hm))
                hlr.mul_vec(1.5, k % 2, made[-1], x, y)
    st.synchronize()
    if what == "workspace":
        assert not busy.query()    # nothing waited for the default stream
    torch.cuda.synchronize()
    for k, y in enumerate(ys):
        assert relerr(y.cpu().numpy() - yh, ref[k % 2]) <= TOL, k
    assert M.device_error() == 0
    for m in made:
        m.free()
    M.free()
