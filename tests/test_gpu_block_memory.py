"""An FP64 upload for many vectors that fits the device only without the tables of
the block kernels, or only with narrower blocks, still works: its products go in
blocks of fewer vectors.  The device is filled up to what the same matrix needs
for 8 vectors and a little more."""
import ctypes as C

import pytest

import hlr_b200 as hlr

from conftest import built

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _fill(cudart, leave):
    """Allocations (of the runtime itself: torch rounds its own up) that leave `leave`
    bytes of the device free, or up to 2 MB more."""
    hold = []
    for step in (1 << 33, 1 << 30, 1 << 26, 2 * MB):
        while torch.cuda.mem_get_info()[0] - leave >= step:
            p = C.c_void_p()
            if cudart.cudaMalloc(C.byref(p), C.c_size_t(step)) != 0:
                cudart.cudaGetLastError()
                break
            hold.append(p)
    return hold


def test_upload_beside_a_full_device():
    hm = built("exp_65536_dev", lambda: hlr.build(hlr.Problem.exp3d(65536, on_device=True)))
    g = torch.Generator(device="cuda").manual_seed(3)
    X = torch.randn((24, hm.n), dtype=torch.float64, device="cuda", generator=g).T

    def product(M):
        out = []
        for op in (0, 2):
            Y = torch.zeros((24, hm.n), dtype=torch.float64, device="cuda").T
            hlr.mul_vec(1.0, op, M, X, Y)
            out.append(Y)
        torch.cuda.synchronize()
        return out

    # what each upload takes of the device
    need, info = {}, {}
    for k in (8, 24):
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        M = hlr.upload(hm, max_nrhs=k)
        need[k], info[k] = before - torch.cuda.mem_get_info()[0], M.info
        if k == 24:
            ref = product(M)
        M.free()
    tables = (info[24]["device_bytes"] - info[24]["workspace_bytes"]) - \
             (info[8]["device_bytes"] - info[8]["workspace_bytes"])
    assert tables > 8 * MB                   # so that they do not fit in the margin below
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    cudart = C.CDLL("/usr/local/cuda/lib64/libcudart.so")
    hold = _fill(cudart, need[8] + 4 * MB)
    try:
        M = hlr.upload(hm, max_nrhs=24)
    finally:
        for p in hold:
            cudart.cudaFree(p)
    assert M.info["device_bytes"] < info[24]["device_bytes"] - tables // 2
    for y, r in zip(product(M), ref):
        assert float((y - r).norm() / r.norm()) <= 1e-13
    assert M.device_error() == 0
    M.free()
