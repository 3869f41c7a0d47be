"""Products of host vectors (hlrc_mvm_host; the reference's scalar_vectors are
host objects) against the oracle: pageable vectors pass through a ring of 16
pinned slots of 128 KiB, filled in packed order whatever the column length;
pinned ones are copied directly.  Short columns that share a slot, columns that
end inside a slot, one column longer than the ring, a ring that grows between
calls, a leading dimension with padding, and every mix of pageable and pinned."""
import ctypes as C

import numpy as np
import pytest

import hlr_b200 as hlr
import oracle
from hlr_b200 import _capi

from conftest import built, relerr

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

TOL = 1e-13   # the FP64 parity bound


def _vectors(n, k, pad, seed, pinned):
    """(array as stored, (n, k) column-major view) with rows of padding after each column."""
    a = torch.from_numpy(np.random.default_rng(seed).standard_normal((k, n + pad)))
    if pinned:
        a = a.pin_memory()
    return a, a.T[:n] if k > 1 else a[0, :n]


def _check(M, hm, k, pad=0, op=0, px=False, py=False, alpha=-1.25):
    n = hm.n
    xs, x = _vectors(n, k, pad, 1, px)
    ys, y = _vectors(n, k, pad, 2, py)
    y0 = ys.numpy().copy()
    hlr.mul_vec(alpha, op, M, x, y)
    got = ys.numpy()
    d = hm.fetch().h_desc() if hm.n > 20000 else hm.h_desc()
    for j in range(k):
        ref = np.zeros(n)
        oracle.hmvm_seq(d, alpha, op, np.ascontiguousarray(xs.numpy()[j, :n]), ref)
        assert relerr(got[j, :n] - y0[j, :n], ref) <= TOL, (k, j)
    assert np.array_equal(got[:, n:], y0[:, n:])


@pytest.mark.parametrize("px,py", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("n,k", [(300, 1), (300, 64), (1000, 16), (5003, 7), (2047, 8)])
def test_short_columns(n, k, px, py):
    hm = built(f"log_{n}", lambda: hlr.build(hlr.Problem.log1d(n)))
    M = hlr.upload(hm, max_nrhs=max(1, k // 2))
    for op in (0, 1):
        _check(M, hm, k, pad=0, op=op, px=px, py=py)
        _check(M, hm, k, pad=5, op=op, px=px, py=py)
    assert M.device_error() == 0
    M.free()


@pytest.mark.parametrize("n,k", [(300007, 1), (40009, 8)])
def test_more_than_the_ring_holds(n, k):
    hm = built(f"log_{n}_dev", lambda: hlr.build(hlr.Problem.log1d(n, on_device=True)))
    assert n * k * 8 > 16 << 17
    M = hlr.upload(hm, max_nrhs=k)
    _check(M, hm, k, pad=3 if k > 1 else 0)
    M.free()


def test_ring_grows_and_mixed_calls():
    hm = built("log_5003", lambda: hlr.build(hlr.Problem.log1d(5003)))
    M = hlr.upload(hm, max_nrhs=8)
    for k, px, py in ((1, False, False), (1, True, True), (4, False, False), (2, True, False), (64, False, False),
                      (3, False, True), (1, False, False)):
        _check(M, hm, k, pad=1, px=px, py=py)
    assert M.device_error() == 0
    M.free()


def test_after_a_call_too_large_for_the_device():
    """A call whose staging buffers do not fit is refused before it touches its
    vectors; the next call works."""
    hm = built("log_300", lambda: hlr.build(hlr.Problem.log1d(300)))
    M = hlr.upload(hm, max_nrhs=2)
    _check(M, hm, 2)
    x, y = np.ones((4, 300)), np.ones((4, 300))
    st = _capi.lib().hlrc_mvm_host(M.handle, 1.0, 0, C.c_void_p(x.ctypes.data), C.c_void_p(y.ctypes.data),
                                   100_000_000, 300, 300)          # 240 GB
    assert st != 0 and np.array_equal(y, np.ones((4, 300)))
    _check(M, hm, 1)
    _check(M, hm, 2, pad=1)
    assert M.device_error() == 0
    M.free()
