"""hlrc_tuning.exact_warps: 8 warps per CTA, one CTA per tile, where the default
chooses per pass (several CTAs per tile, 4 or 16 warps).  The same product to
rounding, other sums where the choice is another; settings survive a round trip."""
import numpy as np
import pytest

import hlr_b200 as hlr
import oracle
from hlr_b200 import tune

from conftest import built, relerr

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

CASES = {   # matrix, whether the default's N-form sums are those of 8 warps
    "exp_6007": (lambda: hlr.build(hlr.Problem.exp3d(6007)), False),                       # clusters of CTAs per tile
    "exp_20011_dev": (lambda: hlr.build(hlr.Problem.exp3d(20011, on_device=True)), False),  # 16 warps
    "log_100003_dev": (lambda: hlr.build(hlr.Problem.log1d(100003, on_device=True)), False),   # 4 warps
    "log_8193": (lambda: hlr.build(hlr.Problem.log1d(8193)), True),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_exactly_eight_warps(name):
    make, same = CASES[name]
    hm = built(name, make)
    M = hlr.upload(hm)
    assert M.tuning == tune.DEFAULT
    xh = np.random.default_rng(4).standard_normal(hm.n)
    x = torch.from_numpy(xh).cuda()

    def product(op):
        y = torch.zeros_like(x)
        hlr.mul_vec(1.5, op, M, x, y)
        torch.cuda.synchronize()
        return y.cpu().numpy()

    auto = {op: product(op) for op in (0, 1)}
    M.set_tuning(exact_warps=1)
    assert M.tuning == dict(tune.DEFAULT, exact_warps=1)
    M.set_tuning(**M.tuning)
    exact = {op: product(op) for op in (0, 1)}
    for op in (0, 1):
        ref = np.zeros(hm.n)
        oracle.hmvm_seq(hm.fetch().h_desc() if name.endswith("_dev") else hm.h_desc(), 1.5, op, xh, ref)
        assert relerr(exact[op], ref) <= 1e-13
        assert relerr(exact[op], auto[op]) <= 1e-14
    assert np.array_equal(exact[0], auto[0]) == same
    M.set_tuning(exact_warps=0)
    assert M.tuning == tune.DEFAULT and np.array_equal(product(0), auto[0])
    M.free()
