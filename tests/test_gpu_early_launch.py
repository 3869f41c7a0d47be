"""Kernels launched before their predecessor has ended read the vectors only
after it has: products on changing vectors, issued one after the other without a
synchronisation, equal those of plain launches (overlap = 0) bit for bit.  All
stores; one vector, blocks of 8 to 64, and workspaces whose passes differ in
width (16 + 1, 16 + 16 + 1 vectors: the second pass's kernels must not take the
first pass's x); every op of the matrix."""
import numpy as np
import pytest

import hlr_b200 as hlr

from conftest import built

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

MATRICES = {
    "exp": lambda: built("exp_3000", lambda: hlr.build(hlr.Problem.exp3d(3000))),
    "log": lambda: built("log_9001", lambda: hlr.build(hlr.Problem.log1d(9001))),
    "uniform": lambda: built("c3_small", lambda: hlr.build(hlr.Problem.laplace_sphere(refine=4, uniform=True))),
    "h2": lambda: built("sphere5_h2", lambda: hlr.build(hlr.Problem.laplace_sphere(refine=5, nested=True))),
}
CASES = [(m, "f64") for m in sorted(MATRICES)] + [("exp", p) for p in ("f32", "mixed", "bfp", "f16", "bf16")] + \
        [("log", "mixed"), ("log", "f16")]


@pytest.mark.parametrize("name,prec", CASES)
def test_early_launches_read_the_latest_vectors(name, prec):
    hm = MATRICES[name]()
    M = hlr.upload(hm, precision=prec, uniform=name == "uniform", h2=name == "h2", max_nrhs=64)
    W = hlr.Workspace(M, max_nrhs=16)
    ops = (0, 2) if name in ("uniform", "h2") else (0, 1)
    kmax, rounds = 66, 4
    g = torch.Generator(device="cuda").manual_seed(17)
    X = torch.randn((rounds, kmax, hm.n), dtype=torch.float64, device="cuda", generator=g)
    for op in ops:
        for k in (1, 2, 8, 9, 17, 18, 33, 64, 66):
            for ws in (None, W):
                out = []
                for overlap in (0, 1):
                    M.set_tuning(overlap=overlap)
                    Y = torch.zeros((kmax, hm.n), dtype=torch.float64, device="cuda")
                    Xw = torch.empty((kmax, hm.n), dtype=torch.float64, device="cuda")
                    for r in range(rounds):
                        Xw.copy_(X[r])          # a kernel on the stream writes x, the next one reads it
                        hlr.mul_vec(1.0 + r, op, M, Xw.T[:, :k], Y.T[:, :k], workspace=ws)
                        # y is the next product's x: two products back to back
                        hlr.mul_vec(0.5, op, M, Y.T[:, :k], Xw.T[:, :k], workspace=ws)
                        Y.add_(Xw)
                    torch.cuda.synchronize()
                    out.append(Y)
                assert torch.equal(out[0], out[1]), (op, k, ws is not None)
    assert M.device_error() == 0
    W.free()
    M.free()
