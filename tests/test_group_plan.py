"""Group T-form tables of products of more than 8 vectors (host only): no slab is
left out or repeated, whatever the distance of a group's tiles in the store
(tests/c/group_plan.cpp compiles the planner with the limit as a parameter)."""
import ctypes as C
import subprocess

import numpy as np
import pytest

import hlr_b200 as hlr

from conftest import ROOT, built


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    so = tmp_path_factory.mktemp("group_plan") / "group_plan.so"
    csrc = ROOT / "hlr_b200" / "csrc"
    cmd = ["g++", "-O1", "-std=c++17", "-fPIC", "-shared", "-fopenmp", f"-I{ROOT / 'include'}", f"-I{csrc}",
           str(ROOT / "tests" / "c" / "group_plan.cpp"), str(csrc / "common.cpp"), "-o", str(so)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    f = C.CDLL(str(so)).group_plan_check

    def run(desc, span):
        n = C.c_int(0)
        st = f(C.byref(desc), C.c_uint64(span), C.byref(n))
        return st, n.value
    return run


MATRICES = {
    "log": lambda: built("c1_small", lambda: hlr.build(hlr.Problem.log1d(2048))),
    "exp_ragged": lambda: built("exp_3001", lambda: hlr.build(hlr.Problem.exp3d(3001))),
    "log_leaf20": lambda: built("dw_h_leaf20", lambda: hlr.build(hlr.Problem.log1d(1700, leaf_size=20))),
}


@pytest.mark.parametrize("name", sorted(MATRICES))
def test_every_slab_is_in_one_group_chunk(check, name):
    d = MATRICES[name]().h_desc()
    st, whole = check(d, 0)
    assert st == 0 and whole > 0
    counts = [whole]
    for span in (1 << 20, 1 << 16, 1 << 13, 1 << 11, 2):   # elements; 2: no two slabs share a segment
        st, n = check(d, span)
        assert st == 0, span
        counts.append(n)
    assert counts[-1] > counts[0]


def test_one_wide_dense_block(check):
    """A single dense block: the tiles of a group lie a whole tile row apart."""
    m = hlr.LeafList(256, 9000)
    m.add_dense(0, 0, np.asfortranarray(np.random.default_rng(0).standard_normal((256, 9000))))
    d = m.h_desc()
    assert check(d, 0)[0] == 0
    for span in (64 * 9000 * 3 - 1, 64 * 9000, 64 * 100):
        assert check(d, span)[0] == 0
