"""CPU test of the sweep's chunk plan for grids with materials in the CPML slabs and for grids swept several at once
(fdtd_gb300/csrc/planner.cpp, plan_sweep), compiled with g++: the chunks cover the planes in order, none is longer than the
kernel's tables, and where the plan cuts at the z slabs its middle chunks meet none."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "fdtd_gb300", "csrc")

PROBE = r"""
#include "planner.h"
extern "C" void plan(const int* g9, double share, int rows, int* out) {
    const fdtd::SweepPlan p =
        fdtd::plan_sweep(fdtd::PlanGrid{g9[0], g9[1], g9[2], g9[3], g9[4], g9[5], g9[6], g9[7], g9[8]}, share, rows != 0);
    const int v[7] = {p.nbx, p.nby, p.zlo, p.zhi, p.n_lo, p.n_mid, p.n_hi};
    for (int q = 0; q < 7; ++q) out[q] = v[q];
    for (int c = 0; c <= p.chunks(); ++c) out[7 + c] = p.chunk(c);
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("sweep_plan_rows")
    src, so = d / "probe.cpp", d / "probe.so"
    src.write_text(PROBE)
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I" + CSRC, "-o", str(so),
                           os.path.join(CSRC, "planner.cpp"), str(src)])
    return ctypes.CDLL(str(so))


@pytest.mark.parametrize("share", [1.0, 2.0, 2 / 64, 2 / 256])
@pytest.mark.parametrize("rows", [0, 1])
@pytest.mark.parametrize("dims,pz", [
    ((64, 64, 64), (10, 10)), ((144, 144, 144), (10, 10)), ((192, 192, 192), (10, 10)), ((225, 225, 225), (8, 12)),
    ((512, 512, 512), (10, 10)), ((1024, 1024, 896), (10, 10)), ((93, 77, 51), (12, 5)), ((512, 512, 70), (0, 0)),
    ((512, 512, 65), (33, 30)), ((600, 600, 40), (1, 0)), ((3, 3, 3), (0, 0)), ((40, 40, 2000), (20, 0)), ((300, 300, 9), (4, 4)),
])
def test_chunks(lib, dims, pz, rows, share):
    g = (ctypes.c_int * 9)(*dims, 0, 0, 0, 0, *pz)
    out = (ctypes.c_int * (8 + dims[2] + 8))()
    lib.plan(g, ctypes.c_double(share), rows, out)
    nbx, nby, zlo, zhi, n_lo, n_mid, n_hi = list(out)[:7]
    assert nbx == (dims[0] + 31) // 32 and nby == (dims[1] + 15) // 16
    c = list(out)[7:8 + n_lo + n_mid + n_hi]
    assert c[0] == 0 and c[-1] == dims[2]
    assert all(0 < b - a <= 32 for a, b in zip(c, c[1:]))
    if n_lo or n_hi:  # the middle chunks' planes and the one above meet no z slab and no z wall
        lo, hi = max(pz[0], 1), min(dims[2] - pz[1], dims[2] - 1)
        mid = c[n_lo:n_lo + n_mid + 1]
        assert mid[0] == zlo >= lo and mid[-1] == zhi < hi
        assert n_lo >= 1 and n_hi >= 1
