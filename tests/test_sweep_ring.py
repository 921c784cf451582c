"""CPU test of the sweep's ring of planes (fdtd_gb300/csrc/planner.h, SweepRing), compiled with g++: a model of the march
issues the copies as the kernel does, and at every plane step where a wait may be found to have failed, the planes that the
chunk then waits for are those asked for and not known to have arrived, the failed one among them, each by the phase of its
own copy."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "fdtd_gb300", "csrc")

PROBE = r"""
#include "planner.h"
using fdtd::SweepRing;
extern "C" int stage(int q, int n) { return SweepRing::stage(q, n); }
extern "C" int parity(int q, int n) { return (int)SweepRing::parity(q, n); }
extern "C" int begin(int k) { return SweepRing::drain_begin(k); }
extern "C" int end(int k, int k1, int n) { return SweepRing::drain_end(k, k1, n); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("sweep_ring")
    src, so = d / "probe.cpp", d / "probe.so"
    src.write_text(PROBE)
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I" + CSRC, "-o", str(so), str(src)])
    return ctypes.CDLL(str(so))


@pytest.mark.parametrize("n", [2, 3, 4])
@pytest.mark.parametrize("planes", [1, 2, 3, 4, 7, 32])
def test_drained_planes(lib, n, planes):
    k0, k1 = 5, 5 + planes
    last = {}                                   # stage -> plane of its latest copy
    copies = {s: 0 for s in range(n)}           # copies asked for per stage: the next one completes phase copies & 1

    def issue(k):
        s = lib.stage(k - (k0 - 1), n)
        assert lib.parity(k - (k0 - 1), n) == copies[s] & 1
        copies[s] += 1
        last[s] = k

    for k in range(k0 - 1, min(k1, k0 + n - 2) + 1):  # the kernel's first copies
        issue(k)
    s, parity = 1 % n, 0
    for k in range(k0, k1 + 2):                 # top of plane step k: the wait for plane k - 1 may have failed
        asked = set(last.values())
        drained = list(range(lib.begin(k), lib.end(k, k1, n)))
        assert k - 1 in drained
        assert set(drained) == {q for q in asked if q >= k - 1}
        for q in drained:                       # waited for by its own phase, the stage's latest
            assert last[lib.stage(q - (k0 - 1), n)] == q
        if k > k1:
            break
        assert (s, parity) == (lib.stage(k - (k0 - 1), n), lib.parity(k - (k0 - 1), n))
        if k + n - 1 <= k1:
            issue(k + n - 1)
        s += 1
        if s == n:
            s, parity = 0, parity ^ 1
