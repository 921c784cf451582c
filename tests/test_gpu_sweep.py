"""The fused schedule's sweep of the whole grid (k_sweep) against the two-pass schedule, bit for bit:
probes of every step and the full state (fields, CPML memory) after an odd and an even count.

The grids sit on the edges of its tiles (32 x 16 nodes, quads of four, chunks of planes): one tile
and one node more or less, both x slabs in one quad, slabs that end inside a quad, faces without
CPML, a grid of a few nodes. Materials reach through the slabs to the walls (rows other than the
background's there), with mixed quads inside and outside; lumped edges, plates and probes lie in the
interior, in the slabs and on the walls; more sources than the launch carries signals for.
"""
import numpy as np
import pytest

from conftest import bitwise_equal
from fdtd_gb300 import scenario as S

pytestmark = pytest.mark.gpu


def case(dims, pml, seed, materials=True, background=None, n_sources=2, plates=False):
    rng = np.random.default_rng(seed)
    nx, ny, nz = dims
    delta, dt = 1e-3, float(S.courant_dt(1e-3, 1e-3, 1e-3, 0.99))
    mats, bricks = [background or S.Material()], []
    if materials:
        for q in range(6):
            lo = [int(rng.integers(0, n)) for n in dims]
            hi = [min(n, a + int(rng.integers(1, max(2, n // 2)))) for a, n in zip(lo, dims)]
            if q == 0:
                lo, hi = [0, 0, 0], [nx, ny, max(1, nz // 3)]  # a half space: through every slab it meets
            mats.append(S.Material(eps_r=tuple(float(v) for v in rng.uniform(1, 9, 3)), sigma_e=float(rng.uniform(0, 0.05)),
                                   mu_r=float(rng.uniform(1, 3)), sigma_m=float(rng.uniform(1, 500))))
            bricks.append(S.Brick((*lo, *hi), q + 1))
    used, sources, loads = set(), [], []
    for q in range(n_sources + 1):
        for _ in range(200):
            e = (int(rng.integers(1, nx - 1)), int(rng.integers(1, ny - 1)), int(rng.integers(0, nz - 1)))
            if e not in used:
                break
        else:
            break
        used.add(e)
        box = (*e, e[0], e[1], e[2] + 1)
        if q < n_sources:
            sources.append(S.LumpedSource(box, 50.0, rng.standard_normal(9).astype(np.float32)))
        else:
            loads.append(S.Resistor(box, 75.0))
    at = lambda: tuple(int(rng.integers(0, n)) for n in dims)  # noqa: E731
    pts = [at() for _ in range(4)] + [(0, 0, 0), (nx - 1, ny - 1, nz - 1), (nx // 2, 0, nz - 1), (nx // 2, ny // 2, nz // 2)]
    probes = [S.Probe(c, *q) for q in pts for c in range(6)]
    sc = S.Scenario("sweep", nx, ny, nz, delta, delta, delta, dt, pml, 16, mats, bricks, sources, loads, probes)
    if plates:
        k = [e[2] for e in used]
        free = [q for q in range(1, nz - 1) if q not in k and q - 1 not in k]
        sc.plates = [S.Plate(2, (1, 1, free[0], nx - 2, ny - 2, free[0]), 1e10, 1e7),
                     S.Plate(2, (nx // 2, 0, free[-1], nx - 1, ny // 2, free[-1]), 3e3, 1e10)]
    return sc


def run(sc, schedule, calls, seed=1):
    import torch
    from fdtd_gb300 import solver
    gen = torch.Generator(device="cuda").manual_seed(seed)
    with solver.Simulation.from_scenario(sc, schedule, probe_capacity=32) as sim:
        for c in range(6):  # every node in use, walls included
            f = torch.rand((sc.nz, sc.ny, sc.nx), generator=gen, device="cuda") - 0.5
            sim.set_field_device(c, f.data_ptr())
            torch.cuda.synchronize()
        states = []
        for n in calls:
            sim.step(n)
            buf = torch.empty(sim.state_bytes(), dtype=torch.uint8, device="cuda")
            torch.cuda.synchronize()
            sim.save_state(buf.data_ptr())
            torch.cuda.synchronize()
            states.append(buf)
        return sim.read_probes(0, sum(calls)), states


def check(sc, schedule=2, calls=(5, 4)):
    import torch
    p1, s1 = run(sc, 1, calls)
    p2, s2 = run(sc, schedule, calls)
    assert np.isfinite(p1).all() and np.abs(p1).max() > 0
    assert bitwise_equal(p2, p1)
    for a, b in zip(s2, s1):
        assert torch.equal(a, b)


@pytest.mark.parametrize("dims,pml", [
    ((32, 16, 32), (4,) * 6),
    ((33, 17, 33), (4, 5, 3, 6, 2, 7)),
    ((31, 15, 31), (6, 6, 6, 6, 6, 6)),
    ((64, 48, 20), (10, 10, 10, 10, 8, 8)),
    ((65, 33, 70), (10, 9, 8, 7, 6, 5)),
    ((97, 61, 40), (0, 5, 0, 6, 7, 0)),
    ((63, 40, 35), (1, 1, 1, 1, 1, 1)),
    ((40, 36, 34), (0,) * 6),
    ((7, 9, 11), (3, 3, 4, 4, 5, 5)),
    ((6, 5, 4), (1, 3, 2, 2, 0, 3)),
    ((3, 3, 3), (0,) * 6),
    ((130, 20, 100), (2, 11, 7, 8, 30, 33)),
    ((130, 210, 45), (5, 4, 8, 7, 6, 6)),  # more CTAs than the two-per-SM kernel takes
])
@pytest.mark.parametrize("materials", [False, True])
def test_sweep_equals_two_pass(gpu_lib, dims, pml, materials):
    check(case(dims, pml, seed=sum(dims) + sum(pml), materials=materials, n_sources=1 if min(dims) < 6 else 3))


@pytest.mark.parametrize("seed", [1, 2])
def test_sweep_plates_sources_and_background(gpu_lib, seed):
    """Plates through the slabs, more sources than kSweepSources, a background material whose H
    coefficients differ from the default entry's; also as FUSED_CPML and AUTO."""
    sc = case((70, 50, 44), (6, 5, 7, 4, 5, 6), seed, n_sources=11, plates=True,
              background=S.Material(eps_r=2.0, sigma_e=0.01, mu_r=1.5, sigma_m=40.0))
    for schedule in (0, 2, 3):
        check(sc, schedule, (3, 1, 4))


@pytest.mark.parametrize("schedule", [1, 2])
def test_more_probes_than_threads(gpu_lib, schedule):
    """Every component of every node a probe, twice over: more probes than the step's kernels have
    threads. Outside the CPML each holds the field after its step."""
    import torch
    from fdtd_gb300 import solver
    nx, ny, nz, p, steps = 20, 18, 16, 3, 3
    sc = case((nx, ny, nz), (p,) * 6, 3, n_sources=1)
    pts = [(i, j, k) for k in range(p, nz - p) for j in range(p, ny - p) for i in range(p, nx - p)]
    sc.probes = [S.Probe(c, *q) for _ in range(2) for q in pts for c in range(6)]
    with solver.Simulation.from_scenario(sc, schedule, probe_capacity=steps) as sim:
        want = []
        for _ in range(steps):
            sim.step(1)
            f = sim.fields()
            want.append([f[c][k, j, i] for i, j, k in pts for c in range(6)] * 2)
        assert bitwise_equal(sim.read_probes(0, steps), np.array(want, np.float32))
    with solver.Simulation.from_scenario(sc, schedule, probe_capacity=steps) as sim:
        sim.step(steps)
        assert bitwise_equal(sim.read_probes(0, steps), np.array(want, np.float32))
    assert np.abs(np.array(want)).max() > 0
