"""Design regions in the sweep against the two-pass schedule, bit for bit: boxes on the edges of its tiles and against the CPML
slabs, among random materials (so that the region's surface has many coefficient rows), eps_r replaced between steps, and
more materials' rows than the table holds (the region's nodes then take the general path)."""
import numpy as np
import pytest

from conftest import bitwise_equal
from fdtd_gb300 import scenario as S

pytestmark = pytest.mark.gpu


def drive(sc, schedule, box, calls, index=None):
    import torch
    from fdtd_gb300 import solver
    gen = torch.Generator(device="cuda").manual_seed(9)
    rng = np.random.default_rng(8)
    shape = (box[5] - box[2], box[4] - box[1], box[3] - box[0])
    with solver.Simulation.from_scenario(sc, schedule, material_index=index, probe_capacity=64) as sim:
        for c in range(6):
            f = torch.rand((sc.nz, sc.ny, sc.nx), generator=gen, device="cuda") - 0.5
            sim.set_field_device(c, f.data_ptr())
            torch.cuda.synchronize()
        base = dict(sigma_e=0.01, mu_r=sc.design_mu, sigma_m=3.0) if sc.design_mu != 1.0 else {}
        for n in calls:
            sim.set_design_region(box, rng.uniform(1, 12, shape).astype(np.float32), **base)
            sim.step(n)
        buf = torch.empty(sim.state_bytes(), dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        sim.save_state(buf.data_ptr())
        torch.cuda.synchronize()
        return sim.read_probes(0, sum(calls)), buf


def grid(dims, pml, mu=1.0, materials=0, seed=1):
    sc = S.vacuum_cube(dims[0], 16, pml=pml, name="design_sweep")
    sc.nx, sc.ny, sc.nz = dims
    sc.design_mu = mu
    rng = np.random.default_rng(seed)
    sc.materials += [S.Material(eps_r=float(rng.uniform(1, 9)), sigma_e=float(rng.uniform(0, 0.05)), mu_r=mu) for _ in range(materials)]
    sc.sources = [S.LumpedSource((2, 2, 2, 2, 2, 3), 50.0, rng.standard_normal(16).astype(np.float32))]
    c = [n // 2 for n in dims]
    sc.probes = [S.Probe(q, *c) for q in range(6)]
    index = rng.integers(0, materials + 1, dims[::-1]).astype(np.uint8) if materials else None
    return sc, index


def same(sc, box, index, calls=(3, 4)):
    import torch
    p1, s1 = drive(sc, 1, box, calls, index)
    p2, s2 = drive(sc, 2, box, calls, index)
    assert np.isfinite(p1).all() and np.abs(p1).max() > 0
    assert bitwise_equal(p1, p2) and torch.equal(s1, s2)


@pytest.mark.parametrize("dims,pml,box", [
    ((64, 48, 40), 6, (6, 6, 6, 57, 41, 33)),          # from slab to slab
    ((97, 61, 40), 8, (31, 15, 12, 33, 17, 20)),       # across tile edges
    ((97, 61, 40), 8, (32, 16, 10, 64, 48, 31)),       # on them
    ((70, 50, 44), 5, (63, 43, 37, 64, 44, 38)),       # one cell, in a corner
    ((130, 210, 45), 8, (20, 30, 10, 110, 180, 30)),   # more CTAs than the two-per-SM kernel takes
    ((40, 36, 34), 0, (1, 1, 1, 38, 34, 32)),          # no CPML: wall to wall
])
@pytest.mark.parametrize("mu,materials", [(1.0, 0), (1.0, 3), (1.7, 3)])
def test_sweep_equals_two_pass(gpu_lib, dims, pml, box, mu, materials):
    sc, index = grid(dims, pml, mu, materials)
    if not pml:
        sc.sources = []  # no room beside the region
    same(sc, box, index)


def test_more_rows_than_the_table(gpu_lib):
    """Random materials throughout: the interface rows fill the table, none is left for the region's nodes."""
    sc, index = grid((64, 48, 40), 6, 1.0, 250)
    same(sc, (20, 12, 10, 45, 30, 30), index)


def test_auto_takes_the_sweep(gpu_lib):
    """A design handle stepped under AUTO takes the sweep where other grids do; the adjoint's forward on it
    stays with the two-pass kernels, which take its records, from either buffer."""
    from fdtd_gb300 import solver
    dims, box, probe = (208, 208, 208), (96, 96, 96, 112, 112, 104), (95, 107, 100)
    sc, _ = grid(dims, 10)
    sc.sources = [S.LumpedSource((95, 104, 100, 95, 104, 101), 50.0, np.ones(16, np.float32))]
    eps = np.random.default_rng(2).uniform(1, 12, (8, 16, 16)).astype(np.float32)
    out = []
    for schedule in (0, 1):
        with solver.Simulation.from_scenario(sc, schedule, probe_capacity=64) as sim:
            sim.set_design_region(box, eps)
            sim.prepare()
            sim.tune_schedule()
            assert sim.active_schedule == (2 if schedule == 0 else 1)
            sim.step(3)
            J = sim.adjoint_forward(24, probe, 4)
            g = sim.adjoint_backward()
            sim.step(2)
            out.append((J, g, sim.fields()))
    assert out[0][0] == out[1][0] and np.array_equal(out[0][1], out[1][1]) and np.abs(out[0][1]).max() > 0
    assert bitwise_equal(out[0][2], out[1][2])


@pytest.mark.parametrize("schedule", [1, 2])
@pytest.mark.parametrize("box", [(10, 8, 7, 16, 14, 11), (14, 11, 9, 19, 16, 14), (16, 8, 11, 19, 14, 14)])
def test_region_moved(gpu_lib, schedule, box):
    """A second region that overlaps the first, or touches it: the first one's other cells hold the base material."""
    import oracle
    from fdtd_gb300 import solver
    sc, _ = grid((26, 24, 22), 4)
    sc.steps, sc.design_mu = 30, 1.0
    sc.sources = [S.LumpedSource((7, 11, 9, 7, 11, 10), 50.0, np.random.default_rng(1).standard_normal(30).astype(np.float32))]
    first = (12, 9, 8, 16, 14, 11)
    rng = np.random.default_rng(6)
    size = lambda b: (b[5] - b[2], b[4] - b[1], b[3] - b[0])  # noqa: E731
    eps = rng.uniform(1, 12, size(box)).astype(np.float32)
    with solver.Simulation.from_scenario(sc, schedule, probe_capacity=64) as sim:
        sim.set_design_region(first, rng.uniform(1, 12, size(first)).astype(np.float32), sigma_e=0.02)
        sim.prepare()
        sim.set_design_region(box, eps, sigma_e=0.02)
        sim.step(sc.steps)
        sim.synchronize()
        p, f, prof = sim.read_probes(0, sc.steps), sim.fields(), sim.cpml_profiles()
    sc.materials.append(S.Material(eps_r=1.0, sigma_e=0.02))
    sc.bricks += [S.Brick(first, 1), S.Brick(box, 1)]  # both boxes hold the base material; the oracle adds eps_r
    po, fo = oracle.run(sc, profile_override=prof, design=(box, eps.astype(np.float64)))
    assert np.abs(po).max() > 0
    assert bitwise_equal(p, po) and bitwise_equal(f, fo)
