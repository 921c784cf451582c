"""What fdtd_prepare leaves behind, on grids whose tables of coefficient rows are large: a block of cells of random
materials in a corner, so that nearly every node of it has a row of its own, between thick CPML slabs."""
import numpy as np
import pytest

from fdtd_gb300 import scenario as S

pytestmark = pytest.mark.gpu

SLAB_ROW_BYTES = 32  # of one row and one plane of a slab, E and H


def key_count(index):
    """Distinct seven-cell material combinations of the grid's nodes (cells outside it count as material 0)."""
    p = np.pad(index, ((1, 0),) * 3).astype(np.uint64)
    at = lambda k, j, i: p[1 - k:p.shape[0] - k, 1 - j:p.shape[1] - j, 1 - i:p.shape[2] - i]  # noqa: E731
    key = np.zeros(index.shape, np.uint64)
    for k, j, i in ((0, 0, 0), (0, 0, 1), (0, 1, 0), (1, 0, 0), (0, 1, 1), (1, 0, 1), (1, 1, 0)):
        key = key * np.uint64(256) + at(k, j, i)
    return np.unique(key).size


def rows_case(n, pml, block, steps=6):
    """A grid of n^3 cells, `pml` cells of CPML on every face and block^3 cells of random materials."""
    rng = np.random.default_rng(n + pml + block)
    sc = S.vacuum_cube(n, steps, pml=pml, name="rows")
    sc.materials += [S.Material(eps_r=float(rng.uniform(1, 9)), sigma_e=float(rng.uniform(0, 0.05)), mu_r=float(rng.uniform(1, 3)))
                     for _ in range(250)]
    index = np.zeros((n, n, n), np.uint8)
    index[:block, :block, :block] = rng.integers(1, 251, (block,) * 3)
    sc.material_index = lambda: index
    c = n // 2
    sc.sources = [S.LumpedSource((c, c, c, c, c, c + 1), 50.0, rng.standard_normal(steps).astype(np.float32))]
    sc.probes = [S.Probe(S.EZ, c, c, c), S.Probe(S.HX, c, c, c)]
    return sc, index


def test_prepare_waits_for_its_kernels(gpu_lib):
    """The slab coefficients of 27000 rows are some 240 MB: nothing of the preparation is still running on its stream
    when the call returns (the next step may use another stream)."""
    import torch
    from fdtd_gb300 import solver
    n, pml, block = 100, 46, 29
    sc, index = rows_case(n, pml, block)
    assert 200e6 < key_count(index) * 6 * pml * SLAB_ROW_BYTES < 260e6
    stream = torch.cuda.Stream()
    with solver.Simulation.from_scenario(sc, 1, material_index=index) as sim:
        torch.cuda.synchronize()
        sim.set_stream(stream.cuda_stream)
        sim.prepare()
        assert stream.query()
        assert sim.device_bytes() > 2e8  # the table was built
        sim.synchronize()


@pytest.mark.parametrize("schedule", [1, 2])
def test_plates_in_slabs_without_the_slab_rows(gpu_lib, schedule):
    """Some 30000 rows times 300 slab planes are more than the table of slab coefficients may hold (256 MiB): it is
    not built, and plates in the slabs are updated all the same, as the oracle has them."""
    import oracle
    from conftest import bitwise_equal
    from fdtd_gb300 import solver
    n, pml, block = 110, 50, 30
    sc, index = rows_case(n, pml, block)
    assert key_count(index) < 32000 and key_count(index) * 6 * pml * SLAB_ROW_BYTES > 257 * 2**20
    sc.plates = [S.Plate(2, (35, 30, 55, 100, 80, 55), 1e10, 1e7),  # from slab to slab through the middle
                 S.Plate(0, (70, 35, 40, 70, 90, 70), 3e3, 1e10),   # inside an x slab
                 S.Plate(1, (40, 0, 35, 60, 0, 60), 1e5, 1e6)]      # on a low wall
    c = n // 2
    sc.sources = [S.LumpedSource((c, c, c + 2, c, c, c + 3), 50.0, sc.sources[0].waveform)]
    sc.probes = [S.Probe(S.EX, 75, 55, 55), S.Probe(S.EY, 70, 60, 55), S.Probe(S.EZ, 70, 60, 50)]
    rng = np.random.default_rng(4)
    start = np.zeros((6, n, n, n), np.float32)
    start[:, 1:-1, 1:-1, 1:-1] = rng.standard_normal((6, n - 2, n - 2, n - 2)).astype(np.float32)
    with solver.Simulation.from_scenario(sc, schedule, material_index=index, probe_capacity=sc.steps) as sim:
        for q in range(6):
            sim.set_field(q, start[q])
        sim.step(sc.steps)
        sim.synchronize()
        got, fields, prof = sim.read_probes(0, sc.steps), sim.fields(), sim.cpml_profiles()
        assert sim.device_bytes() < 250e6  # without the table
    want, want_fields = oracle.run(sc, init_fields=start, profile_override=prof)
    assert bitwise_equal(got, want) and bitwise_equal(fields, want_fields)


def test_second_buffers_filled_on_the_handles_stream(gpu_lib):
    """The fused schedule's second CPML set is filled on the stream that the steps run on: with the legacy stream busy,
    a handle on a non-blocking stream gets the same state."""
    import torch
    from fdtd_gb300 import solver
    sc = S.vacuum_cube(40, 8, pml=8, name="fill")
    sc.sources, sc.probes = [], []
    gen = torch.Generator(device="cuda").manual_seed(5)
    start = [torch.rand((40, 40, 40), generator=gen, device="cuda") - 0.5 for _ in range(6)]
    stream = torch.cuda.Stream()
    states = []
    for busy in (False, True):
        with solver.Simulation.from_scenario(sc, 2) as sim:
            sim.set_stream(stream.cuda_stream)
            for c, f in enumerate(start):
                sim.set_field_device(c, f.data_ptr())
            sim.prepare()
            state = torch.zeros(sim.state_bytes(), dtype=torch.uint8, device="cuda")
            torch.cuda.synchronize()
            if busy:
                torch.cuda._sleep(200_000_000)  # some 0.1 s on the legacy stream
            sim.step(5)
            torch.cuda.synchronize()
            sim.save_state(state.data_ptr())
            torch.cuda.synchronize()
            states.append(state)
    assert torch.equal(*states)


def test_auto_takes_the_sweep_without_waiting(gpu_lib):
    """The call in which AUTO gets its second buffers enqueues its steps behind whatever the stream still does."""
    import torch
    from conftest import bitwise_equal
    from fdtd_gb300 import solver
    sc = S.vacuum_cube(48, 8, pml=8, name="no_wait")
    sc.probes = []
    stream = torch.cuda.Stream()
    with solver.Simulation.from_scenario(sc, 0) as sim, solver.Simulation.from_scenario(sc, 1) as ref:
        with solver.Simulation.from_scenario(sc, 2) as warm:  # the kernels are loaded
            warm.step(2)
            warm.synchronize()
        sim.set_stream(stream.cuda_stream)
        sim.step(10)
        torch.cuda.synchronize()
        assert sim.active_schedule == 1
        with torch.cuda.stream(stream):
            torch.cuda._sleep(1_000_000_000)  # some 0.5 s
            slept = torch.cuda.Event()
            slept.record(stream)
        sim.step(390)
        assert not slept.query()
        assert sim.active_schedule == 2
        sim.synchronize()
        ref.step(400)
        ref.synchronize()
        assert bitwise_equal(sim.fields(), ref.fields())
