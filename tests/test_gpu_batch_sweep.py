"""The batch's chain form in a batch large enough for the sweep (kBatchSweepCells), its instances on both
sides of kAutoSweepCells and on either schedule, against each instance alone on the two-pass schedule,
bit for bit: odd and even calls, so that states change buffers between and inside the captured
chunks, and instances stepped alone in between."""
import pytest

from conftest import bitwise_equal
from test_gpu_sweep import case

pytestmark = pytest.mark.gpu

DIMS = [((32, 32, 32), (4,) * 6), ((31, 32, 33), (5,) * 6), ((65, 33, 40), (10, 9, 8, 7, 6, 5)), ((12, 14, 16), (3,) * 6),
        ((140, 138, 135), (8,) * 6), ((40, 36, 34), (0,) * 6)]


def drive(scs, schedules, calls, alone, form):
    import torch
    from fdtd_gb300 import solver
    sims = [solver.Simulation.from_scenario(sc, s, probe_capacity=128) for sc, s in zip(scs, schedules)]
    try:
        gen = torch.Generator(device="cuda").manual_seed(7)
        for sim, sc in zip(sims, scs):
            for c in range(6):
                f = torch.rand((sc.nz, sc.ny, sc.nx), generator=gen, device="cuda") - 0.5
                sim.set_field_device(c, f.data_ptr())
                torch.cuda.synchronize()
        total = sum(calls) + sum(alone)
        if form is None:
            for sim in sims:
                sim.step(total)
        else:
            with solver.Batch(sims) as batch:
                batch.set_config(*form)
                for n, a in zip(calls, alone):
                    batch.step(n)
                    batch.synchronize()
                    if a:
                        for sim in sims:
                            sim.step(a)
        out = []
        for sim in sims:
            buf = torch.empty(sim.state_bytes(), dtype=torch.uint8, device="cuda")
            torch.cuda.synchronize()
            sim.save_state(buf.data_ptr())
            torch.cuda.synchronize()
            out.append((sim.read_probes(0, total), buf))
        return out
    finally:
        for sim in sims:
            sim.close()


@pytest.mark.parametrize("schedule", [0, 2])
@pytest.mark.parametrize("calls,alone", [((33, 2, 5), (1, 0, 2)), ((1, 1, 1, 1, 3, 3), (0,) * 6), ((64, 37), (0, 0))])
def test_chains_equal_two_pass(gpu_lib, schedule, calls, alone):
    import torch
    scs = [case(d, pml, 11 + q, n_sources=11 if q == 2 else 3) for q, (d, pml) in enumerate(DIMS)]
    want = drive(scs, [1] * len(scs), calls, alone, None)
    got = drive(scs, [schedule] * (len(scs) - 1) + [1], calls, alone, (-1, 256))
    for (p, s), (q, t) in zip(got, want):
        assert bitwise_equal(p, q)
        assert torch.equal(s, t)
