"""When a batch's instances get the sweep's second buffers: not for a call of a few steps, together once the steps asked of the
batch repay them, and in memory that outlives the handles that were closed first."""
import pytest

from conftest import bitwise_equal
from test_gpu_sweep import case

pytestmark = pytest.mark.gpu

DIMS = [(96, 96, 96), (97, 90, 95), (100, 96, 92), (96, 99, 94), (20, 20, 20)]  # the last below the sweep's size


def sims_of(schedules):
    import torch
    from fdtd_gb300 import solver
    out = []
    gen = torch.Generator(device="cuda").manual_seed(3)
    for q, (dims, s) in enumerate(zip(DIMS, schedules)):
        sc = case(dims, (6,) * 6, 40 + q, materials=False)
        sim = solver.Simulation.from_scenario(sc, s, probe_capacity=128)
        for c in range(6):
            f = torch.rand(dims[::-1], generator=gen, device="cuda") - 0.5
            sim.set_field_device(c, f.data_ptr())
            torch.cuda.synchronize()
        sim.prepare()
        out.append(sim)
    return out


def test_second_buffers_of_a_batch(gpu_lib):
    from fdtd_gb300 import solver
    sims, alone = sims_of([0, 0, 1, 0, 0]), sims_of([1] * 5)
    try:
        before = [s.device_bytes() for s in sims]
        batch = solver.Batch(sims)
        batch.step(2)
        batch.synchronize()
        assert [s.device_bytes() for s in sims] == before  # two steps repay nothing
        batch.step(61)
        batch.synchronize()
        grown = [b > a for a, b in zip(before, [s.device_bytes() for s in sims])]
        assert grown == [True, True, False, True, False]  # not the one under TWO_PASS, nor the small one
        batch.close()
        sims[0].close()  # the others' buffers stay
        sims[1].close()
        for s in sims[2:]:
            s.step(4)
        for s in alone:
            s.step(67)
        for s, t in zip(sims[2:], alone[2:]):
            assert bitwise_equal(s.fields(), t.fields())
            assert bitwise_equal(s.read_probes(0, 67), t.read_probes(0, 67))
    finally:
        for s in sims + alone:
            s.close()


def test_fused_instances_at_once(gpu_lib):
    from fdtd_gb300 import solver
    sims, alone = sims_of([2, 0, 2, 2, 2]), sims_of([1] * 5)
    try:
        before = [s.device_bytes() for s in sims]
        with solver.Batch(sims) as batch:
            batch.step(1)
            batch.synchronize()
            assert [b > a for a, b in zip(before, [s.device_bytes() for s in sims])] == [True, False, True, True, False]
            batch.step(2)
            batch.synchronize()
        for s, t in zip(sims, alone):
            t.step(3)
            assert bitwise_equal(s.fields(), t.fields())
    finally:
        for s in sims + alone:
            s.close()
