"""Steps under AUTO and stream capture: a captured call can be replayed between others, also where AUTO had taken the sweep
before, and the allocation of the sweep's buffers leaves a capture elsewhere in the program alone."""
import numpy as np
import pytest

from conftest import bitwise_equal
from fdtd_gb300 import scenario as S

pytestmark = pytest.mark.gpu


def make(n, schedule, stream):
    import torch
    from fdtd_gb300 import solver
    sc = S.vacuum_cube(n, 8, pml=6, name="capture")
    sc.sources, sc.probes = [], []  # a captured call replays its steps' signals and probe rows
    sim = solver.Simulation.from_scenario(sc, schedule)
    sim.set_stream(stream.cuda_stream)
    gen = torch.Generator(device="cuda").manual_seed(2)
    for c in range(6):
        f = torch.rand((n, n, n), generator=gen, device="cuda") - 0.5
        torch.cuda.synchronize()
        sim.set_field_device(c, f.data_ptr())
        torch.cuda.synchronize()
    sim.prepare()
    return sim


@pytest.mark.parametrize("before", [1, 401])  # two-pass still, or the sweep's buffers in use, the state in the second
@pytest.mark.parametrize("count", [1, 2])
def test_replayed_steps(gpu_lib, before, count):
    import torch
    stream = torch.cuda.Stream()
    n = 48
    with make(n, 0, stream) as sim, make(n, 1, stream) as ref:
        sim.step(before)
        torch.cuda.synchronize()
        assert sim.active_schedule == (2 if before > 100 else 1)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            sim.step(count)
        with torch.cuda.stream(stream):
            graph.replay()
            graph.replay()
            sim.step(3)
            graph.replay()
            sim.step(401)
            graph.replay()
        torch.cuda.synchronize()
        ref.step(before + 4 * count + 404)
        torch.cuda.synchronize()
        assert np.abs(ref.fields()).max() > 0 and bitwise_equal(sim.fields(), ref.fields())


def test_buffers_during_a_capture_elsewhere(gpu_lib):
    import torch
    stream = torch.cuda.Stream()
    with make(64, 0, stream) as sim, make(64, 1, stream) as ref:
        x = torch.zeros(16, device="cuda")
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):  # on a stream of its own; global capture mode
            x.add_(1)
            sim.step(1000)
            x.mul_(2)
        assert sim.active_schedule == 2
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(x, torch.full_like(x, 2))
        ref.step(1000)
        torch.cuda.synchronize()
        assert bitwise_equal(sim.fields(), ref.fields())
