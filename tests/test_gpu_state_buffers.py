"""Fields and states set while the fused schedule's state lies in either buffer: the steps after them equal the two-pass
schedule's, bit for bit, and so does the state saved then."""
import numpy as np
import pytest

from test_gpu_sweep import case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,pml", [((33, 17, 20), (4, 5, 3, 6, 2, 7)), ((64, 40, 36), (6,) * 6)])
def test_set_and_load_in_either_buffer(gpu_lib, dims, pml):
    import torch
    from fdtd_gb300 import solver
    sc = case(dims, pml, 12)
    gen = torch.Generator(device="cuda").manual_seed(4)
    fields = [torch.rand(dims[::-1], generator=gen, device="cuda") - 0.5 for _ in range(6)]
    torch.cuda.synchronize()
    out = []
    for schedule in (1, 2):
        with solver.Simulation.from_scenario(sc, schedule, probe_capacity=64) as sim:
            size = sim.state_bytes()
            saved, last = (torch.zeros(size, dtype=torch.uint8, device="cuda") for _ in range(2))
            torch.cuda.synchronize()
            for q, n in enumerate((1, 2, 3)):  # an odd count: the buffers change
                for c, f in enumerate(fields):
                    if (c + q) % 2:
                        sim.set_field_device(c, f.data_ptr())
                    else:
                        sim.set_field(c, f.cpu().numpy())
                sim.step(n)
                if q == 1:
                    sim.save_state(saved.data_ptr())
            sim.load_state(saved.data_ptr())
            sim.step(5)
            sim.load_state(saved.data_ptr())
            sim.step(4)
            sim.save_state(last.data_ptr())
            torch.cuda.synchronize()
            out.append((last, sim.read_probes(3, 4)))
    assert torch.equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
    assert np.abs(out[0][1]).max() > 0
