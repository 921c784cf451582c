"""Lumped elements on the top face of a design region: their Ez edges touch no design cell, but the Ex and Ey of their nodes do
(the nodes lie in the region's edge box). Forward and gradient against the oracle, and the refusal of elements that do touch."""
import numpy as np
import pytest

import oracle
from conftest import bitwise_equal
from fdtd_gb300 import scenario as S
from test_gpu_adjoint import GRAD_TOL, design_case, gpu_grad, rel

pytestmark = pytest.mark.gpu


def top_face_case(steps=120, dims=(24, 22, 20)):
    sc, box, eps, probe = design_case(3, steps=steps)
    sc.nx, sc.ny, sc.nz = dims
    z = box[5]
    sc.sources = [S.LumpedSource((11, 10, z, 12, 11, z + 2), 50.0, S.gaussian_derivative(steps, sc.dt, 30e9, 1e-3))]
    sc.resistors = [S.Resistor((box[3], box[4], z, box[3], box[4], z + 1), 75.0)]  # on an edge of the face
    return sc, box, eps, probe


@pytest.mark.parametrize("schedule,dims,steps", [(1, (24, 22, 20), 120), (2, (24, 22, 20), 120), (2, (90, 60, 40), 40),
                                                  (1, (200, 196, 192), 6)])  # the last: the kernels by node class
def test_forward_bitwise(gpu_lib, schedule, dims, steps):
    from fdtd_gb300 import solver
    sc, box, eps, _ = top_face_case(steps, dims)
    with solver.Simulation.from_scenario(sc, schedule, probe_capacity=steps) as sim:
        sim.set_design_region(box, eps)
        sim.step(steps)
        sim.synchronize()
        p, f, prof = sim.read_probes(0, steps), sim.fields(), sim.cpml_profiles()
    po, fo = oracle.run(sc, profile_override=prof, design=(box, eps.astype(np.float64)))
    assert np.abs(fo).max() > 0
    assert bitwise_equal(p, po) and bitwise_equal(f, fo)


@pytest.mark.parametrize("schedule", [1, 2])
def test_gradient(gpu_lib, schedule):
    from fdtd_gb300 import solver
    sc, box, eps, probe = top_face_case()
    J64, g64 = oracle.fom_grad(sc, probe, box, eps.astype(np.float64), precision="f64")
    grads = []
    for K in (0, 16):
        with solver.Simulation.from_scenario(sc, schedule, probe_capacity=sc.steps) as sim:
            sim.set_design_region(box, eps)
            J = sim.adjoint_forward(sc.steps, probe, K)
            grads.append(sim.adjoint_backward())
        assert abs(J - J64) <= 1e-4 * abs(J64)
        assert rel(grads[-1], g64) < GRAD_TOL
    assert np.array_equal(*grads)
    top = grads[0][-1], g64[-1]  # the cells under the face
    assert rel(*top) < GRAD_TOL


def test_fom_probe_on_the_source(gpu_lib):
    """The figure of merit's probe on the source's own edge, a node of the edge box: its record is taken there."""
    sc, box, eps, _ = top_face_case(80)
    probe = (11, 10, box[5])
    J, g = gpu_grad(sc, box, eps, probe, 8)
    J64, g64 = oracle.fom_grad(sc, probe, box, eps.astype(np.float64), precision="f64")
    assert abs(J - J64) <= 1e-4 * abs(J64) and rel(g, g64) < GRAD_TOL


def test_elements_that_touch_are_refused_in_either_order(gpu_lib):
    from fdtd_gb300 import solver
    sc, box, eps, _ = top_face_case()
    wave = np.ones(4, np.float32)
    with solver.Simulation.from_scenario(sc) as sim:
        sim.set_design_region(box, eps)
        for bad in ((12, 11, box[5] - 1, 12, 11, box[5]), (box[3], 9, box[2], box[3], 9, box[2] + 1)):
            for add in (lambda: sim.add_source(bad, 50.0, wave), lambda: sim.add_resistor(bad, 50.0)):
                with pytest.raises(solver.FDTDError) as e:
                    add()
                assert e.value.code == 1
        sim.add_source((box[0] - 1, 9, box[2], box[0] - 1, 9, box[2] + 1), 50.0, wave)  # beside it
        sim.add_resistor((13, 9, box[5], 13, 9, box[5] + 1), 50.0)                      # on its top face
        sim.step(2)
        sim.synchronize()
