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
