"""Materials that reach through the CPML slabs to the walls, in the sweep against the two-pass schedule, bit for bit: quads of
one row in the slabs and on the low walls, with and without magnetic materials (where there are none, no H update looks at its
row), large blocks so that most quads are of one row, and a background whose H coefficients differ from the default entry's."""
import pytest

from fdtd_gb300 import scenario as S
from test_gpu_sweep import case, check

pytestmark = pytest.mark.gpu


def blocks(dims, pml, seed, magnetic, background=None):
    """test_gpu_sweep's case with its bricks replaced by slabs of the whole grid: four layers along z, half of one along x."""
    sc = case(dims, pml, seed, n_sources=3, background=background)
    nx, ny, nz = dims
    mats = [S.Material(eps_r=1.5 + q, sigma_e=0.01 * q, **(dict(mu_r=1.0 + 0.3 * q, sigma_m=20.0 * q + 5) if magnetic else {}))
            for q in range(4)]
    sc.materials = [sc.materials[0]] + mats
    z = [0, nz // 5, nz // 3, nz // 2, nz]
    sc.bricks = [S.Brick((0, 0, z[0], nx, ny, z[1]), 1), S.Brick((0, 0, z[2], nx, ny, z[3]), 2),
                 S.Brick((0, 0, z[3], nx // 2, ny, z[4]), 3), S.Brick((nx // 3, ny // 2, z[1], nx, ny, z[3]), 4)]
    return sc


@pytest.mark.parametrize("dims,pml", [
    ((64, 48, 40), (6, 7, 5, 8, 4, 9)),
    ((97, 61, 40), (0, 5, 0, 6, 7, 0)),
    ((33, 17, 33), (4, 5, 3, 6, 2, 7)),
    ((40, 36, 34), (0,) * 6),
    ((130, 210, 45), (5, 4, 8, 7, 6, 6)),  # more CTAs than the two-per-SM kernel takes
    ((7, 9, 11), (3, 3, 4, 4, 5, 5)),
])
@pytest.mark.parametrize("magnetic", [False, True])
def test_layers_equal_two_pass(gpu_lib, dims, pml, magnetic):
    check(blocks(dims, pml, sum(dims), magnetic))


@pytest.mark.parametrize("magnetic", [False, True])
def test_layers_magnetic_background(gpu_lib, magnetic):
    for dims in ((70, 50, 44), (150, 200, 48)):
        check(blocks(dims, (6, 5, 7, 4, 5, 6), 3, magnetic, S.Material(eps_r=2.0, sigma_e=0.01, mu_r=1.5, sigma_m=40.0)), calls=(3, 4))


@pytest.mark.parametrize("dims", [(65, 33, 40), (150, 200, 48)])
def test_boxes_without_magnetic_materials(gpu_lib, dims):
    sc = case(dims, (10, 9, 8, 7, 6, 5), 5, n_sources=11, plates=True)
    sc.materials = [S.Material(eps_r=m.eps_r, sigma_e=m.sigma_e) for m in sc.materials]
    check(sc)
