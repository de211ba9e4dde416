"""Plain FP64 on tiles sized at run time (csrc/mfc_flex.cuh): grids of the
smallest extents, one cell more or less than a multiple of the SM count, and
long thin ones give the oracle's bits under every boundary condition, so
partial tiles, tile edges and the faces between tiles are right."""
import numpy as np
import pytest

from microfc_gb300 import cases, preprocess

pytestmark = pytest.mark.gpu


def _run(case, steps):
    import oracle
    from microfc_gb300 import Simulation
    x, y, z, q = preprocess.generate(case)
    o = oracle.Oracle(case, x, y, z)
    o.set_state(q)
    o.run(0, steps, case.dt)
    with Simulation(case, x, y, z, q_cons=q) as sim:
        sim.run(0, steps)
        return sim.download(), o.get_state()


@pytest.mark.parametrize("order", [1, 3, 5])
@pytest.mark.parametrize("cells,bc", [(25, (-3, -3)), (151, (-2, -4)), (153, (-1, -1)), (3041, (-4, -2))])
def test_1d_sizes(cells, bc, order):
    c = cases.sod_1d(m=cells - 1, steps=3, dt=1e-5).replace(weno_order=order, bc_x=bc)
    got, want = _run(c, 3)
    assert np.array_equal(got.view(np.uint64), want.view(np.uint64))


@pytest.mark.parametrize("viscous", [False, True])
@pytest.mark.parametrize("nx,ny,bcx,bcy", [(25, 25, (-3, -3), (-3, -3)), (40, 201, (-4, -3), (-2, -4)),
                                           (305, 26, (-4, -2), (-1, -1)), (153, 152, (-2, -3), (-4, -3))])
def test_2d_sizes(nx, ny, bcx, bcy, viscous):
    c = cases.shock_droplet_2d(nx=nx, ny=ny, steps=2).replace(bc_x=bcx, bc_y=bcy)
    if viscous:
        c = c.replace(re_shear=(10.0, 500.0), re_bulk=(0.0, 200.0))
    got, want = _run(c, 2)
    assert np.array_equal(got.view(np.uint64), want.view(np.uint64))


@pytest.mark.parametrize("order", [1, 3, 5])
@pytest.mark.parametrize("nx,ny,nz,bcx,bcy,bcz",
                         [(25, 26, 27, (-3, -3), (-2, -4), (-1, -1)), (161, 25, 33, (-4, -2), (-1, -1), (-2, -3)),
                          (31, 97, 25, (-2, -3), (-4, -4), (-3, -4))])
def test_3d_sizes(nx, ny, nz, bcx, bcy, bcz, order):
    c = cases.shock_bubble_3d(N=28, steps=2, precision="fp64")
    c = c.replace(m=nx - 1, n=ny - 1, p=nz - 1, dt=c.dt / 8, bc_x=bcx, bc_y=bcy, bc_z=bcz, weno_order=order)
    got, want = _run(c, 2)
    assert np.array_equal(got.view(np.uint64), want.view(np.uint64))
