"""Plain FP64 3-D grids that whole fixed tiles cover, on both sides of the six
waves from which the default takes them (csrc/stage_3d_fp64.cu): the line, and
the bits of the default and of the fixed tiles."""
import numpy as np
import pytest

from microfc_gb300 import cases, preprocess

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz,fixed", [(96, 64, 64, False), (96, 80, 64, True), (64, 96, 80, True), (96, 80, 63, False)])
def test_default_across_the_line(nx, ny, nz, fixed):
    from microfc_gb300 import Simulation
    c = cases.shock_bubble_3d(N=64, steps=1, precision="fp64").replace(m=nx - 1, n=ny - 1, p=nz - 1, bc_y=(-2, -4))
    c = c.replace(dt=c.dt / 4)
    x, y, z, q = preprocess.generate(c)
    outs, shapes = [], []
    for v in (0, 1):
        with Simulation(c, x, y, z, q_cons=q) as sim:
            shapes.append(tuple(sim.select_variant(v)))
            sim.tvd_rk(0, c.dt)
            outs.append(sim.download())
    assert (shapes[0] == shapes[1]) == fixed
    assert np.array_equal(outs[0].view(np.uint64), outs[1].view(np.uint64))
