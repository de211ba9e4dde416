"""Plain FP64 3-D WENO5 on both sides of the line between tiles sized for the
grid and whole fixed tiles (csrc/stage_3d_fp64.cu): both compiled variants and
the default give the same bits, and the default takes the fixed tiles only
where whole ones cover the grid."""
import numpy as np
import pytest

from microfc_gb300 import cases, preprocess

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz,fixed", [(160, 96, 96, True), (160, 96, 95, False), (64, 64, 64, False)])
def test_default_and_variants_agree(nx, ny, nz, fixed):
    from microfc_gb300 import Simulation
    c = cases.shock_bubble_3d(N=64, steps=1, precision="fp64").replace(m=nx - 1, n=ny - 1, p=nz - 1)
    c = c.replace(dt=c.dt / 4, bc_y=(-2, -3), bc_z=(-4, -3))
    x, y, z, q = preprocess.generate(c)
    outs, shapes = [], []
    for v in (None, 0, 1):
        with Simulation(c, x, y, z, q_cons=q) as sim:
            if v is not None:
                shapes.append(tuple(sim.select_variant(v)))
            sim.tvd_rk(0, c.dt)
            outs.append(sim.download())
    assert np.isfinite(outs[0]).all()
    assert (shapes[0] == shapes[1]) == fixed
    for o in outs[1:]:
        assert np.array_equal(o.view(np.uint64), outs[0].view(np.uint64))
