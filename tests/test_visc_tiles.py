"""The tiled velocity-gradient kernel of split weno_Re_flux runs
(csrc/mfc_visc_grad.cu), at grids around its 32x16 tiles: what the viscous
terms change in the momenta must be what they change in plain FP64 (whose
gradients come from other kernels, bit-identical to the oracle).

Tolerance: the viscous change is some 1e-2 of the momenta here and FP32 rounds
them at 1e-7, so the two changes agree to about 1e-4; a face that took a wrong
gradient differs by order one, and a wrong row or column per tile is at least
1/32 of the faces."""
import numpy as np
import pytest

from microfc_gb300 import cases, preprocess

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stretch", [False, True], ids=["uniform", "stretched"])
@pytest.mark.parametrize("nx,ny,bcx,bcy", [(31, 32, (-3, -3), (-2, -3)), (64, 33, (-1, -1), (-3, -3)),
                                           (97, 48, (-2, -3), (-1, -1))])
def test_viscous_change_matches_fp64(nx, ny, bcx, bcy, stretch):
    from microfc_gb300 import Simulation
    base = cases.shock_droplet_2d(nx=nx, ny=ny, steps=2, mach=1.2).replace(bc_x=bcx, bc_y=bcy)
    x, y, z, q = preprocess.generate(base)
    if stretch:  # the same state on a stretched grid (the patches cover the uniform one only)
        x, y, z = preprocess.grid(base.replace(stretch_y=(12.0, 0.004, 0.006, 1)))

    def momenta(prec, viscous):
        c = base.replace(precision=prec)
        if viscous:
            c = c.replace(re_shear=(10.0, 10.0), re_bulk=(0.0, 20.0), weno_re_flux=True)
        with Simulation(c, x, y, z, q_cons=q) as sim:
            for _ in range(2):
                sim.tvd_rk(0, c.dt)
            return sim.download()[2:4]

    want = momenta("fp64", True) - momenta("fp64", False)
    got = momenta("split", True) - momenta("split", False)
    assert np.abs(want).sum() > 0
    assert np.abs(got - want).sum() <= 1e-2 * np.abs(want).sum()
