"""The two forms of the split weno_Re_flux gradient kernel
(visc_gradients_tiled, csrc/mfc_visc_grad.cu): the coefficients that all cells
of a uniform grid share, and per-cell ones.  A grid whose last cell alone is
wider takes the second form; away from that cell both must give the same bits.

And the viscous change of the first against plain FP64's: the change is 1e-3 of
the momenta or more and FP32 rounds them at 1e-7, so the two agree to some
1e-4; nonlinear weights that react to rounding may raise it by ten."""
import numpy as np
import pytest

from microfc_gb300 import cases, preprocess

pytestmark = pytest.mark.gpu

VISCOUS = dict(re_shear=(10.0, 10.0), re_bulk=(0.0, 20.0), weno_re_flux=True)


def _steps(c, x, y, z, q, n):
    from microfc_gb300 import Simulation
    with Simulation(c, x, y, z, q_cons=q) as sim:
        for _ in range(n):
            sim.tvd_rk(0, c.dt)
        return sim.download()


@pytest.mark.parametrize("prec", ["split", "gated"])
@pytest.mark.parametrize("nx,ny", [(64, 96), (97, 75)])
@pytest.mark.parametrize("axis", [0, 1])
def test_shared_and_per_cell_coefficients_agree(nx, ny, axis, prec):
    from microfc_gb300 import Simulation, gate
    c = cases.shock_droplet_2d(nx=nx, ny=ny, steps=1, mach=1.2, precision=prec).replace(**VISCOUS)
    x, y, z, q = preprocess.generate(c)
    outs = []
    for wider in (False, True):
        b = [x.copy(), y.copy()]
        if wider:
            b[axis][-1] += 0.25 * (b[axis][-1] - b[axis][-2])
        with Simulation(c, b[0], b[1], z, q_cons=q) as sim:
            if prec == "gated":
                sim.set_gate(gate.load())
            sim.tvd_rk(0, c.dt)
            outs.append(sim.download())
    keep = (slice(None), slice(None), slice(None, ny - 24 if axis else None), slice(None, None if axis else nx - 24))
    a, b = (np.ascontiguousarray(o[keep]) for o in outs)
    assert np.isfinite(a).all()
    assert np.array_equal(a.view(np.uint64), b.view(np.uint64))


@pytest.mark.parametrize("nx,ny,bcx,bcy", [(64, 33, (-1, -1), (-3, -3)), (97, 48, (-2, -3), (-1, -1))])
def test_viscous_change_is_that_of_fp64(nx, ny, bcx, bcy):
    base = cases.shock_droplet_2d(nx=nx, ny=ny, steps=2, mach=1.2).replace(bc_x=bcx, bc_y=bcy)
    x, y, z, q = preprocess.generate(base)
    change = []
    for prec in ("fp64", "split"):
        c = base.replace(precision=prec)
        change.append(_steps(c.replace(**VISCOUS), x, y, z, q, 2)[2:4] - _steps(c, x, y, z, q, 2)[2:4])
    want, got = change
    assert np.abs(got - want).sum() <= 1e-3 * np.abs(want).sum()
