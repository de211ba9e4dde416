"""The range of the split weno_Re_flux reconstruction (grad_weno in
csrc/mfc_visc_grad.cu), whose FP32 divisors are squares: a small weno_eps where
the velocity is uniform, and a velocity gradient that jumps by 1e11 1/s, on a
uniform grid (shared coefficients) and on a stretched one (per-cell ones).

What the viscous terms change in the momenta must be what they change in plain
FP64, whose gradients come from other kernels and cannot leave their range.
Tolerance: a gradient that is not a number ends the run, a face that took a
wrong one differs by order one; FP32 rounds the momenta at 1e-7 and the viscous
change is 4e-4 of them (first test) or 1e-2 (second), so the two agree to about
1e-3 and 1e-4."""
import numpy as np
import pytest

from microfc_gb300 import cases, preprocess

pytestmark = pytest.mark.gpu


def _stretched(cb):
    t = np.linspace(0.0, 1.0, len(cb))
    return cb[0] + (cb[-1] - cb[0]) * (t + 0.02 * np.sin(2.0 * np.pi * t))


def _viscous_change(base, x, y, z, q, re):
    from microfc_gb300 import Simulation

    def momenta(prec, viscous):
        c = base.replace(precision=prec)
        if viscous:
            c = c.replace(weno_re_flux=True, **re)
        with Simulation(c, x, y, z, q_cons=q) as sim:
            for _ in range(2):
                sim.tvd_rk(0, c.dt)
            return sim.download()[2:4]

    out = []
    for prec in ("fp64", "split"):
        out.append(momenta(prec, True) - momenta(prec, False))
        assert np.isfinite(out[-1]).all(), prec
    return out


@pytest.mark.parametrize("stretch", [False, True], ids=["uniform", "stretched"])
@pytest.mark.parametrize("eps", [1e-16, 1e-18, 1.2e-19])
def test_small_weno_eps(eps, stretch):
    base = cases.shock_droplet_2d(nx=64, ny=40, steps=2, mach=1.2).replace(weno_eps=eps, bc_y=(-2, -3))
    x, y, z, q = preprocess.generate(base)
    if stretch:
        x, y = _stretched(x), _stretched(y)
        base = base.replace(dt=0.7 * base.dt)
    want, got = _viscous_change(base, x, y, z, q, dict(re_shear=(10.0, 10.0), re_bulk=(0.0, 20.0)))
    assert np.abs(want).sum() > 0
    assert np.abs(got - want).sum() <= 1e-2 * np.abs(want).sum()


@pytest.mark.parametrize("stretch", [False, True], ids=["uniform", "stretched"])
def test_gradient_jump(stretch):
    """Air at rest below, sheared above: u rises by 10 m/s a cell of 0.1 nm."""
    h = 1e-10
    base = cases.shock_droplet_2d(nx=40, ny=64, steps=2, dt=5e-14).replace(
        x_domain=(0.0, 40 * h), y_domain=(0.0, 64 * h), bc_x=(-1, -1), bc_y=(-3, -3))
    x, y, z = preprocess.grid(base)
    if stretch:
        y = _stretched(y)
    yc = 0.5 * (y[1:] + y[:-1])
    gam = base.gammas[1]
    q = np.zeros(base.shape)
    u = 1e11 * np.maximum(yc - 32 * h, 0.0)[None, :, None]
    q[1], q[6] = 1.2, 1.0
    q[2] = 1.2 * u
    q[4] = gam * 1e5 + 0.6 * u * u
    want, got = _viscous_change(base, x, y, z, q, dict(re_shear=(1e7, 1e7)))
    assert np.abs(want[0]).max() > 1e-2 * np.abs(q[2]).max()
    assert np.abs(got - want).sum() <= 1e-3 * np.abs(want).sum()
