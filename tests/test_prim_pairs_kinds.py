"""Carried primitive pairs (PrimPairs, csrc/mfc_pair.cuh) on stretched grids, of
gated viscous runs and of runs with WENO velocity gradients: the bits of a run
whose state is uploaded anew before every step."""
import numpy as np
import pytest

from microfc_gb300 import cases, gate, preprocess

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["split", "gated", "viscous", "gated_viscous", "weno_re_flux", "gated_weno_re_flux"])
@pytest.mark.parametrize("stretch", [False, True], ids=["uniform", "stretched"])
@pytest.mark.parametrize("nx,ny", [(47, 61), (321, 209)])
def test_carried_pairs_give_the_bits_of_a_fresh_state(nx, ny, stretch, kind):
    from microfc_gb300 import Simulation
    gated = kind.startswith("gated")
    c = cases.shock_droplet_2d(nx=nx, ny=ny, steps=3, precision="gated" if gated else "split", mach=1.2)
    c = c.replace(bc_x=(-4, -2), bc_y=(-2, -3), dt=0.5 * c.dt)
    if kind.endswith("viscous") or kind.endswith("weno_re_flux"):
        c = c.replace(re_shear=(10.0, 500.0), re_bulk=(0.0, 200.0), weno_re_flux=kind.endswith("weno_re_flux"))
    x, y, z, q = preprocess.generate(c)
    if stretch:
        t = [np.linspace(0.0, 1.0, len(b)) for b in (x, y)]
        x, y = (b[-1] * (s + 0.03 * np.sin(2.0 * np.pi * s)) for b, s in zip((x, y), t))
    with Simulation(c, x, y, z, q_cons=q) as sim:
        if gated:
            sim.set_gate(gate.load())
        for _ in range(3):
            sim.tvd_rk(0, c.dt)
        carried = sim.download()
        sim.upload(q)
        for _ in range(3):
            sim.tvd_rk(0, c.dt)
            sim.upload(sim.download())
        fresh = sim.download()
    assert np.isfinite(carried).all()
    assert np.array_equal(carried.view(np.uint64), fresh.view(np.uint64))
