"""Split-precision stages hand the next stage the FP32 primitives of the state
they make (PrimPairs, csrc/mfc_pair.cuh).  A run that carries them must give
the bits of one whose state is uploaded anew before every step, so that each
step's first stage converts the FP64 state itself; partial tiles, every
boundary condition and both tile sizes are covered."""
import numpy as np
import pytest

from microfc_gb300 import cases, gate, preprocess

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,viscous", [("split", False), ("gated", False), ("split", True)])
@pytest.mark.parametrize("nx,ny,bcx,bcy", [(33, 31, (-3, -3), (-2, -4)), (47, 64, (-1, -1), (-3, -3)),
                                           (400, 209, (-4, -2), (-1, -1))])
def test_carried_pairs_give_the_bits_of_a_fresh_state(nx, ny, bcx, bcy, prec, viscous):
    from microfc_gb300 import Simulation
    c = cases.shock_droplet_2d(nx=nx, ny=ny, steps=3, precision=prec, mach=1.2).replace(bc_x=bcx, bc_y=bcy)
    if viscous:
        c = c.replace(re_shear=(10.0, 500.0), re_bulk=(0.0, 200.0))
    x, y, z, q = preprocess.generate(c)
    with Simulation(c, x, y, z, q_cons=q) as sim:
        if prec == "gated":
            sim.set_gate(gate.load())
        for _ in range(3):
            sim.tvd_rk(0, c.dt)
        carried = sim.download()
        rhs, _ = sim.s_compute_rhs()
        sim.upload(carried)
        fresh_rhs, _ = sim.s_compute_rhs()
        sim.upload(q)
        for _ in range(3):
            sim.tvd_rk(0, c.dt)
            sim.upload(sim.download())
        fresh = sim.download()
    assert np.array_equal(carried.view(np.uint64), fresh.view(np.uint64))
    assert np.array_equal(rhs.view(np.uint64), fresh_rhs.view(np.uint64))
