"""The split-precision 3-D sweeps on pairs (csrc/mfc_pair_sweep.cuh), at grids
around their 16-cell tiles, with every kind of boundary.  First: two steps against
plain FP64 (other kernels, bit-identical to the oracle).

Tolerance: the sweeps' fluxes carry FP32 rounding (1e-7, some ten operations
deep) against changes that are of the fluxes' order in the shock's cells, a
tenth of the domain, so the L1 distance of the two changes is some 1e-5 of the
change; nonlinear weights that react to rounding in quiet cells may raise it by
ten.  A wrong row of a tile is at least one face in seventeen, order 1e-2.  The
volume fractions are left out: the shock has not met the bubble, so their
change is itself of the size of the rounding."""
import numpy as np
import pytest

from microfc_gb300 import cases, preprocess

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz,bcy,bcz", [(33, 31, 26, (-3, -3), (-2, -4)), (26, 48, 33, (-2, -3), (-1, -1)),
                                              (47, 27, 50, (-1, -1), (-4, -2)), (64, 64, 64, (-3, -3), (-3, -3))])
@pytest.mark.parametrize("uniform", [True, False], ids=["uniform", "records"])
def test_changes_match_fp64(nx, ny, nz, bcy, bcz, uniform):
    from microfc_gb300 import Simulation
    base = cases.shock_bubble_3d(N=64, steps=2).replace(m=nx - 1, n=ny - 1, p=nz - 1, bc_y=bcy, bc_z=bcz)
    x, y, z, q = preprocess.generate(base)

    def change(prec):
        with Simulation(base.replace(precision=prec), x, y, z, q_cons=q) as sim:
            if prec == "split":
                sim.set_uniform_coefficients(uniform)
            for _ in range(2):
                sim.tvd_rk(0, base.dt)
            return sim.download() - q

    want, got = change("fp64"), change("split")
    assert np.isfinite(want).all()
    for rows in (slice(0, 2), slice(2, 5), slice(5, 6)):  # densities, momenta, energy
        assert np.abs(got[rows] - want[rows]).sum() <= 1e-3 * np.abs(want[rows]).sum()


@pytest.mark.parametrize("nx,ny,nz,bcx,bcy", [(33, 31, 26, (-3, -3), (-2, -4)), (48, 26, 33, (-1, -1), (-3, -2))])
def test_carried_pairs_give_the_bits_of_a_fresh_state(nx, ny, nz, bcx, bcy):
    """Steps on the primitive pairs that the last stage stored, against steps
    whose first stage converts an uploaded state; exact."""
    from microfc_gb300 import Simulation
    c = cases.shock_bubble_3d(N=64, steps=2).replace(m=nx - 1, n=ny - 1, p=nz - 1, bc_x=bcx, bc_y=bcy,
                                                     precision="split")
    x, y, z, q = preprocess.generate(c)
    with Simulation(c, x, y, z, q_cons=q) as sim:
        for _ in range(3):
            sim.s_compute_rhs()  # must not disturb the stored pairs
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
