"""The upwind choice of the plain FP64 HLLC face (hllc_face in
csrc/mfc_device.cuh: one set of formulas on the chosen side, minima and maxima
on the bits) against the oracle, exactly: faces supersonic to either side, at
rest, mirrored, with mixed and one-sided mixtures, zero volume fractions of
either sign, and states that are not a number."""
import numpy as np
import pytest

from microfc_gb300 import Simulation, cases, preprocess

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [0, 1])
@pytest.mark.parametrize("bad", [False, True], ids=["finite", "nan"])
def test_faces_of_every_kind_match_the_oracle(oracle_lib, d, bad):
    case = cases.shock_droplet_2d(nx=64, ny=40, steps=2)
    x, y, z, q = preprocess.generate(case)
    o = oracle_lib.Oracle(case, x, y, z)
    o.set_state(q)
    rng = np.random.default_rng(7)
    shape = o.weno(d)[0].shape

    def states():
        p = np.empty(shape)
        a = rng.choice([0.0, -0.0, 1e-8, 0.5, 1.0], shape[1:])
        p[0], p[1] = 1000.0 * np.abs(a) + 1e-3, 1.2 * (1.0 - np.abs(a)) + 1e-3
        for v in (2, 3):
            p[v] = rng.choice([0.0, -0.0, 30.0, -30.0, 9000.0, -9000.0], shape[1:])
        p[4] = rng.choice([1.0, 1e5, 3e8], shape[1:])
        p[5], p[6] = a, 1.0 - np.abs(a)
        if bad:
            for v in range(7):
                p[v][rng.random(shape[1:]) < 0.02] = np.nan
        return p

    left, right = states(), states()
    mirrored = rng.random(shape[1:]) < 0.2  # both sides alike but for the velocity's sign
    right[:, mirrored] = left[:, mirrored]
    right[2 + d][mirrored] *= -1.0
    with np.errstate(all="ignore"):
        flux, src = o.riemann(d, left, right)
    with Simulation(case, x, y, z, q_cons=q) as sim:
        got, got_src = sim.s_hllc_riemann_solver(d, left, right)
    # (the oracle adds zero times the downwind side, the kernel leaves it out:
    # where only that side is not a number, the kernel's flux is one)
    for have, want in ((got, flux), (got_src, src)):
        assert np.array_equal(have[~np.isnan(want)], want[~np.isnan(want)])
    assert bad or np.isfinite(flux).mean() > 0.5
