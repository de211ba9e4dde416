"""The face whose two states go to two lanes (flex_lane_pairs in
csrc/mfc_flex.cuh) on small 1-D grids and the face of one lane on larger ones,
against the oracle, exactly.  WENO1 hands the cells' own states to the faces:
supersonic to either side, at rest with either zero, mirrored, with one-sided
mixtures and zero volume fractions, and states that are not a number.  (The
oracle adds zero times the downwind side, the kernel leaves it out: the check
is where the oracle has a number.)"""
import numpy as np
import pytest

from microfc_gb300 import cases, preprocess

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [60, 300, 5000, 60000])
@pytest.mark.parametrize("bc", [(-3, -3), (-4, -2), (-1, -1)])
@pytest.mark.parametrize("bad", [False, True], ids=["finite", "nan"])
def test_faces_between_cells_of_every_kind(oracle_lib, cells, bc, bad):
    from microfc_gb300 import Simulation
    c = cases.sod_1d(m=cells - 1, steps=1, dt=1e-9).replace(weno_order=1, bc_x=bc)
    x, y, z = preprocess.grid(c)
    rng = np.random.default_rng(cells)
    a = rng.choice([0.0, -0.0, 1e-8, 0.5, 1.0], cells)
    u = rng.choice([0.0, -0.0, 0.1, -0.1, 30.0, -30.0], cells)
    p = rng.choice([1e-3, 1.0, 1e5], cells)
    twin = rng.random(cells) < 0.3  # like the cell before but for the velocity's sign
    for w, s in ((a, 1.0), (u, -1.0), (p, 1.0)):
        w[1:][twin[1:]] = s * w[:-1][twin[1:]]
    rho = np.array([10.0 * np.abs(a) + 1e-3, 1.2 * (1.0 - np.abs(a)) + 1e-3])
    q = np.empty(c.shape)
    q[0, 0, 0], q[1, 0, 0] = rho
    q[2, 0, 0] = rho.sum(0) * u
    q[3, 0, 0] = c.gammas[0] * p + 0.5 * rho.sum(0) * u * u
    q[4, 0, 0], q[5, 0, 0] = a, 1.0 - np.abs(a)
    if bad:
        for v in range(6):
            q[v][0, 0, rng.random(cells) < 0.02] = np.nan
    o = oracle_lib.Oracle(c, x, y, z)
    o.set_state(q)
    with np.errstate(all="ignore"):
        want = o.compute_rhs()
    want = want[0] if isinstance(want, tuple) else want
    with Simulation(c, x, y, z, q_cons=q) as sim:
        got, _ = sim.s_compute_rhs()
    there = ~np.isnan(want)
    assert np.array_equal(got[there], want[there])
    assert there.mean() > 0.5
