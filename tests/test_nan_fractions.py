"""A volume fraction that is not finite makes the split path's pressure a NaN,
also where the fluid has no pi_inf and no FP64 product carries it there: the
momentum and energy of the cell and of its neighbours lose their numbers, as in
plain FP64, and cells out of reach keep theirs."""
import numpy as np
import pytest

from microfc_gb300 import cases, preprocess

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nd", [1, 2, 3])
@pytest.mark.parametrize("order", [1, 3, 5])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("fluid", [0, 1])
def test_neighbours_of_a_bad_fraction(nd, order, value, fluid):
    from microfc_gb300 import Simulation
    if nd == 1:
        c = cases.sod_1d(m=59, steps=1, dt=1e-5)
    elif nd == 2:
        c = cases.shock_droplet_2d(nx=40, ny=32, steps=1, dt=1e-9)
        c = c.replace(gammas=(2.5, 2.5), pi_infs=(0.0, 0.0))
    else:
        c = cases.shock_bubble_3d(N=32, steps=1, dt=1e-5).replace(m=30, n=27, p=25)
    c = c.replace(weno_order=order)
    x, y, z, q = preprocess.generate(c)
    at = (0 if nd < 3 else 12, 0 if nd < 2 else 13, 20)
    q[(c.adv_idx + fluid,) + at] = value
    rows = slice(c.mom_idx, c.E_idx + 1)
    lost = {}
    for prec in ("fp64", "split"):
        with Simulation(c.replace(precision=prec), x, y, z, q_cons=q) as sim:
            rhs, _ = sim.s_compute_rhs()
        near = [at] + [tuple(a + (s if d == 2 - k else 0) for d, a in enumerate(at)) for k in range(nd) for s in (-1, 1)]
        lost[prec] = [not np.isfinite(rhs[(rows,) + n]).any() for n in near]
        reach = np.abs(np.indices(rhs.shape[1:]) - np.reshape(at, (3, 1, 1, 1))).max(0) > 3
        assert np.isfinite(rhs[:, reach]).all()
    assert all(lost["fp64"]) and all(lost["split"]), lost
