"""1-D plain FP64 on both sides of the lines where small tiles give every face
value an item and every face two lanes (flex_sides and flex_lane_pairs in
csrc/mfc_flex.cuh): the oracle's bits, with the Riemann-state boundaries whose
faces take one state twice."""
import numpy as np
import pytest

from microfc_gb300 import cases, preprocess

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [3, 5])
@pytest.mark.parametrize("cells,bc", [(1000, (-4, -4)), (2433, (-3, -4)), (4864, (-4, -2)), (9729, (-1, -1))])
def test_small_and_large_tiles_of_a_line(cells, bc, order):
    import oracle
    from microfc_gb300 import Simulation
    c = cases.sod_1d(m=cells - 1, steps=4, dt=1e-5).replace(weno_order=order, bc_x=bc)
    x, y, z, q = preprocess.generate(c)
    o = oracle.Oracle(c, x, y, z)
    o.set_state(q)
    o.run(0, 4, c.dt)
    with Simulation(c, x, y, z, q_cons=q) as sim:
        sim.run(0, 4)
        got = sim.download()
    assert np.array_equal(got.view(np.uint64), o.get_state().view(np.uint64))
