"""3-D characteristic fields on both sides of the line between the sweeps' two
register budgets (csrc/stage_char_fp64.cu): the oracle's bits."""
import numpy as np
import pytest

from microfc_gb300 import cases, preprocess

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(26, 27, 25), (32, 32, 38), (33, 30, 40)])
def test_sweeps_match_the_oracle(oracle_lib, nx, ny, nz):
    from microfc_gb300 import Simulation
    c = cases.shock_bubble_3d(N=32, steps=2, precision="fp64").replace(m=nx - 1, n=ny - 1, p=nz - 1, bc_y=(-2, -4),
                                                                       bc_z=(-1, -1), char_decomp=True)
    x, y, z, q = preprocess.generate(c)
    o = oracle_lib.Oracle(c, x, y, z)
    o.set_state(q)
    o.run(0, 2, c.dt)
    with Simulation(c, x, y, z, q_cons=q) as sim:
        sim.run(0, 2)
        got = sim.download()
    assert np.array_equal(got.view(np.uint64), o.get_state().view(np.uint64))
