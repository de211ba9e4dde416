"""Split 3-D grids on both sides of the line between blocks of 384 and of 128
threads (csrc/stage_3d_fp32.cu): the bits do not depend on the block, nor on
whether its tiles come by bulk copy, and the line is where the tiles of a sweep
outnumber the SMs."""
import numpy as np
import pytest

from microfc_gb300 import cases, preprocess

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz,threads", [(26, 26, 26, 384), (32, 32, 32, 384), (48, 25, 25, 384),
                                              (47, 27, 25, 128), (32, 32, 33, 128)])
@pytest.mark.parametrize("bcx,bcy", [((-3, -3), (-2, -4)), ((-1, -1), (-4, -2))])
def test_variants_agree_across_the_line(nx, ny, nz, threads, bcx, bcy):
    from microfc_gb300 import Simulation
    c = cases.shock_bubble_3d(N=32, steps=3).replace(m=nx - 1, n=ny - 1, p=nz - 1, bc_x=bcx, bc_y=bcy)
    x, y, z, q = preprocess.generate(c)
    outs = []
    for v in (0, 1):
        with Simulation(c, x, y, z, q_cons=q) as sim:
            shape = tuple(sim.select_variant(v))
            assert v == 1 or shape == (16, 16, threads)
            for _ in range(3):
                sim.tvd_rk(0, c.dt)
            outs.append(sim.download())
    assert np.isfinite(outs[0]).all()
    assert np.array_equal(outs[0].view(np.uint64), outs[1].view(np.uint64))
