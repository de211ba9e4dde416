"""The tile size that split, gated and viscous 2-D runs take on both sides of
the line (kSmallTiles, csrc/mfc_launch.h), and that the bits do not depend on it."""
import numpy as np
import pytest

from microfc_gb300 import cases, gate, preprocess

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["split", "gated", "viscous"])
@pytest.mark.parametrize("nx,ny,tile", [(333, 167, 8), (320, 192, 8), (321, 192, 16), (360, 180, 16)])
def test_tile_across_the_line(kind, nx, ny, tile):
    from microfc_gb300 import Simulation
    c = cases.shock_droplet_2d(nx=64, ny=32, steps=2, dt=1e-8).replace(m=nx - 1, n=ny - 1, precision="split")
    if kind == "gated":
        c = c.replace(precision="gated")
    if kind == "viscous":
        c = c.replace(re_shear=(10.0, 500.0))
    x, y, z, q = preprocess.generate(c)
    outs = []
    for v in (0, 1, 2):  # the default, 16x16, 8x8
        with Simulation(c, x, y, z, q_cons=q) as sim:
            if kind == "gated":
                sim.set_gate(gate.load())
            shape = sim.select_variant(v)
            assert shape[0] == (tile, 16, 8)[v]
            for _ in range(2):
                sim.tvd_rk(0, c.dt)
            outs.append(sim.download())
    for o in outs[1:]:
        assert np.array_equal(o.view(np.uint64), outs[0].view(np.uint64))
