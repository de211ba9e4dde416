"""A time step captured in a CUDA graph from the context's stream and replayed:
a replay advances whatever state register 0 holds then.  The primitive pairs
that a split stage leaves for the next one (mfc_pair.cuh, mfc_pair_sweep.cuh)
must not be carried across it: neither into the graph's first stage from the
steps before the capture, nor out of a replay into the steps after it.  Exact,
against the same steps launched directly from freshly uploaded states."""
import numpy as np
import pytest

from microfc_gb300 import cases, gate, preprocess

pytestmark = pytest.mark.gpu


def _capture(sim, dt):
    import torch
    g, s = torch.cuda.CUDAGraph(), torch.cuda.ExternalStream(sim.stream)
    with torch.cuda.stream(s):
        g.capture_begin(capture_error_mode="thread_local")
        sim.tvd_rk(0, dt)
        g.capture_end()
    return g, s


@pytest.mark.parametrize("kind", ["2d_fp64", "2d_split", "2d_gated", "3d_split"])
@pytest.mark.parametrize("stepper", [2, 3])
def test_replayed_steps_equal_launched_ones(kind, stepper):
    import torch
    from microfc_gb300 import Simulation
    nd, prec = kind.split("_")
    if nd == "2d":
        c = cases.shock_droplet_2d(nx=61, ny=47, steps=9, precision=prec, mach=1.2)
    else:
        c = cases.shock_bubble_3d(N=32, steps=9).replace(m=32, n=26, p=27, precision=prec)
    c = c.replace(time_stepper=stepper)
    x, y, z, q = preprocess.generate(c)
    with Simulation(c, x, y, z, q_cons=q) as sim:
        if prec == "gated":
            sim.set_gate(gate.load())
        want = [q]
        for _ in range(7):
            sim.upload(want[-1])
            sim.tvd_rk(0, c.dt)
            want.append(sim.download())
        sim.upload(q)
        sim.tvd_rk(0, c.dt)  # leaves the pairs of its state
        g, s = _capture(sim, c.dt)

        def replay():
            with torch.cuda.stream(s):
                g.replay()

        replay()
        replay()  # after the first one the pairs are the graph's own
        got = [sim.download()]
        sim.tvd_rk(0, c.dt)
        replay()
        sim.tvd_rk(0, c.dt)  # a launched step on a replayed state
        got.append(sim.download())
        sim.upload(want[1])
        replay()
        got.append(sim.download())
    for have, k in zip(got, (3, 6, 2)):
        assert np.array_equal(have.view(np.uint64), want[k].view(np.uint64)), k
