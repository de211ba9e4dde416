"""The primitive pairs of split and gated runs (mfc_pair.cuh) are not needed: a
state that fills the device runs without them, and they are given back to a
later buffer that needs the room.  The device is filled up to what the case
takes without its pairs; the results are those of a run with them, bit for bit."""
import numpy as np
import pytest

from microfc_gb300 import cases, gate, preprocess

pytestmark = pytest.mark.gpu

MB = 1 << 20
NX, NY = 1000, 1024
PAIRS = 2 * 4 * 8 * NY * ((NX + 2 + 15) // 16 * 16)


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _fill(leave):
    import torch
    torch.cuda.empty_cache()
    blocks = []
    for rest in (256 * MB, 0):  # the large block's own page tables take some room, too
        blocks.append(torch.empty((_free() - leave - rest) // (2 * MB) * (2 * MB), dtype=torch.uint8, device="cuda"))
    assert leave - 8 * MB <= _free() <= leave + 8 * MB
    return blocks


def _case(prec):
    c = cases.shock_droplet_2d(nx=64, ny=32, steps=4, precision=prec, dt=4e-9).replace(m=NX - 1, n=NY - 1)
    return (c, *preprocess.generate(c))


def _release():
    import torch
    torch.cuda.empty_cache()


@pytest.mark.parametrize("prec", ["split", "gated"])
def test_context_runs_without_pairs(prec):
    from microfc_gb300 import Simulation
    c, x, y, z, q = _case(prec)
    outs = []
    before = _free()
    block = None
    try:
        for _ in range(2):
            with Simulation(c, x, y, z, q_cons=q) as sim:
                if block is None:
                    used = before - _free()
                if prec == "gated":
                    sim.set_gate(gate.load())
                sim.tune(1)
                for _ in range(2):
                    sim.tvd_rk(0, c.dt)
                outs.append(sim.download())
            if block is None:
                block = _fill(used - PAIRS // 2)
    finally:
        del block
        _release()
    assert np.array_equal(outs[0].view(np.uint64), outs[1].view(np.uint64))


def test_pairs_give_way_to_the_gradient_buffers():
    from microfc_gb300 import Simulation
    c, x, y, z, q = _case("split")
    c = c.replace(re_shear=(10.0, 500.0))
    outs = []
    before = _free()
    block = None
    try:
        for _ in range(2):
            with Simulation(c, x, y, z, q_cons=q) as sim:
                held = before - _free()
                sim.tvd_rk(0, c.dt)
                sim.set_viscous_gradients(True)
                gradients = before - _free() - held
                sim.tvd_rk(0, c.dt)
                sim.snapshot(0)
                outs.append(sim.snapshot_wait(0).copy())
                snapshot = c.cells * 56
            if block is None:
                block = _fill(held + gradients + snapshot - PAIRS // 2)
    finally:
        del block
        _release()
    assert np.array_equal(outs[0].view(np.uint64), outs[1].view(np.uint64))


def test_gradient_buffers_hold_what_the_precision_stores():
    """Split: velocity and two face-gradient pairs of each direction, 40 bytes a cell."""
    from microfc_gb300 import Simulation
    c, x, y, z, q = _case("split")
    with Simulation(c.replace(re_shear=(10.0, 500.0)), x, y, z, q_cons=q) as sim:
        before = _free()
        sim.set_viscous_gradients(True)
        assert before - _free() <= 40 * (NX + 10) * (NY + 10) + 16 * MB


@pytest.mark.parametrize("stepper", [2, 3])
def test_ensemble_runs_without_pairs(stepper):
    from microfc_gb300.ensemble import Ensemble
    c = _case("split")[0].replace(time_stepper=stepper)
    outs = []
    before = _free()
    block = None
    try:
        for _ in range(2):
            with Ensemble([c, c], ic="device") as ens:
                used = before - _free() if block is None else used
                ens.tune(1)
                ens.run(0, 2)
                outs.append(ens.download(1))
            if block is None:
                block = _fill(used - PAIRS)
    finally:
        del block
        _release()
    assert np.array_equal(outs[0].view(np.uint64), outs[1].view(np.uint64))
