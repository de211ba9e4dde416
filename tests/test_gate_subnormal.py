"""Gate samples of volume fractions below FP32's normal range: the split path
takes them as zero, so the features and the labels are those of zeros, exactly."""
import numpy as np
import pytest

from microfc_gb300 import cases, preprocess

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("direction", [0, 1])
def test_subnormal_volume_fractions_are_zeros(direction):
    import torch
    from microfc_gb300 import Simulation
    c = cases.shock_droplet_2d(nx=40, ny=32, steps=2, precision="split")
    x, y, z, q = preprocess.generate(c)
    rng = np.random.default_rng(3)
    zero = q[c.adv_idx] == 0.0
    assert zero.mean() > 0.1
    got = []
    for scale in (0.0, 1.0):
        tiny = scale * rng.choice([0.0, 1e-39, -3e-39, 1e-310, 8e-46], zero.shape)
        state = q.copy()
        state[c.adv_idx][zero] = tiny[zero]
        X = torch.empty(c.cells, 10, dtype=torch.float32, device="cuda")
        D = torch.empty(c.cells, dtype=torch.float32, device="cuda")
        with Simulation(c, x, y, z, q_cons=state) as sim:
            sim.gate_samples(direction, X.data_ptr(), D.data_ptr())
            torch.cuda.synchronize()
        got.append((X.cpu().numpy(), D.cpu().numpy()))
    assert np.array_equal(got[0][0], got[1][0])
    assert np.array_equal(got[0][1], got[1][1])
