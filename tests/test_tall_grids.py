"""Grids with rows for 65535 tiles, the most that a launch takes along y."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from microfc_gb300 import cases

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "microfc_gb300", "csrc")

PLAN = r"""
#include "mfc_launch.h"
#include <cstdio>
template <int NF, int WO, int NT, bool VISC> void rows() {
  for (int nx : {25, 64, 100, 128, 400, 1200})
    for (int ny : {65535, 262141, 524280, 740000, 900001, 990606, 1010618, 1031033, 1048560}) {
      const auto p = mfc::flex::plan<2, NF, WO, NT, VISC>(nx, ny);
      if (p.x < 4 || p.y < 4 || (ny + p.y - 1) / p.y > 65535) std::printf("%d %d %d %d: %d %d\n", NF, WO, nx, ny, p.x, p.y);
    }
}
int main() {
  rows<2, 5, 640, false>(); rows<1, 5, 640, false>(); rows<2, 3, 512, false>(); rows<2, 1, 512, false>();
  rows<1, 3, 512, false>(); rows<1, 1, 512, false>(); rows<2, 5, 512, true>(); rows<1, 5, 512, true>();
  std::printf("done\n");
}
"""


def test_plans_of_tall_grids_can_be_launched(tmp_path):
    """The tiles sized for a 2-D grid (flex::plan) leave at most 65535 rows of
    them wherever tiles of 16 rows do."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    src, exe = tmp_path / "plan.cu", tmp_path / "plan"
    src.write_text(PLAN)
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "--expt-relaxed-constexpr",
                    "-I", CSRC, "-o", str(exe), str(src)], check=True, capture_output=True)
    r = subprocess.run([str(exe)], check=True, capture_output=True, text=True)
    assert r.stdout == "done\n", r.stdout


@pytest.mark.gpu
def test_gradients_of_the_tallest_grid():
    """Split weno_Re_flux on 25 x 1048560 cells: 65535 rows of 16 cells and one
    row of faces more."""
    from microfc_gb300 import Simulation
    ny = 65535 * 16
    c = cases.shock_droplet_2d(nx=64, ny=32, steps=1, dt=1e-15, precision="split")
    c = c.replace(m=24, n=ny - 1, patches=c.patches[:2], re_shear=(1e6, 1e6), weno_re_flux=True)  # the shock alone
    with Simulation(c, ic="device") as sim:
        sim.tvd_rk(0, c.dt)
        assert sim.status() == 0
        u = np.zeros((ny, 25))
        sim.download_var(2, u, 25)
    assert np.isfinite(u).all() and np.abs(u).max() > 0
