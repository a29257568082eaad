"""The block banded solver (csrc/band_block.cuh) on frames of bands up to just under its
limit of 256: the last row slots of the trailing columns (from 241), the panel's last
rows and the second row of each thread in the backward substitution, against the
oracle's SweepX{0}, to the bar of the other frames."""
import pytest

from muscade_gpu import workloads as W
from muscade_gpu.device import DeviceModel
from test_gpu_block import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid, least, most", [((6, 6, 5), 177, 192), ((7, 6, 6), 209, 224), ((6, 7, 7), 241, 256)])
def test_wide_frames_match_oracle(grid, least, most):
    m, _ = W.lattice(*grid)
    dm = DeviceModel(m, m.initialize().dis, linsolve="block")
    info = dm.linear_solver_info()
    dm.close()
    assert least <= info["max_kl"] and least <= info["max_ku"]
    m, times = W.lattice(*grid)
    _check(m, times[:2], most)
