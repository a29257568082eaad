"""The block banded solver (csrc/band_block.cuh) on frames: panels with a
remainder, bands from below one panel to the widest one that it takes, one
component over a cluster of blocks and several components side by side, against
the oracle's SweepX{0} (SuperLU).  States to 1e-9 of the largest dof and
multiplier, the bar of the other solvers' trajectories."""
import numpy as np
import pytest

from muscade_gpu import workloads as W
from muscade_gpu.device import DeviceModel
from oracle import reference as REF

pytestmark = pytest.mark.gpu
TOL = 1e-9


@pytest.mark.parametrize("grid, band", [((2, 2, 2), 64), ((3, 3, 3), 128), ((6, 5, 4), 160), ((4, 4, 9), 256)])
def test_frames_of_every_band_match_oracle(grid, band):
    m, times = W.lattice(*grid)
    _check(m, times[:2], band)


@pytest.mark.parametrize("nel", [1, 2, 3, 30])
def test_chains_match_oracle(nel):
    """Fewer rows than a panel, and bands below its width."""
    m, times = W.cantilever(nel=nel, length=2.0)
    _check(m, times[:2], 16, maxdx=1e-9)


def test_several_frames_in_one_model_match_oracle():
    """Components of different size and band, one block each or several."""
    params = [dict(kind="portal", nel=n, EA=1e8, EI2=1e4, EI3=1e4, GJ=1e4, load=1e3) for n in (10, 11, 17, 33)]
    m, _, times = W.build_batched(params)
    _check(m, times[:2], 32, maxdx=1e-9)


def _check(m, times, band, **kw):
    st = m.initialize()
    kw = kw or dict(maxdx=1e-6, maxLl=1e-3)
    dm = DeviceModel(m, st.dis, linsolve="block")
    info = dm.linear_solver_info()
    assert info["kind"] == "block" and info["max_kl"] <= band
    rc, X, _ = dm.sweepx(0, times, st.time, list(st.X), **kw)
    assert rc == 0
    again = dm.sweepx(0, times, st.time, list(st.X), **kw)[1]
    dm.close()
    assert np.array_equal(X, again)
    ref = np.stack([Xr[0] for _, Xr in REF.sweepx(m, st.dis, st, times, OX=0, **kw)])
    lam = np.array([str(f).startswith("λ") for f in st.dis.fieldX])
    for sel in (~lam, lam):
        err = np.max(np.abs(X[:, 0][:, sel] - ref[:, sel])) / np.max(np.abs(ref[:, sel]))
        assert err <= TOL, (err, info)
