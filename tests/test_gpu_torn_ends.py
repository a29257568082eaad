"""Partitioned solves whose end interiors go without spikes (csrc/band_torn.cuh,
tb_end): two, three and many interiors to a component, components left whole beside
them, FP64 and FP32 factors, Lλx and (adjoint) its transpose, against the row-band
solver, which factorises every component whole.  A direction is exact to some 1e-12
in each, and a converged state forgets it: 1e-9 of the largest state, the bar of the
other solvers' trajectories."""
import numpy as np
import pytest

from muscade_gpu import workloads as W
from muscade_gpu.device import DeviceModel

pytestmark = pytest.mark.gpu


def _states(m, st, times, kind, OX=0, **kw):
    dm = DeviceModel(m, st.dis, linsolve=kind)
    rc, X, _ = dm.sweepx(OX, times, st.time, [st.X[0]] * (OX + 1), **kw)
    again = dm.sweepx(OX, times, st.time, [st.X[0]] * (OX + 1), **kw)[1]
    dm.close()
    assert rc == 0 and np.array_equal(X, again)
    return X


def _same(st, a, b):
    lam = np.array([str(f).startswith("λ") for f in st.dis.fieldX])
    for sel in (~lam, lam):
        x, y = a[:, 0][:, sel], b[:, 0][:, sel]
        assert np.max(np.abs(x - y)) <= 1e-9 * np.max(np.abs(y))


@pytest.mark.parametrize("kind", ["torn", "torn32"])
@pytest.mark.parametrize("nels", [(85,), (90, 20, 133), (200, 85)])
def test_frame_chains_match_whole_components(nels, kind):
    params = [dict(kind="portal" if n % 2 else "cantilever", nel=n, EA=1e8, EI2=1e4, EI3=1e4, GJ=1e4, load=1e2) for n in nels]
    m, _, times = W.build_batched(params)
    st = m.initialize()
    _same(st, _states(m, st, times[:2], kind, maxdx=1e-9), _states(m, st, times[:2], "f64", maxdx=1e-9))


def test_many_components_in_two_interiors_match_whole_components():
    params = [dict(kind="cantilever", nel=85 + k % 7, EA=1e8, EI2=1e4, EI3=1e4, GJ=1e4, load=1e2) for k in range(490)]
    m, _, times = W.build_batched(params)
    st = m.initialize()
    _same(st, _states(m, st, times[:1], "torn", maxdx=1e-9), _states(m, st, times[:1], "f64", maxdx=1e-9))


@pytest.mark.parametrize("kind", ["torn", "torn32"])
def test_risers_match_whole_components(kind):
    m, times = W.risers(nriser=3, nel=97)
    st = m.initialize(time=0.0)
    kw = dict(OX=2, fixed_iter=4)
    _same(st, _states(m, st, times[:3], kind, **kw), _states(m, st, times[:3], "f64", **kw))
