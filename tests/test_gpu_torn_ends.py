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
    assert rc == 0 and (kind == "auto" or np.array_equal(X, again))  # auto may leave FP32 factors for good
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


@pytest.mark.parametrize("nel, every, ncomp", [(120, 60, 1), (120, 7, 3), (120, 1, 1), (120, 2, 2), (120, 60, 490)])
def test_intermediate_supports_match_whole_components(nel, every, ncomp):
    """Multipliers along the chain: no separator may part one from its dof (the interior
    would have a zero row), so separators move, or a component stays whole."""
    m = W.Model("supports")
    mat = W.BeamCrossSection(EA=1e8, EI2=1e4, EI3=1e4, GJ=1e4, mu=10.0, iota1=1.0)
    x = np.linspace(0.0, 0.5 * nel, nel + 1)
    ends, held = [], []
    for c in range(ncomp):
        nodes = m.addnode(np.stack([x, np.full_like(x, 5.0 * c), np.zeros_like(x)], axis=1))
        m.addelement(W.EulerBeam3D, np.stack([nodes[:-1], nodes[1:]], axis=1), mat=mat, orient2=(0.0, 1.0, 0.0))
        ends += [nodes[0]]
        held += list(nodes[every:-1:every])
        m.addelement(W.DofLoad, nodes[every // 2 : every // 2 + 1, None], field="t3", value=lambda t: 50.0 * t)
        m.addelement(W.DofLoad, nodes[-1:, None], field="t1", value=lambda t: 100.0 * t)
    for f in ("t1", "t2", "t3", "r1", "r2", "r3"):
        m.addelement(W.Hold, np.asarray(ends)[:, None], field=f)
    for f in ("t2", "t3"):
        m.addelement(W.Hold, np.asarray(held)[:, None], field=f)
    st = m.initialize()
    times = np.array([0.5, 1.0])
    _same(st, _states(m, st, times, "auto", maxdx=1e-9), _states(m, st, times, "f64", maxdx=1e-9))


def test_driven_risers_keep_their_fp32_factors():
    """Elimination from the driven end too left the FP32 factors short of their
    refinement within these 20 steps, and the rest of the sweep to FP64 factors."""
    m, times = W.risers()
    st = m.initialize(time=0.0)
    dm = DeviceModel(m, st.dis)
    rc, _, _ = dm.sweepx(2, times[:20], st.time, [st.X[0]] * 3, fixed_iter=3)
    info = dm.linear_solver_info()
    dm.close()
    assert rc == 0 and info["kind"] == "torn32" and info["last_fallback"] == 0


def test_a_second_model_leaves_the_first_ones_solver_alone():
    """Models in one process: the shared memory of the fused solve is a setting of its
    kernels, and a later model of fewer interiors must not lower it for an earlier one."""
    m, times = W.risers(nriser=3, nel=200)
    st = m.initialize(time=0.0)
    few, ftimes = W.cantilever(nel=85, length=42.5)
    fst = few.initialize()
    kw = dict(fixed_iter=3)
    alone = _states(m, st, times[:2], "torn32", OX=2, **kw)
    first = DeviceModel(m, st.dis, linsolve="torn32")
    second = DeviceModel(few, fst.dis, linsolve="torn32")
    rc, X, _ = first.sweepx(2, times[:2], st.time, [st.X[0]] * 3, **kw)
    rc2, _, _ = second.sweepx(0, ftimes[:1], fst.time, [fst.X[0]], **kw)
    first.close()
    second.close()
    assert rc == 0 and rc2 == 0 and np.array_equal(X, alone)


@pytest.mark.parametrize("kind", ["torn", "torn32"])
@pytest.mark.parametrize("nel, ncomp", [(85, 1), (200, 3), (85, 490)])
def test_transposed_solves_match_whole_components(nel, ncomp, kind):
    """Gradients by the adjoint, whose solves are of Lλx's transpose: one first end
    without a spike, many interiors, and (490 components) a last end numbered
    backwards.  Chains swaying with drag: Lλx and its transpose differ by up to 1,150
    where the lateral stiffnesses are 8e5.  To 1e-6 of the largest component, the bar of
    the adjoint tests."""
    m = W.Model("swaying chains")
    x = np.linspace(0.0, 0.5 * nel, nel + 1)
    mat = W.BeamCrossSection(EA=1e8, EI2=1e4, EI3=1e4, GJ=1e4, mu=10.0, iota1=1.0, Ca2=5.0, Cq2=400.0, Ca3=6.0, Cq3=500.0)
    ends, sense = [], []
    for c in range(ncomp):
        nodes = m.addnode(np.stack([x, np.full_like(x, 5.0 * c), np.zeros_like(x)], axis=1))
        own = m.addnode(np.stack([0.5 * (x[1:] + x[:-1]), np.full(nel, 5.0 * c + 1.0), np.zeros(nel)], axis=1))
        m.addelement(W.EulerBeam3D, np.stack([nodes[:-1], nodes[1:], own], axis=1), mat=mat, orient2=(0.0, 1.0, 0.0), adof=True)
        ends.append(nodes[0])
        sense += [nodes[nel // 2], nodes[-1]]
        m.addelement(W.DofLoad, nodes[nel // 2 : nel // 2 + 1, None], field="t3", value=lambda t: 3e4 * t)
        m.addelement(W.DofLoad, nodes[-1:, None], field="t2", value=lambda t: 2e4 * t)
    for f in ("t1", "t2", "t3", "r1", "r2", "r3"):
        m.addelement(W.Hold, np.asarray(ends)[:, None], field=f)
    st = m.initialize(time=0.0)
    times = np.array([0.1, 0.2, 0.3])
    dofs = np.sort(W.node_dofs(m, np.asarray(sense))[:, 1:3].reshape(-1)) + 1
    out = {}
    for k in (kind, "f64"):
        dm = DeviceModel(m, st.dis, linsolve=k)
        dm.set_A(np.linspace(0.8, 1.25, dm.nA))
        C, g, _, _ = dm.adjoint(2, times, st.time, list(st.X), dofs, 1.0, np.zeros((len(times), len(dofs))), maxdx=1e-9)
        out[k] = (C, g)
        dm.close()
    (C, g), (Cr, gr) = out[kind], out["f64"]
    assert C == pytest.approx(Cr, rel=1e-9)
    assert np.max(np.abs(g - gr)) <= 1e-6 * np.max(np.abs(gr)) and np.max(np.abs(gr)) > 0.0
