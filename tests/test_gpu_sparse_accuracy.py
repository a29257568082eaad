"""The multifrontal solver (csrc/sparse_lu.cu) where it was wrong or refused: a solve counts
as converged only where the residual b − Lλx x of the solution itself does, and fronts of
every size have their substitutions."""
import numpy as np
import pytest

from muscade_gpu import workloads as W
from muscade_gpu.device import DeviceModel
from muscade_gpu.model import Model

pytestmark = pytest.mark.gpu


def tower(nx, ny, nz, decades, seed=0):
    """A space frame whose members' stiffnesses are spread over some decades, the nodes
    up to 1 % out of place, held at its base and pushed at the top."""
    rng = np.random.default_rng(seed)
    m = Model("tower")
    ix, iy, iz = [a.ravel() for a in np.meshgrid(range(nx + 1), range(ny + 1), range(nz + 1), indexing="ij")]
    at = {p: k for k, p in enumerate(zip(ix, iy, iz))}
    nodes = m.addnode(np.stack([4.0 * ix, 4.0 * iy, 3.0 * iz], axis=1) + 0.01 * rng.normal(size=(len(ix), 3)))
    for step, orient in (((1, 0, 0), (0.0, 1.0, 0.0)), ((0, 1, 0), (0.0, 0.0, 1.0)), ((0, 0, 1), (1.0, 0.0, 0.0))):
        pairs = [(k, at[q]) for p, k in at.items()
                 if (q := tuple(np.add(p, step))) in at and (step == (0, 0, 1) or p[2] > 0)]
        f = 10.0 ** (decades * (rng.random(len(pairs)) - 0.5))
        mat = W.BeamCrossSection(EA=4.2e9 * f, EI2=1e8 * f, EI3=1e8 * f, GJ=8e7 * f, mu=100.0, iota1=1.0)
        m.addelement(W.EulerBeam3D, nodes[np.asarray(pairs)], mat=mat, orient2=orient)
    for f in ("t1", "t2", "t3", "r1", "r2", "r3"):
        m.addelement(W.Hold, nodes[iz == 0][:, None], field=f)
    m.addelement(W.DofLoad, nodes[iz == nz][:, None], field="t1", value=lambda t: 1e5 * t)
    m.addelement(W.DofLoad, nodes[iz == nz][:, None], field="t2", value=lambda t: 2e4 * t)
    return m


def test_factors_that_cannot_converge_give_way_to_fp64():
    """Forty storeys with stiffnesses over six decades: the corrections of the residuals
    formed from the solution level off at 5e-10 of it or more, above the 1e-10 at which a
    solve may stop short, whatever a recursion for the residual says (it went to 1e-14
    in nine sweeps)."""
    m = tower(3, 3, 40, 6.0)
    st = m.initialize()
    dm = DeviceModel(m, st.dis, linsolve="sparse")
    rc, _, _ = dm.sweepx(0, np.array([1.0]), st.time, list(st.X), fixed_iter=1)
    info = dm.sparse_info()
    dm.close()
    assert rc == 0 and info["last_fallback"] == 1


def test_one_block_substitutions_of_a_front_near_48_kb(monkeypatch):
    """Fronts whose vector fits the 48 KB of shared memory that need no opt-in, but not
    beside the substitution kernels' own tables, against the blocked substitutions."""
    m, times = W.lattice(23, 23, 23)
    st = m.initialize()
    out = {}
    for threshold in ("128", "100000"):
        monkeypatch.setenv("MGPU_SPARSE_BLOCKED_PIVOTS", threshold)
        dm = DeviceModel(m, st.dis, linsolve="sparse")
        rc, X, _ = dm.sweepx(0, times[:1], st.time, list(st.X), fixed_iter=1)
        info = dm.sparse_info()
        dm.close()
        assert rc == 0 and info["last_fallback"] == 0
        assert 36 * 1024 < 8 * info["max_front"] <= 48 * 1024
        out[threshold] = X
    a, b = out.values()
    lam = np.array([str(f).startswith("λ") for f in st.dis.fieldX])
    for sel in (lam, ~lam):
        assert np.max(np.abs(a[0, 0][sel] - b[0, 0][sel])) <= 1e-9 * np.max(np.abs(b[0, 0][sel]))


@pytest.mark.parametrize("kind", ["sparse", "sparse64"])
@pytest.mark.parametrize("kept", ["1", "2", "3"])
def test_sweeps_with_fewer_directions_reach_the_same_solution(monkeypatch, kind, kept):
    """Where there is no room for the directions of all sweeps, the conjugation starts
    again after fewer; a solve is as accurate, after some sweeps more perhaps."""
    m, times = W.lattice(12, 12, 6)
    st = m.initialize()
    out = {}
    for n in ("12", kept):
        monkeypatch.setenv("MGPU_SPARSE_DIRECTIONS", n)
        dm = DeviceModel(m, st.dis, linsolve=kind)
        rc, out[n], _ = dm.sweepx(0, times[:2], st.time, list(st.X), maxdx=1e-8, maxLl=1e-3)
        info = dm.sparse_info()
        dm.close()
        assert rc == 0 and info["last_fallback"] == 0
    lam = np.array([str(f).startswith("λ") for f in st.dis.fieldX])
    a, b = out[kept][:, 0], out["12"][:, 0]
    for sel in (lam, ~lam):
        assert np.max(np.abs(a[:, sel] - b[:, sel])) <= 1e-9 * np.max(np.abs(b[:, sel]))


def stubs(nels, axis, hold=0, seed=0):
    """Clamped beams of a few elements side by side, each floating until the multipliers
    of its one support are eliminated."""
    rng = np.random.default_rng(seed)
    m = Model("stubs")
    held, tip = [], []
    for c, nel in enumerate(nels):
        xyz = np.zeros((nel + 1, 3))
        xyz[:, axis] = np.arange(nel + 1.0)
        nodes = m.addnode(xyz + [0.0, 0.0, 50.0 * c] + 0.02 * rng.normal(size=xyz.shape))
        EA, EI2, EI3, GJ = (v * np.exp(rng.normal(0.0, 0.5, nel)) for v in (1e7, 1e4, 1e4, 1e4))
        mat = W.BeamCrossSection(EA=EA, EI2=EI2, EI3=EI3, GJ=GJ, mu=10.0, iota1=1.0)
        m.addelement(W.EulerBeam3D, np.stack([nodes[:-1], nodes[1:]], axis=1), mat=mat,
                     orient2=[(0.0, 1.0, 0.0), (0.0, 0.0, 1.0), (1.0, 0.0, 0.0)][axis])
        held.append(nodes[hold])
        tip.append(nodes[-1])
    for f in ("t1", "t2", "t3", "r1", "r2", "r3"):
        m.addelement(W.Hold, np.asarray(held)[:, None], field=f)
    m.addelement(W.DofLoad, np.asarray(tip)[:, None], field="t1", value=lambda t: 10.0 * t)
    m.addelement(W.DofLoad, np.asarray(tip)[:1, None], field="t2", value=lambda t: 13.0 * t)
    return m


STUBS = [((3,) * 9, 0, 0, 1e-9), ((3,) * 9, 0, 1, 1e-9), ((2, 3, 4), 2, 0, 1e-9), ((2, 60), 0, 1, 1e-6)]


@pytest.mark.parametrize("nels, axis, hold, tol, kind", [(*s, k) for k in ("sparse", "sparse64") for s in STUBS]
                         + [((1, 2), 0, 0, 1e-9, "sparse"), ((1,), 1, 0, 1e-9, "sparse")])  # FP64 without row exchanges meets a zero pivot there
def test_short_clamped_beams(nels, axis, hold, tol, kind):
    """One solve against the banded FP64 solver, which pivots: the factors are as good as
    rounding in the direction in which a component floats, so the first corrections are
    large and raise the residual, and steps that may only lessen it came to nothing
    (states wholly wrong, or FP32 factors given up for singular FP64 ones).  A component
    of 60 beams has a condition of some 1e10."""
    m = stubs(nels, axis, hold)
    st = m.initialize()
    out = {}
    for k in (kind, "f64"):
        dm = DeviceModel(m, st.dis, linsolve=k)
        rc, X, _ = dm.sweepx(0, np.array([1.0]), st.time, list(st.X), fixed_iter=1)
        dm.close()
        assert rc == 0
        out[k] = X[0, 0]
    lam = np.array([str(f).startswith("λ") for f in st.dis.fieldX])
    for sel in (lam, ~lam):
        assert np.max(np.abs(out[kind][sel] - out["f64"][sel])) <= tol * np.max(np.abs(out["f64"][sel]))
