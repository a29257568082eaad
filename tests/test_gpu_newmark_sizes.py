"""Newmark assemblies at the sizes where the element kernel changes: less than a
warp of beams, a warp and one more, the largest model of the four-warp kernel and
the smallest of the thread-per-beam kernel, with and without drag, in a step's first
and later iterations, against the oracle's assembly (1e-12 of the largest entry, the
bar of the assembly parity tests)."""
import numpy as np
import pytest

from muscade_gpu.device import DeviceModel
from muscade_gpu.elements import BeamCrossSection, EulerBeam3D, Hold
from muscade_gpu.model import Model
from oracle import reference as REF

pytestmark = pytest.mark.gpu
TOL = 1e-12


@pytest.mark.parametrize("drag", [False, True])
@pytest.mark.parametrize("nel", [1, 31, 33, 9000, 9001])
def test_newmark_assembly_matches_oracle_at_the_kernels_limits(nel, drag):
    m = Model("chain")
    nodes = m.addnode(np.stack([np.arange(nel + 1.0), np.zeros(nel + 1), np.zeros(nel + 1)], axis=1))
    d = dict(Ca1=0.1, Cl1=0.2, Cq1=0.3, Ca2=5.0, Cl2=0.4, Cq2=3.0, Ca3=6.0, Cl3=0.7, Cq3=4.0) if drag else {}
    mat = BeamCrossSection(EA=1e4, EI2=3e2, EI3=2e2, GJ=4e2, mu=10.0, iota1=1.0, w=3.0, **d)
    m.addelement(EulerBeam3D, np.stack([nodes[:-1], nodes[1:]], axis=1), mat=mat, orient2=(0.0, 1.0, 0.0))
    m.addelement(Hold, [nodes[0]], field="t1")
    st = m.initialize()
    rng = np.random.default_rng(nel)
    X = [rng.normal(size=m.ndof["X"]) * s for s in (0.05, 0.5, 0.5)]
    c = REF.newmark_coefficients(2, 0.05, 0.25, 0.5)
    prep = REF.Prepared(m, st.dis)
    dm = DeviceModel(m, st.dis)
    for mission, name in ((1, "step"), (2, "iter")):
        Ll, nz = dm.assemble(X, t=0.5, mission=mission, c=c)
        Lr, nr = REF.assemble(prep, tuple(X), (np.zeros(0),), 0.5, name, c)
        assert np.max(np.abs(Ll - Lr)) <= TOL * np.max(np.abs(Lr)), name
        assert np.max(np.abs(nz - nr)) <= TOL * np.max(np.abs(nr)), name
    dm.close()
