"""Memory at the edges of the calls: states in arrays of which some are page-locked, and
what a model keeps on the device between calls for results."""
import ctypes

import numpy as np
import pytest

from muscade_gpu import _lib as L
from muscade_gpu import workloads as W
from muscade_gpu.device import DeviceModel

pytestmark = pytest.mark.gpu


def _chain(nel, *holds):
    m = W.Model("chain")
    x = np.arange(nel + 1.0)
    nodes = m.addnode(np.stack([x, 0 * x, 0 * x], axis=1))
    mat = W.BeamCrossSection(EA=1e4, EI2=3e2, EI3=2e2, GJ=4e2, mu=10.0, iota1=1.0, w=3.0)
    m.addelement(W.EulerBeam3D, np.stack([nodes[:-1], nodes[1:]], axis=1), mat=mat, orient2=(0.0, 1.0, 0.0))
    for f in holds:
        m.addelement(W.Hold, nodes[:1, None], field=f)
    return m, m.initialize()


def test_a_state_of_which_a_part_is_page_locked():
    """Position, velocity and acceleration one after the other in one array, the first
    alone page-locked: no copy may span both kinds."""
    m, st = _chain(1364, "t1", "t2")
    n = m.ndof["X"]
    assert n == 8192  # 64 KB: whole pages
    dm = DeviceModel(m, st.dis)
    raw = np.zeros(3 * n + 8192)
    at = (-raw.ctypes.data % 65536) // 8
    big = raw[at : at + 3 * n]
    big[:] = np.random.default_rng(0).normal(size=3 * n) * 0.05
    X = [big[:n], big[n : 2 * n], big[2 * n :]]
    kw = dict(mission=L.ASM_ITER, c=dict(a1=20.0, a2=2.0, a3=0.1, b1=400.0, b2=40.0, b3=1.0))
    ref = dm.assemble([x.copy() for x in X], **kw)
    first = ctypes.c_void_p(big.ctypes.data)
    assert dm.lib.mgpu_host_register(first, 8 * n) == L.MGPU_OK
    try:
        got = dm.assemble(X, **kw)
    finally:
        dm.lib.mgpu_host_unregister(first)
        dm.close()
    assert np.array_equal(got[0], ref[0]) and np.array_equal(got[1], ref[1])


def test_results_hold_no_more_than_their_allowance():
    """The records of 600,000 beams are 330 MB, above the 256 MB that a model keeps for
    its next results: neither they nor the workspace stay."""
    torch = pytest.importorskip("torch")
    m, st = _chain(600_000, "t1")
    dm = DeviceModel(m, st.dis)
    x = np.random.default_rng(1).normal(size=m.ndof["X"]) * 1e-3
    few = _chain(3)
    small = DeviceModel(few[0], few[1].dis)  # the library's own first allocations
    small.beam_results(0, [np.zeros(few[0].ndof["X"])])
    free = torch.cuda.mem_get_info()[0]
    a = dm.beam_results(0, [x])
    held = free - torch.cuda.mem_get_info()[0]
    b = dm.beam_results(0, [x])
    dm.close()
    small.close()
    assert held <= 256 << 20
    for p, q in zip(a.values(), b.values()):
        assert np.array_equal(p, q)
