"""Static beams in four parts on four warps (small models) and whole in one thread
(large ones) take the same operations: a chain assembled alone and among others, on
either side of the switch, gives the same residual and matrix bit for bit."""
import numpy as np
import pytest

from muscade_gpu import workloads as W
from muscade_gpu.device import DeviceModel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [1e-3, 0.3, 3.0])  # rotations: series of 8 terms, of 15, sines
@pytest.mark.parametrize("nel", [10, 33])
def test_split_and_whole_static_beams_agree_bitwise(nel, size):
    x = np.random.default_rng(nel).normal(size=(nel + 1, 6)) * size
    out = []
    for others in (0, 14):  # 33 beams at most; 5,600 beside them
        params = [dict(kind="cantilever", nel=n, EA=1e8, EI2=1e4, EI3=1.3e4, GJ=2e4, load=1e2) for n in [nel] + [400] * others]
        m, _, _ = W.build_batched(params)
        st = m.initialize()
        dm = DeviceModel(m, st.dis)
        d = W.node_dofs(m, np.arange(1, nel + 2))
        d = d[:, (d >= 0).all(axis=0)].ravel()  # the six dofs of every node
        X = np.zeros(dm.nX)
        X[d] = x.ravel()
        Ll, nz = dm.assemble([X])
        colptr, rowval = dm.pattern()
        dm.close()
        K = np.zeros((len(d), dm.nX))
        for q, j in enumerate(d):
            s = slice(colptr[j] - 1, colptr[j + 1] - 1)
            K[q, rowval[s] - 1] = nz[s]
        out.append((Ll[d], K[:, d]))
    assert np.count_nonzero(out[0][1]) > 0
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
