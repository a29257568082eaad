"""The state that DeviceModel.assemble hands to the library, without a device: the
derivatives one after the other in the arrays' own order, whatever their shapes."""
import ctypes

import numpy as np
import pytest

from muscade_gpu import _lib as L
from muscade_gpu.device import DeviceModel

NX = 7


class _Library:
    def mgpu_assemble_parts(self, ctx, mission, nXder, x, *rest):
        self.at = [ctypes.cast(x[k], ctypes.c_void_p).value for k in range(nXder)]
        self.first = np.ctypeslib.as_array(x[0], (NX,)).copy()
        return L.MGPU_OK

    def mgpu_host_register(self, ptr, nbytes):
        return L.MGPU_OK


def _assemble(X, **kw):
    dm = DeviceModel.__new__(DeviceModel)
    dm.lib, dm.ctx, dm._registered = _Library(), None, []
    dm.nX, dm.nU, dm.nnz = NX, 0, 3
    dm.tvals = lambda t: np.zeros(0)
    dm._check = lambda rc: None
    try:
        dm.assemble(X, mission=L.ASM_ITER, **kw)
    finally:
        dm.ctx = None
    return dm.lib


@pytest.mark.parametrize("shapes", [[(NX,), (NX,)], [(2 * NX,), (0,)], [(2, NX), (2, NX)], [(NX, 1), (NX, 1)],
                                    [(1, NX), (1, NX)], [(NX + 1,), (NX - 1,)]])
def test_derivatives_lie_one_after_the_other(shapes):
    rng = np.random.default_rng(0)
    X = [rng.normal(size=s) for s in shapes]
    lib = _assemble(X)
    assert np.array_equal(lib.first, np.concatenate(X).reshape(-1)[:NX])
    if shapes != [(NX,), (NX,)]:  # those are taken where they are
        assert lib.at[1] - lib.at[0] == 8 * NX


@pytest.mark.parametrize("shapes, reuse", [([(NX, 1), (NX, 1)], True), ([(1, NX), (1, NX)], True),
                                           ([(2 * NX,), (1,)], True), ([(NX,), (NX, 1)], False),
                                           ([(NX,), (NX - 1,)], False), ([], False)])
def test_what_is_no_state_is_refused(shapes, reuse):
    with pytest.raises(ValueError):
        _assemble([np.zeros(s) for s in shapes], reuse=reuse)
