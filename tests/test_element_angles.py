"""The device element code (csrc/beam_spin.hpp, compiled for the host) at the
rotation angles where its functions change branch: zero and almost zero
rotations, both sides of the switches of the angle series (θ² = 1 and 10, the
latter past a half turn), and both sides of the switch of scac (1 − x = 1e-3 for
the relative rotation of the nodes), against the oracle's nested duals.  The
bound is that of the element parity tests, relative to the largest entry."""
import numpy as np
import pytest

from muscade_gpu.elements import beam_fields
from oracle import lib as O

from test_element_host import TOL, _relerr, host_eval  # noqa: F401  (fixture)

SCAC = float(np.arccos(1 - 1e-3))
ANGLES = [0.0, 1e-15, 1e-8, 1e-3, 1 - 1e-6, 1 + 1e-6, 3.0, 10**0.5 - 1e-6, 10**0.5 + 1e-6, 5.0]


@pytest.mark.parametrize("relative", [0.0, 1e-6, SCAC * (1 - 1e-3), SCAC * (1 + 1e-3), 1.2])
@pytest.mark.parametrize("angle", ANGLES)
def test_beam_at_the_branches_of_its_angle_functions(angle, relative, host_eval):  # noqa: F811
    rng = np.random.default_rng(17)
    n = 6
    c1 = rng.normal(size=(n, 3))
    c2 = c1 + rng.normal(size=(n, 3))
    mat = np.zeros((n, 16))
    mat[:, :4] = rng.uniform(1.0, 4.0, (n, 4))
    mat[:, 6] = rng.uniform(0.5, 1.0, n)  # weight: the external loads' part of R and K
    fields = beam_fields(c1, c2, rng.normal(size=(n, 3)), mat)
    unit = rng.normal(size=(n, 3))
    unit /= np.linalg.norm(unit, axis=1)[:, None]
    X = np.zeros((n, 3, 12))
    X[:, 0] = rng.normal(size=(n, 12)) * 0.1
    X[:, 0, 3:6] = angle * unit
    X[:, 0, 9:12] = (angle + relative) * unit  # same axis: the relative rotation is `relative`
    d = O.diffed("beam", fields, X, t=0.0)
    R, K = host_eval("beam", fields, X[:, 0], X[:, 1], X[:, 2], 1)
    assert _relerr(R, d["R"]) <= TOL
    assert _relerr(K, d["K"]) <= TOL
