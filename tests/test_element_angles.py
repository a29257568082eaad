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


def _elements(angle, relative, drag=None):
    rng = np.random.default_rng(17)
    n = 6
    c1 = rng.normal(size=(n, 3))
    c2 = c1 + rng.normal(size=(n, 3))
    mat = np.zeros((n, 16))
    mat[:, :4] = rng.uniform(1.0, 4.0, (n, 4))
    mat[:, 6] = rng.uniform(0.5, 1.0, n)  # weight: the external loads' part of R and K
    if drag is not None:
        mat[:, 4] = 1.3
        mat[:, 7:] = rng.uniform(0.1, 0.8, (n, 9)) if drag else 0.0
    fields = beam_fields(c1, c2, rng.normal(size=(n, 3)), mat)
    unit = rng.normal(size=(n, 3))
    unit /= np.linalg.norm(unit, axis=1)[:, None]
    X = rng.normal(size=(n, 3, 12)) * 0.5
    X[:, 0] *= 0.2
    X[:, 0, 3:6] = angle * unit
    X[:, 0, 9:12] = (angle + relative) * unit  # same axis: the relative rotation is `relative`
    return fields, X


@pytest.mark.parametrize("relative", [0.0, 1e-6, SCAC * (1 - 1e-3), SCAC * (1 + 1e-3), 1.2])
@pytest.mark.parametrize("angle", ANGLES)
def test_beam_at_the_branches_of_its_angle_functions(angle, relative, host_eval):  # noqa: F811
    fields, X = _elements(angle, relative)
    d = O.diffed("beam", fields, X, t=0.0)
    R, K = host_eval("beam", fields, X[:, 0], X[:, 1], X[:, 2], 1)
    assert _relerr(R, d["R"]) <= TOL
    assert _relerr(K, d["K"]) <= TOL


@pytest.mark.parametrize("drag", [False, True])
@pytest.mark.parametrize("relative", [0.0, 1e-6, 1.2])
@pytest.mark.parametrize("angle", ANGLES)
def test_moving_beam_at_the_branches_of_its_angle_functions(angle, relative, drag, host_eval):  # noqa: F811
    """The same with rates and inertia, with the mass alone (the Gram sums) and with
    drag (point by point).  Below |v| = 1e-14 the reference takes sinc1 for a
    constant, which shows in ∂R/∂X when the node turns.  Relative rotations near
    scac's switch are left out: its closed-form third derivative loses half its
    digits there in the oracle."""
    fields, X = _elements(angle, relative, drag)
    d = O.diffed("beam", fields, X, t=0.0)
    for p, name in (((1.0, 0.0, 0.0), "K"), ((0.0, 1.0, 0.0), "C"), ((0.0, 0.0, 1.0), "M")):
        R, K = host_eval("beam", fields, X[:, 0], X[:, 1], X[:, 2], 3, p)
        assert _relerr(R, d["R"]) <= TOL
        assert _relerr(K, d[name]) <= TOL, name
