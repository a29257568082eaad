"""When the multifrontal solver's sweeps stop (csrc/sparse_stop.hpp), on sequences of
corrections relative to a solution of largest entry 1."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "muscade.jl_gb300", "csrc")
U = 2.0**-53


@pytest.fixture(scope="module")
def stop():
    build = os.path.join(HERE, "_build")
    os.makedirs(build, exist_ok=True)
    so = os.path.join(build, "libsparse_stop_check.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, "-o", so + ".tmp",
                    os.path.join(HERE, "sparse_stop_check.cpp")], check=True)
    os.replace(so + ".tmp", so)
    f = ctypes.CDLL(so).sparse_stop_check
    f.argtypes = [ctypes.c_int] * 2 + [ctypes.c_void_p] * 4 + [ctypes.c_int]

    def run(c, r=None, y=None, a=None, nrow=40, mixed=True):
        n = len(c)
        v = [np.ascontiguousarray(np.broadcast_to(np.asarray(q, dtype=np.float64), (n,)).copy())
             for q in (c, 1.0 if y is None else y, 0.0 if r is None else r, 1.0 if a is None else a)]
        return f(int(mixed), n, *[q.ctypes.data for q in v], nrow)

    return run


@pytest.mark.parametrize("c, at", [
    ([1.0, 1e-14], 2),                            # a correction that is small enough itself
    ([1e-15], 1),                                 # the solution was there before
    ([0.0, 0.0], 1),                              # no load
    ([1.0, 1e-4, 1e-8, 1e-12], 4),                # the next one is 1e-16
    ([1.0, 3e-8, 1e-9, 1e-10], 0),                # 3e-8 and, at its rate, 9e-16: the rate was not to last
    ([1.0, 1e-12, 1e-15], 3),                     # two sweeps tell a rate, not its run
    ([1.0, 1e-2, 1e-8, 1e-12, 1e-14], 5),         # at the worst rate, not the last one
    ([1.0, 1e-3, 1e-6, 2e-11, 4e-16], 5),         # 2e-11 is still too much to go by a rate
    ([1.0, 1e-6, 1e-11, 0.8e-11, 0.7e-11, 1e-12], 3),  # 1e-11 at a rate of 1e-5
])
def test_corrections_that_shrink(stop, c, at):
    assert stop(c, r=1.0) == at


def test_a_plateau_counts_where_the_residual_is_rounding_or_it_lasts(stop):
    c = [1.0, 1e-2, 5e-11, 4e-11, 3.5e-11, 1e-12]
    assert stop(c, r=44 * U) == 4
    assert stop(c, r=[1.0, 1e-4, 1e-9, 1e-10, 44 * U, 44 * U]) == 5  # two orders above it in the fourth
    assert stop(c, r=1e-12) == 5  # the second time in a row
    assert stop([1.0, 1e-2, 5e-11, 4e-11, 1e-13, 9e-14], r=1e-12) == 0  # it did not last
    assert stop(c, r=1e-12, mixed=False) == 4  # plain sweeps have none of their own
    assert stop([1.0, 1e-6, 2e-10, 1.9e-10, 1.8e-10], r=0.0) == 0  # too far off to stop at all


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_what_is_not_finite_never_converges(stop, bad):
    assert stop([bad], y=[bad]) == -1
    assert stop([1.0, bad], y=[1.0, bad]) == -2
    assert stop([1.0, 1e-5], y=[1.0, bad]) == -2
