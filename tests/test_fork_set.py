"""The server's side streams (csrc/fork_set.h): what cannot be created is done
without, so a group whose chains have no streams runs them one after another
instead of failing its requests."""
import ctypes
import os
import subprocess

import pytest

from conftest import NATIVE, PKG


@pytest.fixture(scope="module")
def lib():
    out = os.path.join(NATIVE, "_build")
    os.makedirs(out, exist_ok=True)
    so = os.path.join(out, "libfork_check.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I" + os.path.join(PKG, "csrc"), "-o", so,
                    os.path.join(NATIVE, "fork_check.cpp")], check=True)
    return ctypes.CDLL(so)


@pytest.mark.parametrize("streams,events,held,most", [
    (100, 100, (5, 6), 5),  # all of them
    (0, 100, (0, 6), 0),    # no stream can be created
    (2, 100, (2, 6), 2),    # streams run out
    (100, 0, (5, 0), 0),    # no event can be created
    (100, 3, (5, 3), 2),    # events run out
    (1, 100, (1, 6), 0),    # one chain does not use a side stream
])
def test_creation_that_runs_out(lib, streams, events, held, most):
    out = (ctypes.c_uint * 2)()
    served = lib.fork_create(5, streams, events, out)
    assert tuple(out) == held
    assert served == sum(1 << k for k in range(2, most + 1))

