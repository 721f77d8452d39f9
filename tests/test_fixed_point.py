"""The double path's integer arithmetic (block_fixed.cuh) in its host build,
element by element: the same integers as on the GPU, without one."""
from __future__ import annotations

import ctypes as C
import subprocess

import numpy as np
import pytest

from conftest import PKG_DIR, ROOT

DOUBLES = np.ctypeslib.ndpointer(np.float64, flags="C_CONTIGUOUS")
INTS = np.ctypeslib.ndpointer(np.int32, flags="C_CONTIGUOUS")


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    lib = tmp_path_factory.mktemp("host") / "fixed_point_host.so"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC", f"-I{PKG_DIR / 'csrc'}",
                    str(ROOT / "tests" / "fixed_point_host.cpp"), "-o", str(lib)], check=True)
    lib = C.CDLL(str(lib))
    lib.host_forces.argtypes = [C.c_int] + [DOUBLES] * 6 + [INTS]
    return lib


SIGNS = np.array([[-1, 1, 1, -1, -1, 1, 1, -1], [-1, -1, 1, 1, -1, -1, 1, 1], [-1, -1, -1, -1, 1, 1, 1, 1]])


def _forces(host, x, vel, coef, press):
    n = len(x)
    out, fits = np.empty((n, 3, 8)), np.empty((n, 3), np.int32)
    volume = np.full(n, (1.125 / 30) ** 3)
    host.host_forces(n, np.ascontiguousarray(x), np.ascontiguousarray(vel), 1.0 / (192.0 * volume),
                     np.broadcast_to(float(coef), n).copy(), np.broadcast_to(float(press), n).copy(), out, fits)
    return out, fits


@pytest.mark.parametrize("coef", [-1e-26, -0.3, 0.0])
@pytest.mark.parametrize("press", [0.0, 2.5])
def test_forces_of_still_corners(host, coef, press):
    """Corner velocities that are zeros of both signs are rest: the forces of
    all +0. Velocities that are all subnormal are not rest, and are left to
    the double form."""
    rng = np.random.default_rng(7)
    n, h = 64, 1.125 / 30
    x = h * (3.0 + 0.5 * SIGNS + rng.uniform(-0.1, 0.1, (n, 3, 8)))
    x[0] = h * (3.0 + 0.5 * SIGNS)
    rest, fits = _forces(host, x, np.zeros((n, 3, 8)), coef, press)
    assert fits.all()
    if press == 0.0:
        assert not rest.any()
    signed = np.where(rng.integers(0, 2, (n, 3, 8)) == 1, -0.0, 0.0)
    signed[0] = 0.0
    signed[0, :, 3] = -0.0
    got, fits = _forces(host, x, signed, coef, press)
    assert fits.all()
    np.testing.assert_array_equal(got, rest)
    for tiny in (5e-324, 1e-320, 1e-312, 2e-308):
        slow = np.zeros((n, 3, 8))
        slow[:, :, 5] = tiny
        assert not _forces(host, x, slow, coef, press)[1].any()
