"""The double path's integer arithmetic (block_fixed.cuh, eos_fixed.cuh) in its host build,
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
    lib.host_eos.argtypes = [C.c_int, DOUBLES, C.c_double, DOUBLES, INTS]
    lib.host_eos_above.argtypes = [C.c_int, DOUBLES, C.c_double, C.c_double, DOUBLES, INTS]
    lib.host_q_sums.argtypes = [C.c_int] + [DOUBLES] * 6 + [INTS]
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


def eos_reference(kind, e0, p0, q0, ql, qq, delv, v, p_cut):
    """One EOS evaluation (lulesh.cc:1692-1871, with 2/3 / v for the
    reference's 2/3 (comp + 1)) in the arithmetic of numpy type `kind`."""
    e0, p0, q0, ql, qq, delv, v = (np.asarray(a, kind) for a in (e0, p0, q0, ql, qq, delv, v))
    cls, half = kind(2) / kind(3), delv / 2

    def pressure(bvc, e):
        return np.where(bvc * e < p_cut, kind(0), bvc * e)

    def viscosity(e, vol, p):
        ss2 = cls * (e + vol * p)
        ss = np.where(ss2 <= .1111111e-36, kind(.3333333e-18), np.sqrt(np.maximum(ss2, kind(0))))
        return np.where(delv > 0, kind(0), ss * ql + qq), ss

    def cut(e):
        return np.where(np.abs(e) < 1e-7, kind(0), e)

    vhalf, pq = v - half, p0 + q0
    e = e0 - half * pq
    p = pressure(cls / vhalf, e)
    pqh = p + viscosity(e, vhalf, p)[0]
    e = cut(e + half * (3 * pq - 4 * pqh))
    p = pressure(cls / v, e)
    e = cut(e - (7 * pq - 8 * pqh + p + viscosity(e, v, p)[0]) * (delv / 6))
    p = pressure(cls / v, e)
    q, ss = viscosity(e, v, p)
    return e, p, np.where((delv <= 0) & (np.abs(q) < 1e-7), kind(0), q), ss


def _eos_errors(host, state, p_cut=1e-7, all_fit=True):
    """Worst relative error over the elements of e, p, q and ss: of the
    integers (those that fit), and of plain double arithmetic."""
    state = np.array(np.broadcast_arrays(*state), np.float64)
    n = state.shape[1]
    out, fits = np.empty((4, n)), np.empty(n, np.int32)
    host.host_eos(n, state, p_cut, out, fits)
    assert fits.all() or not all_fit
    exact, plain = eos_reference(np.longdouble, *state, p_cut), eos_reference(np.float64, *state, p_cut)
    errors = []
    for got, want, dbl in zip(*(np.array(x)[:, fits != 0] for x in (out, exact, plain))):
        np.testing.assert_array_equal(got == 0.0, want == 0)
        live = want != 0
        errors.append([float(np.max(np.abs((x - want)[live] / want[live]), initial=0.0)) for x in (got, dbl)])
    return errors


def _assert_no_worse_than_double(errors):
    # 4 units of half a last place: a few truncations of integers of 2^57
    for name, (got, plain) in zip(("e", "p", "q", "ss"), errors):
        assert got <= max(plain, 4 * 2.0 ** -53), (name, got, plain)


@pytest.mark.parametrize("delv", [-1e-5, -0.01, -0.1, -0.2])
@pytest.mark.parametrize("du2", [1e-3, 1.0, 1e4, 1e6, 1e10])
@pytest.mark.parametrize("e0", [1e-6, 1e-3, 1.0, 1e4])
def test_eos_at_a_shock_front(host, e0, du2, delv):
    """Cold elements that a shock of velocity jump du compresses: the work of
    the viscosity is many orders above the old energy, which still counts
    through the sound speed."""
    rng = np.random.default_rng(23)
    n = 2000
    v, e = rng.uniform(0.75, 1.0, n), e0 * rng.uniform(0.5, 1.0, n)
    p = 2.0 / 3.0 * e / v
    du2 = du2 * rng.uniform(0.5, 1.0, n)
    state = e, np.where(p < 1e-7, 0.0, p), 0.0, np.sqrt(du2) / 2, 2.0 / 3.0 * du2, delv * v * rng.uniform(0.9, 1.0, n), v
    _assert_no_worse_than_double(_eos_errors(host, state))


@pytest.mark.parametrize("delv", [1e-5, 0.01, 0.1])
@pytest.mark.parametrize("ratio", [0.0, 1.0, 1e6, 1e12])
def test_eos_of_opening_elements(host, ratio, delv):
    """Opening elements take no viscosity: whatever qq and ql hold (here the
    pressure times `ratio` and its root) has no part in the result."""
    rng = np.random.default_rng(29)
    n = 2000
    v, e = rng.uniform(0.8, 1.5, n), 10.0 ** rng.uniform(-4, 4, n)
    p = 2.0 / 3.0 * e / v
    state = e, p, 0.0, np.sqrt(ratio * p), ratio * p, delv * v * rng.uniform(0.9, 1.0, n), v
    _assert_no_worse_than_double(_eos_errors(host, state))


@pytest.mark.parametrize("p_cut", [1e-7, 1e-3])
@pytest.mark.parametrize("delv", [-1e-5, -0.01, -0.1])
@pytest.mark.parametrize("e0", [1e-5, 1e-2])
def test_eos_cuts_pressures_by_their_own_size(host, e0, delv, p_cut):
    """Whether a pressure is below the cutoff decides the sound speed that
    goes into the viscosity, at a front so strong that the pressure itself is
    lost beside the viscosity."""
    rng = np.random.default_rng(31)
    n = 2000
    v, e = rng.uniform(0.75, 1.0, n), e0 * rng.uniform(0.01, 1.0, n)
    p = 2.0 / 3.0 * e / v
    du2 = 1e14 * rng.uniform(0.5, 1.0, n)
    state = e, np.where(p < p_cut, 0.0, p), 0.0, np.sqrt(du2) / 2, 2.0 / 3.0 * du2, delv * v * rng.uniform(0.9, 1.0, n), v
    _assert_no_worse_than_double(_eos_errors(host, state, p_cut))


@pytest.mark.parametrize("delv", [-1e-5, -0.01, -0.2])
@pytest.mark.parametrize("ql", [1.0, 1e3, 1e8, 1e12])
@pytest.mark.parametrize("qq", [1e-3, 1e3, 1e9])
@pytest.mark.parametrize("e0", [1e-3, 1e3])
def test_eos_of_linear_viscosity(host, e0, qq, ql, delv):
    """A linear viscosity far above the quadratic one (of coefficients other
    than the reference's) follows the root of an energy that the small
    pressures have made: those that the integers take keep it exact."""
    rng = np.random.default_rng(37)
    n = 2000
    v, e = rng.uniform(0.75, 1.0, n), e0 * rng.uniform(0.5, 1.0, n)
    q = np.where(np.arange(n) % 3 == 0, 0.0, qq * rng.uniform(0.0, 1.0, n))
    qq = np.where(np.arange(n) % 5 == 0, 0.0, qq * rng.uniform(0.5, 1.0, n))
    state = e, 0.0, q, ql * rng.uniform(0.5, 1.0, n), qq, delv * v * rng.uniform(0.9, 1.0, n), v
    _assert_no_worse_than_double(_eos_errors(host, state, all_fit=False))


@pytest.mark.parametrize("delv", [-1e-4, -0.01, -0.2])
@pytest.mark.parametrize("ql", [0.0, 1.0, 6.0, 1e8])
@pytest.mark.parametrize("qq", [2e-3, 1e3, 1e9])
@pytest.mark.parametrize("e0", [0.0, -1e-7, -1e-3, -1e3, 1e-60])
def test_eos_of_no_energy(host, e0, qq, ql, delv):
    """Energies at and below zero, and those whose root is below the least
    sound speed, have that sound speed: its part in the viscosity counts."""
    rng = np.random.default_rng(37)
    n = 2000
    v, e = rng.uniform(0.75, 1.0, n), e0 * rng.uniform(0.5, 1.0, n)
    q = np.where(np.arange(n) % 3 == 0, 0.0, qq * rng.uniform(0.0, 1.0, n))
    qq = np.where(np.arange(n) % 5 == 0, 0.0, qq * rng.uniform(0.5, 1.0, n))
    state = e, 0.0, q, ql * rng.uniform(0.5, 1.0, n), qq, delv * v * rng.uniform(0.9, 1.0, n), v
    _assert_no_worse_than_double(_eos_errors(host, state, all_fit=False))


@pytest.mark.parametrize("length", [0.01, 1e-100, 1e100])
@pytest.mark.parametrize("scale", [1e250, 1e140, 1e100, 1e4, 1e-7, 1e-100, 1e-152, 1e-160, 1e-300, 1e-310])
def test_viscosity_sums(host, scale, length):
    """The limited sums of the viscosity (lulesh.cc:1600-1656) over every size
    of gradient (subnormal ones count as zero) and length: those that the
    integers take are exact, those of which a square or a limited part would
    leave the range they do not take."""
    rng = np.random.default_rng(43)
    n = 4000
    dv, dm, dp = (scale * rng.uniform(-1.0, 1.0, (n, 3)) for _ in range(3))
    for a in (dv, dm, dp):
        a[rng.uniform(size=a.shape) < 0.1] = 0.0
    dx = length * rng.uniform(0.1, 1.0, (n, 3))
    lin, quad, fits = np.empty(n), np.empty(n), np.empty(n, np.int32)
    host.host_q_sums(n, dv, dm, dp, dx, lin, quad, fits)
    if 1e-130 < scale * length < 1e130:
        assert fits.all()

    dv[np.abs(dv) < 2.0 ** -1022] = 0.0

    def limited(kind):
        norm = 1 / (kind(1) * dv + kind(1e-36))
        m, p = dm * norm, dp * norm
        phi = np.clip(np.minimum(np.minimum((m + p) / 2, 2 * m), 2 * p), 0, 1)
        d = np.minimum(kind(1) * dv * dx, 0)
        return -(d * (1 - phi)).sum(axis=1), (d * d * (1 - phi * phi)).sum(axis=1)

    with np.errstate(over="ignore", invalid="ignore"):
        exact, plain = limited(np.longdouble), limited(np.float64)
    for got, want, dbl in zip(*((a[fits != 0] for a in x) for x in ((lin, quad), exact, plain))):
        np.testing.assert_array_equal(got == 0.0, want == 0)
        live = want != 0
        err = [np.max(np.abs((x - want)[live] / want[live]), initial=0.0) for x in (got, dbl)]
        assert err[0] <= max(err[1], 4 * 2.0 ** -53), err


@pytest.mark.parametrize("delv", [-0.1, -1e-12, 1e-3])
@pytest.mark.parametrize("v0", [1e-90, 1.0, 1e100])
@pytest.mark.parametrize("power", [-306, -200, 150, 230])
@pytest.mark.parametrize("field", ["e", "p", "q", "ql", "qq"])
@pytest.mark.parametrize("base", [1.0, 1e-6])
def test_eos_of_extreme_magnitudes(host, base, field, power, v0, delv):
    """One input of extreme size beside ordinary ones, with relative volumes
    and an energy floor far outside the reference's: what the integers take
    is exact, and what would leave the range of a double they do not take."""
    rng = np.random.default_rng(47)
    n = 300
    v = v0 * rng.uniform(0.75, 1.0, n)
    e, p, q, ql, qq = (base * rng.uniform(0.5, 1.0, n) for _ in range(5))
    big = 10.0 ** power * rng.uniform(0.5, 1.0, n)
    state = [e, p, q, ql, qq, delv * v * rng.uniform(0.9, 1.0, n), v]
    state["epq".index(field) if len(field) == 1 else 3 if field == "ql" else 4] = big
    state = np.array(state)
    out, fits = np.empty((4, n)), np.empty(n, np.int32)
    host.host_eos_above(n, state, 1e-7, -1e300, out, fits)
    taken = fits != 0
    with np.errstate(all="ignore"):
        exact, plain = (np.array(eos_reference(k, *state[:, taken], 1e-7)) for k in (np.longdouble, np.float64))
    for got, want, dbl in zip(out[:, taken], exact, plain):
        np.testing.assert_array_equal(got == 0.0, want == 0)
        assert np.all(np.abs(want) < 1.7e308)
        live = want != 0
        err = [np.max(np.abs((x - want)[live] / want[live]), initial=0.0) for x in (got, dbl)]
        assert err[0] <= max(err[1], 4 * 2.0 ** -53), err
