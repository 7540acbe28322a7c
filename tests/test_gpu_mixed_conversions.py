"""The mixed form's conversions from and to FP64 arrays, whose truncations
and roundings are integer instructions: against numpy's conversions, for
positions on faces and a rounding short of them, and for velocities from zero
and denormals to the largest FP32 binades. The non-relativistic state and
positions on unit cells are bit-exact; gamma and the velocities formed from it
are within 1e-15 (the sum 1 + u^2 may be fused on the GPU: three roundings)."""

import numpy as np
import pytest

from apc_524_project_gb300 import abi, configs
from backends import GpuBackend, dptr

pytestmark = pytest.mark.gpu

N = (5, 3, 7)


def _positions(n, rng, dx):
    off = rng.uniform(0, 1, n)
    tiny = np.array([0.0, 5e-324, 1e-310, 1e-45, 2.0 ** -24, 0.5, 1 - 2.0 ** -24, 1 - 2.0 ** -25, 1 - 2.0 ** -26,
                     1 - 2.0 ** -40])
    off[:min(n, len(tiny))] = tiny[:n]
    out = []
    for a in range(3):
        # away from the last cell where the offset may round up into the next
        cell = rng.integers(0, N[a] - 1, n)
        out.append((cell + np.roll(off, 3 * a)) * dx[a])
    return out


def _expected_position(x, dx, a):
    t = x * (1.0 / dx)
    cell = np.floor(t)
    o = np.float32(t - cell)
    cell, o = np.where(o >= 1, cell + 1, cell), np.where(o >= 1, np.float32(0), o)
    return dx * (cell + np.float64(o))


def _velocities(n, rng):
    v = rng.uniform(-1, 1, n) * 10.0 ** rng.uniform(-12, 0, n)
    edge = np.array([0.0, -0.0, 5e-324, -1e-310, 1e-45, -1.1754942e-38, 1e-40, 2.0 ** -149 * 1.5, 1 + 2.0 ** -24,
                     1 + 3 * 2.0 ** -24, -(1 + 2.0 ** -24 + 2.0 ** -50), 1e30, -3.4e38, 2.0 ** 127 * (2 - 2.0 ** -24.5)])
    v[:min(n, len(edge))] = edge[:n]
    return v


@pytest.mark.parametrize("dx", [(1.0, 1.0, 1.0), (0.7, 1.3, 0.5)])
@pytest.mark.parametrize("n", [1, 33, 700])
def test_nonrelativistic_state_is_numpys(n, dx):
    cfg = configs.tiny("conv", n=N, dx=dx, init="constant")
    g = GpuBackend(configs.input_info(cfg), 0.4, precision=abi.MIXED)
    rng = np.random.default_rng(n)
    pos = _positions(n, rng, dx)
    vel = [np.roll(_velocities(n, rng), a) for a in range(3)]
    p = dict(zip(("x", "y", "z", "vx", "vy", "vz"), pos + vel), gamma=np.zeros(n))
    g.add_species(0, p)
    got = g.particles()
    for a, k in enumerate("xyz"):
        want = _expected_position(pos[a], dx[a], a)
        if dx == (1.0, 1.0, 1.0):
            np.testing.assert_array_equal(got[k], want, err_msg=k)
        else:
            np.testing.assert_allclose(got[k], want, rtol=1e-15, err_msg=k)
    with np.errstate(over="ignore", under="ignore"):
        for a, k in enumerate(("vx", "vy", "vz")):
            want = np.float64(np.float32(vel[a]))
            np.testing.assert_array_equal(got[k], want, err_msg=k)
            np.testing.assert_array_equal(np.signbit(got[k]), np.signbit(want), err_msg=k)
    assert g.check() == abi.OK
    g.close()


@pytest.mark.parametrize("n", [1, 33, 700])
def test_relativistic_state(n):
    cfg = configs.tiny("conv", n=N, relativity=1, init="constant")
    g = GpuBackend(configs.input_info(cfg), 0.4, precision=abi.MIXED)
    rng = np.random.default_rng(n)
    pos = _positions(n, rng, (1.0,) * 3)
    vel = [rng.uniform(-0.57, 0.57, n) * 10.0 ** rng.uniform(-6, 0, n) for _ in range(3)]
    vel[1][0] = 0.0
    ga = 1 / np.sqrt(1 - vel[0] ** 2 - vel[1] ** 2 - vel[2] ** 2)
    p = dict(zip(("x", "y", "z", "vx", "vy", "vz"), pos + vel), gamma=ga)
    g.add_species(0, p)
    loaded = g.particles()  # before the first push the loaded words come back
    for k in ("vx", "vy", "vz", "gamma"):
        np.testing.assert_array_equal(loaded[k], np.float64(np.float32(p[k])), err_msg=k)
    g.init_fields()
    g.step(1)
    arr = [np.ascontiguousarray(p[k]) for k in ("x", "y", "z", "vx", "vy", "vz", "gamma")]
    abi.check(g.L.emoo_set_particles(g.h, 0, n, *[dptr(a) for a in arr]), "emoo_set_particles")
    got = g.particles()
    u = [np.float64(np.float32(ga * v)) for v in vel]
    gg = np.sqrt(1 + u[0] ** 2 + u[1] ** 2 + u[2] ** 2)
    np.testing.assert_allclose(got["gamma"], gg, rtol=1e-15)
    for a, k in enumerate(("vx", "vy", "vz")):
        np.testing.assert_allclose(got[k], u[a] / gg, rtol=1e-15, err_msg=k)
    g.close()


def test_positions_outside_the_box_are_refused():
    cfg = configs.tiny("conv", n=N, init="constant")
    for bad in (-1e-9, -3.0, 5.0, 1e6, 3e9, 1e300, np.inf, np.nan):
        g = GpuBackend(configs.input_info(cfg), 0.4, precision=abi.MIXED)
        p = {k: np.array([bad if k == "x" else 1.5]) for k in ("x", "y", "z")}
        p.update({k: np.zeros(1) for k in ("vx", "vy", "vz", "gamma")})
        g.add_species(0, p)
        if bad == -1e-9:  # its offset 1 - 1e-9 rounds to the face at 0, as the conversion always took it
            assert g.L.emoo_check(g.h) == abi.OK and g.particles()["x"][0] == 0.0
        else:
            assert g.L.emoo_check(g.h) == abi.ERR_BOUNDS, bad
        g.close()
