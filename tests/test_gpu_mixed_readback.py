"""gamma and velocities read back from the mixed form's FP32 u against extended
precision, for |u| from far below to far above 1. With e = 2^-53: 1 + u^2 by
three roundings is within 3 e, its root within half of that, 1.5 e; gamma adds
its own rounding and a little (2.6 e), and so does v. The smallest u (1 + u^2 rounds to 1) keeps its own value."""
import numpy as np
import pytest

from apc_524_project_gb300 import abi, configs
from backends import GpuBackend, dptr

pytestmark = pytest.mark.gpu

E = 2.0 ** -53


@pytest.mark.parametrize("n", [1, 31, 1000])
@pytest.mark.parametrize("scale", [1e-30, 1e-9, 1e-3, 1.0, 30.0, 1e6, 1e18, 1e37])
def test_velocity_and_gamma(scale, n):
    g = GpuBackend(configs.input_info(configs.tiny("readback", relativity=1, init="constant")), 0.4, precision=abi.MIXED)
    rng = np.random.default_rng(n)
    u = [np.float64(np.float32(scale * rng.uniform(-3, 3, n))) for _ in range(3)]
    first = dict(zip(("x", "y", "z"), [np.full(n, 1.5)] * 3), **{k: np.zeros(n) for k in ("vx", "vy", "vz")},
                 gamma=np.ones(n))
    g.add_species(0, first)
    g.init_fields()
    g.step(1)  # from here u is kept, set as gamma v with gamma 1
    arr = [np.full(n, 1.5)] * 3 + u + [np.ones(n)]
    abi.check(g.L.emoo_set_particles(g.h, 0, n, *[dptr(np.ascontiguousarray(a)) for a in arr]), "emoo_set_particles")
    got = g.particles()
    x = [np.longdouble(a) for a in u]
    ga = np.sqrt(1 + x[0] ** 2 + x[1] ** 2 + x[2] ** 2)
    assert np.abs(got["gamma"] / ga - 1).max() <= 2.6 * E
    for k, a in zip(("vx", "vy", "vz"), x):
        want = a / ga
        assert np.all(np.abs(got[k] - want) <= 2.6 * E * np.abs(want)), k
    g.close()


def test_u_beyond_fp32():
    g = GpuBackend(configs.input_info(configs.tiny("readback", relativity=1, init="constant")), 0.4, precision=abi.MIXED)
    one = np.ones(1)
    g.add_species(0, dict(x=1.5 * one, y=1.5 * one, z=1.5 * one, vx=0 * one, vy=0 * one, vz=0 * one, gamma=one))
    g.init_fields()
    g.step(1)
    arr = [1.5 * one] * 3 + [0.5 * one, -1e-290 * one, 1e-290 * one, 1e300 * one]
    abi.check(g.L.emoo_set_particles(g.h, 0, 1, *[dptr(np.ascontiguousarray(a)) for a in arr]), "emoo_set_particles")
    got = g.particles()
    assert np.isnan(got["vx"][0]) and got["gamma"][0] == np.inf
    assert got["vy"][0] == 0 and np.signbit(got["vy"][0]) and got["vz"][0] == 0 and not np.signbit(got["vz"][0])
    g.close()
