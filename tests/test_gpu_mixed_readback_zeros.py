"""Velocities read back from the mixed form's u keep the sign of a zero: v = u /
gamma is -0 where u is -0, whatever the other components make of gamma."""
import numpy as np
import pytest

from apc_524_project_gb300 import abi, configs
from backends import GpuBackend, dptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 1000])
def test_zeros_keep_their_sign(n):
    g = GpuBackend(configs.input_info(configs.tiny("zeros", relativity=1, init="constant")), 0.4, precision=abi.MIXED)
    rng = np.random.default_rng(n)
    first = dict(zip(("x", "y", "z"), [np.full(n, 1.5)] * 3), **{k: np.zeros(n) for k in ("vx", "vy", "vz")},
                 gamma=np.ones(n))
    g.add_species(0, first)
    g.init_fields()
    g.step(1)  # from here u is kept, set as gamma v with gamma 1
    u = [rng.uniform(-2, 2, n) * rng.integers(0, 2, n) for _ in range(3)]
    u[0] = np.where(rng.integers(0, 2, n) == 1, -0.0, 0.0)
    arr = [np.full(n, 1.5)] * 3 + u + [np.ones(n)]
    abi.check(g.L.emoo_set_particles(g.h, 0, n, *[dptr(np.ascontiguousarray(a)) for a in arr]), "emoo_set_particles")
    got = g.particles()
    for k, a in zip(("vx", "vy", "vz"), u):
        np.testing.assert_array_equal(got[k] == 0, a == 0)
        np.testing.assert_array_equal(np.signbit(got[k]), np.signbit(a), err_msg=k)
    g.close()
