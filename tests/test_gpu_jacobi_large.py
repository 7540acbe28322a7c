"""The Jacobi start on periodic grids past the shared-memory tiles: batches of
sweeps in a graph, with the stop test in the sweep up to 2^21 points and in a
kernel of its own beyond. Potentials, fields and iteration counts are bit-exact
against the oracle. Sources of a few stop thresholds, so that the solves end
within a batch of 32 sweeps, in a later one, and at once."""
import numpy as np
import pytest

from apc_524_project_gb300 import abi, configs
from backends import GpuBackend, OracleBackend
from helpers import FIELDS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(107, 103, 111), (129, 131, 127)])
def test_large_periodic_start_is_the_oracles(n):
    info = configs.input_info(configs.tiny("jac", n=n, init="poisson"))
    g, o = GpuBackend(info, 0.4), OracleBackend(info, 0.4)
    rng = np.random.default_rng(1)
    for i, scale in ((abi.RHO, 1e-11), (abi.JX, 3e-12), (abi.JY, 1e-12), (abi.JZ, 0.0)):
        f = np.zeros(g.shape)
        v = rng.normal(0, 1, n) * scale
        f[1:n[0] + 1, 1:n[1] + 1, 1:n[2] + 1] = v - v.mean()
        g.set_field(i, f)
        o.set_field(i, f)
    rg, itg = g.poisson_init()
    ro, ito = o.initialize_fields_only()
    assert itg == ito and rg == ro == abi.OK, (itg, ito, rg, ro)
    assert itg[0] > 32 and 0 < itg[2] < 32 and itg[3] == 0, itg
    for i in FIELDS + [abi.PHI1, abi.PHI2, abi.AX1, abi.AX2, abi.AY1, abi.AY2, abi.AZ1, abi.AZ2]:
        np.testing.assert_array_equal(g.get_field(i), o.get_field(i), err_msg=abi.FIELD_NAMES[i])
    g.close()
    o.close()
