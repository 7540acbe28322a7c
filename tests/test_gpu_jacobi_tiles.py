"""The Jacobi start on periodic grids, whose whole iteration runs on tiles in
shared memory: potentials, fields and iteration counts are bit-exact against
the oracle, at grids of one point, of a tile a point, of ragged tiles; for
runs that stop at their stop test (odd sides: anywhere in a batch of sweeps)
and at the iteration cap (even sides)."""
import numpy as np
import pytest

from apc_524_project_gb300 import abi, configs
from backends import GpuBackend, OracleBackend
from helpers import FIELDS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(1, 1, 1), (1, 3, 1), (3, 5, 7), (5, 5, 5), (9, 7, 11), (4, 5, 6), (13, 17, 11),
                               (21, 15, 9)])
@pytest.mark.parametrize("dx", [(1.0, 1.0, 1.0), (0.7, 1.3, 0.5)])
def test_periodic_start_is_the_oracles(n, dx):
    cfg = configs.tiny("jac", n=n, dx=dx, init="poisson")
    info = configs.input_info(cfg)
    g, o = GpuBackend(info, 0.4), OracleBackend(info, 0.4)
    rng = np.random.default_rng(sum(n))
    for k, i in enumerate((abi.RHO, abi.JX, abi.JY, abi.JZ)):
        f = np.zeros(g.shape)
        v = rng.normal(0, 10.0 ** -(3 + 2 * k), n)  # spread of scales: spread of iteration counts
        f[1:n[0] + 1, 1:n[1] + 1, 1:n[2] + 1] = v - v.mean()
        g.set_field(i, f)
        o.set_field(i, f)
    rg, itg = g.poisson_init()
    ro, ito = o.initialize_fields_only()
    assert itg == ito and rg == ro, (itg, ito, rg, ro)
    for i in FIELDS + [abi.PHI1, abi.PHI2, abi.AX1, abi.AX2, abi.AY1, abi.AY2, abi.AZ1, abi.AZ2]:
        np.testing.assert_array_equal(g.get_field(i), o.get_field(i), err_msg=abi.FIELD_NAMES[i])
    print(n, itg)
    g.close()
    o.close()
