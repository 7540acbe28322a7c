"""The history row's sums over particles and cells (momentum, kinetic and field
energies) against the oracle's, at counts around a warp, a block and beyond one
pass of the grid. All terms are of one sign, so the sums are compared
relatively: FP64 to n 2^-53 (640,000 terms in another order, 1e-10); the mixed
form sums at most eight FP32 terms at a time, each within a few roundings of
2^-24 (velocities, products, square root and quotient, the eight additions: 16
in all, 1e-6)."""
import numpy as np
import pytest

from apc_524_project_gb300 import abi, configs
from backends import GpuBackend, OracleBackend

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [(abi.FP64, 1e-10), (abi.MIXED, 1e-6)])
@pytest.mark.parametrize("n,cells", [(1, (1, 1, 1)), (31, (2, 3, 5)), (33, (3, 11, 1)), (257, (5, 4, 9)),
                                     (320000, (70, 70, 80))])
def test_history_row(n, cells, precision, tol):
    cfg = configs.tiny("sums", n=cells, relativity=1, init="constant", E0=(0.1, 0.2, 0.3), B0=(0.3, 0.1, 0.2))
    rng = np.random.default_rng(n)
    info = configs.input_info(cfg)
    o, g = OracleBackend(info, cfg.dt), GpuBackend(info, cfg.dt, precision=precision)
    for s in range(2):
        v = rng.uniform(0.1, 0.5, (3, n))
        pos = rng.uniform(0.0, 0.9, (3, n)) * np.array(cells)[:, None]
        p = dict(x=pos[0], y=pos[1], z=pos[2], vx=v[0], vy=v[1], vz=v[2], gamma=1 / np.sqrt(1 - (v ** 2).sum(0)))
        for b in (o, g):
            b.add_species(s, p)
    o.init_fields()
    g.init_fields()
    want, got = np.array(o.history(0.0)), np.array(g.history())
    assert (want[1:] > 0).all()
    np.testing.assert_allclose(got[1:], want[1:], rtol=tol)
    o.close()
    g.close()
