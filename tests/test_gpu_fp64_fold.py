"""The reference policy's folds of J inside the E half (FP64 form): J, with its
ghost planes, and E after two steps against the oracle's fold by fold (1e-9),
on sides of one to three cells, where planes 1 and n + 1 meet, and around a
warp, periodic and with external x sides."""
import numpy as np
import pytest

from apc_524_project_gb300 import abi, configs, loading
from backends import GpuBackend, OracleBackend, rel_l2
from test_corrected_walls import FP64_RTOL, _fields, _load

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("walled", [False, True])
@pytest.mark.parametrize("n", [(1, 2, 3), (2, 1, 4), (3, 3, 1), (4, 33, 2), (5, 7, 31), (33, 2, 5)])
def test_current_and_e(n, walled):
    if walled and n[0] == 1:
        pytest.skip("external x sides want two cells")
    x = ("reflecting", "external") if walled else ("periodic", "periodic")
    cfg = configs.tiny("fold", n=n, dx=(0.9, 1.1, 0.8), ppc=6, relativity=1, init="constant", vth=0.2, steps=2, dt=0.3,
                       part_bc=(x[0],) * 2 + ("periodic",) * 4, field_bc=(x[1],) * 2 + ("periodic",) * 4)
    info, parts = configs.input_info(cfg), loading.sample_all(cfg)
    o, g = OracleBackend(info, cfg.dt), GpuBackend(info, cfg.dt)
    for b in (o, g):
        _load(b, parts)
        b.init_fields()
    for ti in range(cfg.steps):
        o.step(ti)
        g.step(1)
    fo, fg = _fields(o), _fields(g)
    for i in fo:
        assert np.isfinite(fg[i]).all() and rel_l2(fg[i], fo[i]) <= FP64_RTOL, (abi.FIELD_NAMES[i], rel_l2(fg[i], fo[i]))
    o.close()
    g.close()
