"""The corrected policy's boundary points, which the fold, the B half, the
ghost copies and their transpose give threads of their own: boxes of one to
three cells a side, where a point has several images along one dimension, and
sides at a warp's width; periodic and with walls along x. FP64 against the
oracle (1e-9, ghost planes included), the mixed form against the FP64 form
(1e-5, three steps; sides of two cells or more) with its E, B and B_tm1 ghosts the exact images of their
points, and the transpose of the copies by the dot-product test."""
import numpy as np
import pytest

from apc_524_project_gb300 import abi, configs, loading
from apc_524_project_gb300.differentiate import Problem
from backends import OracleBackend, rel_l2
from test_corrected_walls import FP64_RTOL, MIXED_RTOL, _fields, _gpu, _load

pytestmark = pytest.mark.gpu

SIZES = [(1, 2, 3), (2, 3, 1), (3, 1, 2), (4, 3, 33), (7, 2, 31), (33, 5, 4)]
STEPS = 3


def _cfg(n, walled):
    part, field = ("reflecting",) * 2 if walled else ("periodic",) * 2, ("external" if walled else "periodic",) * 2
    return configs.tiny("corr_edges", n=n, dx=(0.9, 1.1, 0.8), ppc=6, relativity=1, init="constant", vth=0.2,
                        steps=STEPS, dt=0.3, part_bc=part + ("periodic",) * 4, field_bc=field + ("periodic",) * 4)


CASES = [(n, w) for n in SIZES for w in (False, True) if n[0] > 1 or not w]


@pytest.mark.parametrize("n,walled", CASES)
def test_fields_at_small_and_ragged_sizes(n, walled):
    cfg = _cfg(n, walled)
    o = OracleBackend(configs.input_info(cfg), cfg.dt)
    o.set_policy(1)
    _load(o, loading.sample_all(cfg))
    f, m = _gpu(cfg), _gpu(cfg, abi.MIXED)
    for b in (o, f, m):
        b.init_fields()
    for ti in range(STEPS):
        o.step(ti)
    f.step(STEPS)
    m.step(STEPS)
    fo, ff, fm = _fields(o), _fields(f), _fields(m)
    for i in fo:
        assert rel_l2(ff[i], fo[i]) <= FP64_RTOL, (abi.FIELD_NAMES[i], rel_l2(ff[i], fo[i]))
    phys = (slice(1, n[0] + (2 if walled else 1)), slice(1, n[1] + 1), slice(1, n[2] + 1))
    fields = [abi.EX, abi.EY, abi.EZ, abi.BX, abi.BY, abi.BZ]
    # a periodic side of one cell: the two forms fold the deposit beyond its
    # second image differently (FP64 deposits into unwrapped cells)
    for i in (fields + [abi.JX, abi.JY, abi.JZ]) if min(n) > 1 else []:
        assert rel_l2(fm[i][phys], ff[i][phys]) <= MIXED_RTOL, (abi.FIELD_NAMES[i], rel_l2(fm[i][phys], ff[i][phys]))
    of = [np.arange(k + 3) if d == 0 and walled else (np.arange(k + 3) - 1) % k + 1 for d, k in enumerate(n)]
    for i in fields + [abi.BX_TM1, abi.BY_TM1, abi.BZ_TM1]:
        v = m.get_field(i)
        np.testing.assert_array_equal(v, v[np.ix_(*of)], abi.FIELD_NAMES[i])
    for b in (o, f, m):
        b.close()


@pytest.mark.parametrize("n,walled", [((4, 2, 3), False), ((5, 3, 2), True), ((3, 33, 2), False)])
def test_copies_are_transposed(n, walled):
    P = Problem(_cfg(n, walled), nsteps=STEPS, slab=(1, n[0]), checkpoint_every=2, policy=abi.POLICY_CORRECTED)
    g = P.gradient()
    ddv = 1e-3 * np.random.default_rng(1).uniform(-1, 1, (3, P.np))
    t = P.tangent(np.zeros(P.theta0.shape), ddv)
    adj = float(np.sum(g["grad_v"] * ddv))
    assert abs(adj - t["tangent"]) <= 1e-9 * abs(t["tangent"]), (adj, t["tangent"])
