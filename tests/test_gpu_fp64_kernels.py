"""The FP64 particle kernels at the sizes and values where their integer and
shared-memory paths could go wrong: warps and blocks cut short, runs of equal
cells of every length, unit and other cells, field strengths from zero to
overflow. One step from given fields against the oracle: positions,
velocities and gamma are bit-exact per particle (the kernels' operations are
the oracle's, or give the same word); the current differs by summation order
only, 1e-13 in relative L2."""
import numpy as np
import pytest

from apc_524_project_gb300 import abi, configs
from backends import GpuBackend, OracleBackend, by_id, rel_l2
from helpers import FIELDS

pytestmark = pytest.mark.gpu

KEYS = ("x", "y", "z", "vx", "vy", "vz", "gamma")


def _run(dx, n, scale, rel, policy, dt, vmax=0.6, walls=False):
    bc = dict(part_bc=("absorbing", "reflecting") + ("periodic",) * 4, field_bc=("external",) * 2 + ("periodic",) * 4)
    cfg = configs.tiny("kern", n=(5, 4, 6), dx=dx, relativity=int(rel), init="constant", **(bc if walls else {}))
    info = configs.input_info(cfg)
    g, o = GpuBackend(info, dt, policy=policy), OracleBackend(info, dt)
    if policy == abi.POLICY_CORRECTED:
        o.set_policy(policy)
    rng = np.random.default_rng(n)
    # runs of equal cells of random length, cells and offsets random
    cells = np.repeat(rng.integers(0, cfg.n, (n, 3)), rng.integers(1, 40, n), axis=0)[:n]
    p = {k: (cells[:, a] + rng.uniform(0, 1, n)) * dx[a] for a, k in enumerate("xyz")}
    if n > 3:  # on faces and walls
        for a, k in enumerate("xyz"):
            p[k][0], p[k][1] = 0.0, dx[a]
    for k in ("vx", "vy", "vz"):
        p[k] = rng.uniform(-vmax, vmax, n) * min(dx) / max(dt, 1.0)
    p["gamma"] = 1 / np.sqrt(1 - p["vx"] ** 2 - p["vy"] ** 2 - p["vz"] ** 2) if rel else np.zeros(n)
    half = n // 3
    for b in (g, o):
        nid = 0
        for si, sl in enumerate((slice(0, half), slice(half, n))):
            q = {k: v[sl] for k, v in p.items()}
            b.add_species(si, q, ids=np.arange(nid, nid + len(q["x"])))
            nid += len(q["x"])
        b.init_fields()
        for i in FIELDS:
            b.set_field(i, scale * np.random.default_rng(i).uniform(-1, 1, g.shape))
    o.interpolate()  # the oracle pushes with the fields cached before the step
    cg = g.step(1)
    co, _ = o.step(0)
    assert cg == co
    pg, po = by_id(g.particles()), by_id(o.particles())
    for k in KEYS:
        np.testing.assert_array_equal(pg[k], po[k], err_msg=k)
    for i in (abi.JX, abi.JY, abi.JZ):
        assert rel_l2(g.get_field(i), o.get_field(i)) <= 1e-13, i
    g.close()
    o.close()


@pytest.mark.parametrize("policy", [abi.POLICY_REFERENCE, abi.POLICY_CORRECTED])
@pytest.mark.parametrize("rel", [True, False])
@pytest.mark.parametrize("dx", [(1.0, 1.0, 1.0), (0.7, 1.3, 0.5), (2.0, 0.5, 1.0)])
@pytest.mark.parametrize("n", [1, 31, 33, 257, 1000])
def test_one_step_at_ragged_sizes(n, dx, rel, policy):
    _run(dx, n, 0.05, rel, policy, 0.45)


@pytest.mark.parametrize("dt", [0.5, 0.45])
@pytest.mark.parametrize("scale", [0.0, 1e-300, 1e-20, 3.0, 1e90])
def test_field_strengths(scale, dt):
    _run((1.0, 1.0, 1.0), 400, scale, True, abi.POLICY_REFERENCE, dt, vmax=0.3)


def test_walls_under_the_corrected_policy():
    _run((1.0, 1.0, 1.0), 700, 0.05, True, abi.POLICY_CORRECTED, 0.5, walls=True)
