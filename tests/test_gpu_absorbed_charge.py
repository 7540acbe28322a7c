"""The current of particles that an absorbing wall removes, at time steps small
against the cell's light crossing time (d / dt of 5e3 and 1e5). The exit piece
of such a particle runs on to the next vertex plane whatever its speed, so its
current is qd D d / dt with D of the order of a cell: no velocity bounds it, and
in the mixed form's fixed point it passes 2^44 quanta. One step from zero
fields, charges of both signs, both walls: J of the mixed form, ghost and wall
planes included, against the oracle. The FP32 piece terms carry a handful of
roundings (start, end, charge, d / dt, the weights' products: 2^-24 each), an
offset half of 2^-24 cells against an extent of about one (for the transverse
components too, so the three are compared together): 1e-5 in relative L2 is ten
times that."""
import numpy as np
import pytest

from apc_524_project_gb300 import abi, configs
from backends import GpuBackend, OracleBackend, rel_l2

pytestmark = pytest.mark.gpu

N, DX = (4, 5, 3), (1.0, 0.5, 2.0)
RTOL = 1e-5


def _species(sign, count, dt, rng):
    """Half at each wall, within 0.2..0.7 of a step's way of it; every fifth moves inwards."""
    v = {k: rng.uniform(-0.4, 0.4, count) for k in ("vx", "vy", "vz")}
    left = np.arange(count) % 2 == 0
    speed = rng.uniform(0.5, 0.8, count)
    v["vx"] = np.where(left, -speed, speed) * np.where(np.arange(count) % 5 == 0, -1.0, 1.0)
    depth = speed * dt * rng.uniform(0.2, 0.7, count)
    p = {"x": np.where(left, depth, N[0] * DX[0] - depth)}
    # away from the transverse faces, which a step's way would cross in one form only
    for a, k in ((1, "y"), (2, "z")):
        p[k] = (rng.integers(0, N[a], count) + rng.uniform(0.1, 0.9, count)) * DX[a]
    v2 = sum(v[k] ** 2 for k in v)
    scale = np.where(v2 > 0.9, np.sqrt(0.9 / np.maximum(v2, 1e-300)), 1.0)
    p["gamma"] = 1.0 / np.sqrt(1.0 - v2 * scale ** 2)
    for k in v:
        p[k] = v[k] * scale
    return p


@pytest.mark.parametrize("relativity", [1, 0])
@pytest.mark.parametrize("dt", [2e-4, 1e-5])
def test_exit_current_matches_the_oracle(dt, relativity):
    cfg = configs.tiny("absorbed", n=N, dx=DX, init="constant", relativity=relativity, dt=dt,
                       part_bc=("absorbing",) * 2 + ("periodic",) * 4,
                       field_bc=("external",) * 2 + ("periodic",) * 4)
    info = configs.input_info(cfg)
    rng = np.random.default_rng(3)
    parts = [_species(s, 40, dt, rng) for s in (-1, 1)]
    o, m = OracleBackend(info, dt), GpuBackend(info, dt, precision=abi.MIXED, policy=abi.POLICY_CORRECTED)
    o.set_policy(1)
    for b in (o, m):
        for si, p in enumerate(parts):
            b.add_species(si, p, ids=np.arange(40 * si, 40 * si + 40))
        b.init_fields()
    co, _ = o.step(0)
    cm = m.step(1)
    assert list(cm) == list(co) and co[0] > 0 and co[1] > 0, (co, cm)
    # vertex planes 0..n+2 along the walled x; periodic ghosts hold what each form's fold left
    at = (slice(0, N[0] + 3), slice(1, N[1] + 1), slice(1, N[2] + 1))
    got, want = (np.stack([b.get_field(i)[at] for i in (abi.JX, abi.JY, abi.JZ)]) for b in (m, o))
    assert rel_l2(got, want) <= RTOL, rel_l2(got, want)
    assert m.check() == abi.OK
    o.close()
    m.close()
