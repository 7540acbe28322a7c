"""The relativistic FP64 push word by word against the oracle - zeros with their
signs - where the quotients by gamma have zero and tiny numerators: fields of
zeros of either sign, and magnetic fields from 2^-920 down to 1e-304, under
which a particle at rest along an axis moves by as little. (Offsets, speeds and
field values keep clear of zero, so that no product of a field by a weight or a
speed is denormal: the kernel takes some of these doubled and halves the sum.)
The step's operations are the reference's or give the same word, so no
tolerance."""
import numpy as np
import pytest

from apc_524_project_gb300 import abi, configs
from backends import GpuBackend, OracleBackend, by_id

pytestmark = pytest.mark.gpu

KEYS = ("x", "y", "z", "vx", "vy", "vz", "gamma")
FIELDS = (abi.EX, abi.EY, abi.EZ, abi.BX, abi.BY, abi.BZ, abi.BX_TM1, abi.BY_TM1, abi.BZ_TM1)


def case(scale, seed, count=600):
    """Config, particles (a third at rest along each axis, zeros of either sign), and field values."""
    cfg = configs.tiny("words", n=(5, 4, 6), relativity=1, init="constant")
    rng = np.random.default_rng(seed)
    p = {k: rng.integers(0, n, count) + rng.uniform(0.1, 0.9, count) for k, n in zip("xyz", cfg.n)}
    zero = np.where(rng.integers(0, 2, (3, count)) == 1, 0.0, -0.0)
    for a, k in enumerate(("vx", "vy", "vz")):
        v = rng.uniform(0.1, 0.5, count) * rng.choice([-1.0, 1.0], count)
        p[k] = np.where(np.arange(count) % 3 == a, zero[a], v)
    p["gamma"] = 1.0 / np.sqrt(1.0 - p["vx"] ** 2 - p["vy"] ** 2 - p["vz"] ** 2)
    shape = tuple(n + 3 for n in cfg.n)
    sign = rng.choice([-1.0, 1.0], 6)
    f = {}
    for i in FIELDS:
        c = i if i <= abi.BZ else i - abi.BX_TM1 + abi.BX
        f[i] = sign[c] * (scale if c >= abi.BX else 0.0) * rng.uniform(0.5, 1.0, shape)
    return cfg, p, f


def run(b, p, fields, step):
    half = len(p["x"]) // 2
    for si, sl in enumerate((slice(0, half), slice(half, None))):
        b.add_species(si, {k: v[sl] for k, v in p.items()}, ids=np.arange(len(p["x"]))[sl])
    b.init_fields()
    for i, f in fields.items():
        b.set_field(i, f)
    step(b)
    out = by_id(b.particles())
    b.close()
    return out


def oracle_step(o):
    o.interpolate()  # the oracle pushes with the fields cached before the step
    o.step(0)


@pytest.mark.parametrize("seed", range(4))
@pytest.mark.parametrize("scale", [0.0, 2.0 ** -920, 1e-290, 1e-304])
@pytest.mark.parametrize("dt", [0.5, 0.45])
@pytest.mark.parametrize("policy", [abi.POLICY_REFERENCE, abi.POLICY_CORRECTED])
def test_push_gives_the_oracles_words(policy, dt, scale, seed):
    cfg, p, fields = case(scale, seed)
    info = configs.input_info(cfg)
    o = OracleBackend(info, dt)
    if policy == abi.POLICY_CORRECTED:
        o.set_policy(policy)
    want = run(o, p, fields, oracle_step)
    got = run(GpuBackend(info, dt, policy=policy), p, fields, lambda g: g.step(1))
    for k in KEYS:
        np.testing.assert_array_equal(got[k].view(np.int64), want[k].view(np.int64), err_msg=k)
