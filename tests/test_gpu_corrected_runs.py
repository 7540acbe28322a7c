"""The corrected policy's commit of run totals in the mixed form: J after one
step against the FP64 form (1e-5) for the patterns of cells that a warp can
hold - one run, runs that span its middle, every particle alone, a few ends -
at particle counts around a warp and a block, with a third species that deposits
nothing (its particles share warps with the others and commit nothing)."""
import numpy as np
import pytest

from apc_524_project_gb300 import abi, configs
from backends import GpuBackend, rel_l2
from test_corrected_walls import MIXED_RTOL

pytestmark = pytest.mark.gpu

N = (6, 5, 7)
PATTERNS = {
    "one_run": lambda i: 0 * i,
    "pairs_across_the_middle": lambda i: (i + 1) // 2,
    "alone": lambda i: i,
    "runs_of_15": lambda i: i // 15,
    "one_odd_one_out": lambda i: (i % 32 == 16) * 3,
}


@pytest.mark.parametrize("pattern", sorted(PATTERNS))
@pytest.mark.parametrize("n", [1, 15, 33, 130])
def test_current_of_run_patterns(n, pattern):
    cfg = configs.tiny("corr_runs", n=N, relativity=1, init="constant", test_species=True, dt=0.3)
    rng = np.random.default_rng(n)
    cell = PATTERNS[pattern](np.arange(n)) % (N[0] * N[1] * N[2])
    at = np.stack(np.unravel_index(cell, N)).astype(float)
    parts = []
    for _ in range(3):
        # FP32 offsets away from the faces, so that both forms see the same cells
        off = np.float64(np.float32(rng.uniform(0.2, 0.8, (3, n))))
        v = rng.uniform(-0.5, 0.5, (3, n))
        parts.append(dict(x=at[0] + off[0], y=at[1] + off[1], z=at[2] + off[2], vx=v[0], vy=v[1], vz=v[2],
                          gamma=1 / np.sqrt(1 - (v ** 2).sum(0))))
    J = []
    for precision in (abi.FP64, abi.MIXED):
        g = GpuBackend(configs.input_info(cfg), cfg.dt, precision=precision, policy=abi.POLICY_CORRECTED)
        for s, k in ((0, 0), (1, 1), (2, 2)):
            g.add_species(s, parts[k])
        g.init_fields()
        g.step(1)
        J.append([g.get_field(f)[1:N[0] + 1, 1:N[1] + 1, 1:N[2] + 1] for f in (abi.JX, abi.JY, abi.JZ)])
        g.close()
    for a, b in zip(*J):
        assert rel_l2(b, a) <= MIXED_RTOL, rel_l2(b, a)
