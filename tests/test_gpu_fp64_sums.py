"""The rounding of the FP64 deposit's sums: J and rho of particles in cell order,
against the sums of the same terms in extended precision. The yardstick is a
warp's run of particles of one cell summed by a tree and added to the grid at
once, in double (worked out here): the deposit's error, over all grid values,
may be no larger. Root mean squares over some 4,000 values are within 2 %
(three standard deviations 5 %) of their expectation on either side, so a tenth
is allowed; sums in sequence, with an atomic for each half of a warp, take a
fifth more."""
import numpy as np
import pytest

from apc_524_project_gb300 import abi, configs
from backends import GpuBackend

pytestmark = pytest.mark.gpu

N = (16, 15, 14)
EDGE = ((0, 0), (1, 0), (1, 1), (0, 1))  # of the two transverse dimensions
VERTEX = ((0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 1, 1), (1, 1, 1), (1, 0, 1), (0, 0, 1))


def _terms(p, q):
    """(array, offset of the point, term a particle) as the deposit forms them, over the cell's own vertex."""
    r = np.stack([p[k] - np.floor(p[k]) for k in "xyz"])
    l, v = 1.0 - r, np.stack([p[k] for k in ("vx", "vy", "vz")])
    for i in range(3):
        j, k = (i + 1) % 3, (i + 2) % 3
        for a, b in EDGE:
            off = np.zeros(3, dtype=int)
            off[j], off[k] = a, b
            yield i, off, configs.UNIT_RHOJ * q * v[i] * (r[j] if a else l[j]) * (r[k] if b else l[k])
    for off in VERTEX:
        c = np.full(p["x"].shape, configs.UNIT_RHOJ * q)
        for d in range(3):
            c = c * (r[d] if off[d] else l[d])
        yield 3, np.array(off), c


def _run_totals(c, key):
    """Sums of each warp's runs of equal keys by a shuffle tree; zero except at the runs' first particles."""
    n = len(c)
    pad = -n % 32
    c, key = np.pad(c, (0, pad)).reshape(-1, 32), np.pad(key, (0, pad), constant_values=-1).reshape(-1, 32)
    head = np.ones(c.shape, dtype=bool)
    head[:, 1:] = key[:, 1:] != key[:, :-1]
    run = np.cumsum(head, axis=1)
    for off in (1, 2, 4, 8, 16):
        o = np.zeros_like(c)
        o[:, :-off] = np.where(run[:, :-off] == run[:, off:], c[:, off:], 0.0)
        c = c + o
    return c.reshape(-1)[:n], head.reshape(-1)[:n]


@pytest.mark.parametrize("ppc", [16, 61])
def test_rounding_is_a_trees(ppc):
    cfg = configs.tiny("sums", n=N, init="constant")
    info = configs.input_info(cfg)
    rng = np.random.default_rng(ppc)
    cells = np.repeat(np.stack(np.unravel_index(np.arange(np.prod(N)), N)), ppc, axis=1)
    count = cells.shape[1]
    p = {k: cells[a] + rng.uniform(0, 1, count) for a, k in enumerate("xyz")}
    p.update({k: rng.uniform(0, 0.5, count) for k in ("vx", "vy", "vz")}, gamma=np.zeros(count))
    g = GpuBackend(info, 0.4, policy=abi.POLICY_CORRECTED)
    g.add_species(0, p)
    g.deposit(True)
    got = [g.get_field(i) for i in (abi.JX, abi.JY, abi.JZ, abi.RHO)]
    g.close()
    exact = [np.zeros(g.shape, dtype=np.longdouble) for _ in range(4)]
    tree, size = [np.zeros(g.shape) for _ in range(4)], [np.zeros(g.shape) for _ in range(4)]
    key = np.ravel_multi_index(tuple(cells), N)
    for f, off, c in _terms(p, info.charge_ratio[0]):
        at = tuple(cells[d] + 1 + off[d] for d in range(3))
        np.add.at(exact[f], at, c.astype(np.longdouble))
        np.add.at(size[f], at, np.abs(c))
        total, head = _run_totals(c, key)
        np.add.at(tree[f], tuple(a[head] for a in at), total[head])

    def rms(values, f):
        on = size[f] > 0
        return float(np.sqrt(np.mean(((values - exact[f])[on] / size[f][on]).astype(float) ** 2)))

    for name, fs in (("J", (0, 1, 2)), ("rho", (3,))):
        have, want = (np.sqrt(np.mean([rms(x[f], f) ** 2 for f in fs])) for x in (got, tree))
        print(name, have / 2.0 ** -53, want / 2.0 ** -53)
        assert have <= 1.1 * want, (name, have / want)
