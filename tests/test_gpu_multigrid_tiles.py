"""The multigrid levels between the one-block tail and those large enough for
a kernel a stage, which are cycled in shared-memory tiles with halos: grids at
the edges of the tile sizes, with remainders, with dimensions shorter than a
halo, of either smoother and boundary, and coarsest levels too large for the
tail. Each solution against the discrete equations, and the number of cycles
against the same V-cycle in numpy: a wrong correction would still end at the
right solution, only later. The counts may differ by one where the last
cycle's residual falls next to the tolerance."""
import numpy as np
import pytest

from apc_524_project_gb300 import abi
from test_poisson_multigrid import FOUR_PI, SLOTS, SOURCES, _box, _gpu, _residual, _set_sources, _sources

PER, EXT = ("periodic",) * 6, ("external",) * 6
EXT_X = ("external", "external") + ("periodic",) * 4
CASES = {
    "tile4_red_black": ((40, 12, 10), PER),
    "tile4_thin": ((4, 40, 32), PER),
    "tile4_external": ((23, 19, 18), EXT),
    "tile4_jacobi": ((18, 15, 20), PER),
    "tile4_jacobi_short": ((3, 44, 36), PER),
    "tile8_red_black": ((36, 44, 34), PER),
    "tile8_remainders": ((33, 37, 30), EXT_X),
    "tile8_jacobi": ((33, 40, 28), PER),
    "tile8_below_stages": ((64, 48, 52), PER),
    "coarsest_in_tiles": ((19, 17, 15), PER),
    "coarsest_below_in_tiles": ((38, 34, 30), EXT),
}


class Level:
    def __init__(self, n, h, per):
        self.n, self.per = n, per
        self.lo = [1 if p else 2 for p in per]
        self.c = [1.0 / x ** 2 for x in h]
        self.diag = 2.0 * sum(self.c)
        self.rb = not any(p and m % 2 for p, m in zip(per, n))
        self.crs = [m % 2 == 0 and m >= 4 for m in n]
        self.sl = tuple(slice(lo, m + 1) for lo, m in zip(self.lo, n))
        idx = np.indices([m + 2 for m in n]).sum(0)[self.sl]
        self.colour = [idx % 2 == 0, idx % 2 == 1]

    def wrap(self, u):
        for d in range(3):
            if self.per[d]:
                v = np.moveaxis(u, d, 0)
                v[0], v[-1] = v[-2], v[1]

    def nb(self, u):
        self.wrap(u)
        s = 0.0
        for d in range(3):
            for o in (-1, 1):
                s = s + self.c[d] * u[tuple(slice(a.start + o * (e == d), a.stop + o * (e == d))
                                            for e, a in enumerate(self.sl))]
        return s

    def smooth(self, u, f, sweeps):
        for half in range(2 * sweeps):
            x = (self.nb(u) - f[self.sl]) / self.diag
            if self.rb:
                u[self.sl][self.colour[half % 2]] = x[self.colour[half % 2]]
            else:
                u[self.sl] += 6.0 / 7.0 * (x - u[self.sl])

    def residual(self, u, f):
        r = np.zeros_like(u)
        r[self.sl] = f[self.sl] - (self.nb(u) - self.diag * u[self.sl])
        return r


def _cycle(lv, l, f):
    L = lv[l]
    u = np.zeros_like(f)
    if l + 1 == len(lv):
        m = max(n + 1 - lo for n, lo in zip(L.n, L.lo))
        L.smooth(u, f, min(500, 2 * m * m + 8))
        return u
    L.smooth(u, f, 2)
    r = L.residual(u, f)
    L.wrap(r)
    for d in range(3):
        if L.crs[d]:
            v = np.moveaxis(r, d, 0)
            w = np.zeros((L.n[d] // 2 + 2,) + v.shape[1:])
            w[1:-1] = 0.25 * v[0:-2:2] + 0.5 * v[1:-1:2] + 0.25 * v[2::2]
            r = np.moveaxis(w, 0, d)
    C = lv[l + 1]
    g = np.zeros_like(r)
    g[C.sl] = r[C.sl]
    e = _cycle(lv, l + 1, g)
    C.wrap(e)
    for d in range(3):
        if L.crs[d]:
            v = np.moveaxis(e, d, 0)
            w = np.zeros((L.n[d] + 2,) + v.shape[1:])
            w[1:-1:2] = v[1:-1]
            w[2:-1:2] = 0.5 * (v[1:-1] + v[2:])
            e = np.moveaxis(w, 0, d)
    u[L.sl] += e[L.sl]
    L.smooth(u, f, 2)
    return u


def _cycles(n, h, per, f, rtol):
    lv = []
    while True:
        lv.append(Level(list(n), list(h), per))
        if not any(lv[-1].crs):
            break
        n = [m // 2 if c else m for m, c in zip(n, lv[-1].crs)]
        h = [2.0 * x if c else x for x, c in zip(h, lv[-1].crs)]
    u = np.zeros_like(f)
    L = lv[0]
    if all(per):
        f[L.sl] -= f[L.sl].mean()
    r = L.residual(u, f)
    first = np.abs(r).max()
    for it in range(1, 201):
        u += _cycle(lv, 0, r)
        r = L.residual(u, f)
        if np.abs(r).max() <= rtol * first:
            return it
    return 200


@pytest.mark.gpu
@pytest.mark.parametrize("case", sorted(CASES))
def test_gpu_multigrid_tiles(case):
    n, fb = CASES[case]
    cfg = _box(n, fb)
    g = _gpu(cfg, rtol=1e-10)
    rho, J = _sources(g.shape)
    _set_sources(g, rho, J)
    rc, it = g.poisson_init()
    assert rc == 0, (rc, it)
    for s, r in zip(SLOTS, SOURCES):
        res, scale = _residual(g.get_field(s), g.get_field(r), cfg)
        assert res <= 2e-10 * scale, (abi.FIELD_NAMES[s], res, scale)
    f = -FOUR_PI * g.get_field(abi.RHO)[:n[0] + 2, :n[1] + 2, :n[2] + 2]
    want = _cycles(n, cfg.dx, [b == "periodic" for b in fb[::2]], f, 1e-10)
    assert abs(it[0] - want) <= 1, (it, want)
    g.close()
