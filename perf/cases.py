"""The work that is measured: what a program built on this framework has it do.

Five kinds of pass, each through the public entry points (the C ABI through
`abi`, and `differentiate.Problem`):

  loop      a run of the time loop from a loaded particle set: particles handed
            over, fields started, `steps` steps, then the particles, E, B and
            the charge density read back
  host      steps on particles that stay in the caller's host arrays
  jacobi    the Poisson field start of a loaded particle set, default solver
  multigrid the field start on a given charge and current density
  gradient  objective and adjoint gradient of a laser run

The mixed form takes and fills particle arrays in device memory; the FP64 form
copies from and to pinned host memory, as do all field reads. Particles that a
pass sorts at its start come in the order that a loop hands to its sort: by the
cell they sat in `DRIFT` steps earlier.
"""
import ctypes as C
import math

import torch

from apc_524_project_gb300 import abi, configs, differentiate

DRIFT = 20  # steps between two sorts
OMEGA_PE = {"thermal": 0.5, "beams": 0.5, "laser": 0.3, "langmuir": 0.5}
MASS_RATIO = 1836.0


# ------------------------------------------------------------------ the cases

def _loop(name, plasma, precision, n, ppc, steps, sort, policy="reference", rel=True, walls=False, dt=0.5, dx=1.0):
    c = {"kind": "loop", "plasma": plasma, "precision": precision, "policy": policy, "rel": rel, "walls": walls,
         "nx": n[0], "ny": n[1], "nz": n[2], "ppc": ppc, "steps": steps, "sort": sort, "dt": dt, "dx": dx}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest box anyone runs (a first check of an input): latency and launches
        _loop("mixed_tiny", "thermal", "mixed", (8, 8, 8), 3, 20, False),
        # a production run at full size, one sort interval
        _loop("mixed_large", "thermal", "mixed", (192, 192, 192), 16, 20, True),
        # an ordinary box, one sort interval
        _loop("mixed_medium", "thermal", "mixed", (64, 64, 64), 16, 20, True),
        # counter-streaming beams under the charge-conserving policy, odd sizes
        _loop("mixed_beams_corrected", "beams", "mixed", (97, 61, 53), 16, 20, True, policy="corrected", dt=0.45),
        # a laser into a plasma slab between walls, charge-conserving policy
        _loop("mixed_laser_walls", "laser", "mixed", (128, 48, 48), 8, 20, True, policy="corrected", walls=True),
        # the parity form on the Langmuir box: unsorted, non-relativistic
        _loop("fp64_langmuir", "langmuir", "fp64", (32, 32, 32), 8, 20, False, rel=False),
        # the parity form on the thermal plasma, sorted
        _loop("fp64_thermal", "thermal", "fp64", (48, 48, 48), 16, 10, True),
        # the parity form of the beams, odd sizes
        _loop("fp64_beams_corrected", "beams", "fp64", (49, 37, 29), 16, 10, True, policy="corrected", dt=0.45),
        # particles in the caller's host memory, as a host program keeps them
        {"name": "host_resident", "kind": "host", "nx": 48, "ny": 40, "nz": 36, "ppc": 16, "steps": 2},
        # the Langmuir field start with the default solver
        {"name": "poisson_jacobi", "kind": "jacobi", "nx": 32, "ny": 32, "nz": 32, "ppc": 8},
        # the field start of a larger box with the fast solver
        {"name": "poisson_multigrid", "kind": "multigrid", "nx": 128, "ny": 64, "nz": 64},
        # forward and backward of the differentiated loop
        {"name": "gradient_fp64", "kind": "gradient", "precision": "fp64", "policy": "corrected", "nx": 32, "ny": 32,
         "nz": 32, "ppc": 8, "steps": 24, "every": 8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["loop"] * 6 + ["host", "jacobi", "multigrid", "gradient", "gradient"])
    if kind == "loop":
        precision = rng.choice(["mixed", "mixed", "fp64"])
        plasma = rng.choice(["thermal", "beams", "laser"])
        policy = rng.choice(["reference", "corrected"]) if plasma == "thermal" else "corrected"
        big = 144 if precision == "mixed" else 40
        n = [_log(rng, 8, big) for _ in range(3)]
        return _loop(None, plasma, precision, n, rng.choice([2, 3, 8, 16]),
                     2 * rng.randint(2, 6 if policy == "reference" else 10),
                     rng.random() < 0.8, policy=policy, rel=plasma != "thermal" or rng.random() < 0.7,
                     walls=plasma == "laser", dt=rng.choice([0.5, 0.45]),
                     dx=rng.choice([1.0, 1.0, 1.0, 1.25]))
    if kind == "host":
        return {"kind": kind, "nx": _log(rng, 8, 64), "ny": _log(rng, 8, 64), "nz": _log(rng, 8, 64),
                "ppc": rng.choice([3, 8, 16]), "steps": 2 * rng.randint(1, 2)}
    if kind == "jacobi":
        return {"kind": kind, "nx": _log(rng, 8, 40), "ny": _log(rng, 8, 40), "nz": _log(rng, 8, 40),
                "ppc": rng.choice([2, 8])}
    if kind == "multigrid":
        return {"kind": kind, "nx": _log(rng, 8, 192), "ny": _log(rng, 8, 128), "nz": _log(rng, 8, 128)}
    return {"kind": kind, "precision": rng.choice(["fp64", "mixed"]), "policy": rng.choice(["reference", "corrected"]),
            "nx": _log(rng, 12, 40), "ny": _log(rng, 8, 32), "nz": _log(rng, 8, 32), "ppc": rng.choice([2, 4, 8]),
            "steps": rng.randint(8, 24), "every": rng.choice([4, 8])}


def _full(case):
    """A case with every field of the general run."""
    c = dict(case)
    if c["kind"] == "host":
        c.update(plasma="thermal", precision="mixed", policy="corrected", rel=True, walls=False, sort=True, dt=0.5,
                 dx=1.0)
    elif c["kind"] == "jacobi":
        c.update(plasma="langmuir", precision="fp64", policy="reference", rel=False, walls=False, sort=False, dt=0.5,
                 dx=1.0)
    elif c["kind"] == "gradient":
        c.update(plasma="laser", rel=True, walls=True, sort=False, dt=0.5, dx=1.0)
    c["n"] = (c["nx"], c["ny"], c["nz"])
    return c


def _species(c):
    """(charge, mass, thermal speed, x drift) of each species."""
    ion = math.sqrt(MASS_RATIO)
    if c["plasma"] == "beams":
        return [(-1.0, 1.0, 0.02, 0.3), (-1.0, 1.0, 0.02, -0.3)]
    vth = {"thermal": 0.1, "laser": 0.05, "langmuir": 0.05}[c["plasma"]]
    return [(-1.0, 1.0, vth, 0.0), (1.0, MASS_RATIO, vth / ion, 0.0)]


def _count(c):
    """Particles of one species; the laser's plasma fills the middle half of the box in x."""
    return c["nx"] * c["ny"] * c["nz"] * c["ppc"] // (2 if c["plasma"] == "laser" else 1)


def _wave(c):
    """(amplitude, omega, 1 / width, delay) of the injected pulse of the walled cases."""
    omega = 2.0 * math.pi / 16.0
    fwhm = 8 * c["dt"]
    return 0.5 * omega, omega, math.sqrt(math.log(2.0)) / (0.5 * fwhm), fwhm


# --------------------------------------------------------------------- inputs

def _uniform(shape, gen):
    return torch.rand(shape, dtype=torch.float64, device="cuda", generator=gen)


def _particles(c, seed):
    """Per species [x, y, z, vx, vy, vz, gamma], float64 on the GPU: uniform (with the Langmuir start's
    density wave), Maxwellian, drifting."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    k = _count(c)
    out = []
    for si, (q, m, vth, drift) in enumerate(_species(c)):
        pos = []
        for a in range(3):
            u = _uniform(k, gen)
            if c["plasma"] == "langmuir" and a == 0 and si == 0:
                u = (u - 0.1 / (2.0 * math.pi) * torch.sin(2.0 * math.pi * u)).clamp_(0.0, 1.0 - 2.0 ** -40)
            if c["plasma"] == "laser" and a == 0:
                u.mul_(0.5).add_(0.25)
            # on a grid of 2^-24 cells, as a store of cell and single-precision offset holds positions
            pos.append(u.mul_(c["n"][a] * 2.0 ** 24).floor_().add_(0.25).mul_(c["dx"] * 2.0 ** -24))
        vel = [torch.randn(k, dtype=torch.float64, device="cuda", generator=gen).mul_(vth).clamp_(-0.45, 0.45)
               for _ in range(3)]
        for v in vel:
            v -= v.mean()
        vel[0] += drift
        if c["sort"]:
            key = torch.zeros(k, dtype=torch.int32, device="cuda")
            for a in range(3):
                back = pos[a] - DRIFT * c["dt"] * vel[a]
                key.mul_(c["n"][a]).add_(torch.floor(back / c["dx"]).to(torch.int32).remainder_(c["n"][a]))
                del back
            order = torch.sort(key, stable=True)[1]
            del key
            for arr in (pos, vel):
                for a in range(3):
                    arr[a] = arr[a][order]
            del order
        p = pos + vel
        if c["rel"]:
            p.append((1.0 - vel[0] ** 2 - vel[1] ** 2 - vel[2] ** 2).rsqrt_())
        out.append(p)
    return out


def _densities(c, seed):
    """Charge and current densities of the given-density field start, (n+3)^3 arrays on the GPU: smooth
    clumps over particle noise, mean-free, zero ghost planes."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n = c["n"]
    out = []
    for _ in range(4):
        f = torch.randn(n, dtype=torch.float64, device="cuda", generator=gen).mul_(0.02)
        for a in range(3):
            x = torch.arange(n[a], dtype=torch.float64, device="cuda") / n[a]
            ph = _uniform(1, gen)
            shape = [1, 1, 1]
            shape[a] = n[a]
            f += 0.1 * torch.sin(2.0 * math.pi * (x + ph)).reshape(shape)
        f -= f.mean()
        g = torch.zeros([v + 3 for v in n], dtype=torch.float64, device="cuda")
        g[1:n[0] + 1, 1:n[1] + 1, 1:n[2] + 1] = f
        out.append(g)
    return out


# -------------------------------------------------------------------- prepare

def _config(c, init="constant"):
    names = ("a", "b")
    species = [configs.Species(names[i], q, m, c.get("ppc", 1), vth) for i, (q, m, vth, _) in enumerate(_species(c))]
    kw = {}
    if c["walls"]:
        amp, omega, iw, delay = _wave(c)
        kw = {"waves": [configs.Wave(side=-1, pol=2, amp=amp, omega=omega, inv_width=iw, delay=delay)],
              "part_bc": ("reflecting",) * 2 + ("periodic",) * 4, "field_bc": ("external",) * 2 + ("periodic",) * 4}
    return configs.Config(name="case", n=c["n"], dx=(c["dx"],) * 3, dt=c["dt"], steps=c.get("steps", 1),
                          species=species, omega_pe=OMEGA_PE[c["plasma"]], relativity=int(c["rel"]), init=init,
                          nstep_sort=DRIFT if c["sort"] else 0, **kw)


def _ptr(t):
    return None if t is None else C.cast(t.data_ptr(), C.POINTER(C.c_double))


class _Handle:
    """A simulation handle, freed with the object."""

    def __init__(self, c, info, multigrid=False):
        L = self.L = abi.lib()
        o = abi.Opts()
        L.emoo_default_opts(C.byref(o))
        o.precision = abi.MIXED if c["precision"] == "mixed" else abi.FP64
        o.policy = abi.POLICY_CORRECTED if c["policy"] == "corrected" else abi.POLICY_REFERENCE
        o.dt = c["dt"]
        o.capacity = max(1, info.nparticles_tot)
        o.track_ids = 0
        if multigrid:
            o.poisson_solver = abi.POISSON_MULTIGRID
        self.h = C.c_void_p()
        abi.check(L.emoo_create(C.byref(info), C.byref(o), C.byref(self.h)), "emoo_create")

    def __del__(self):
        if getattr(self, "h", None):
            self.L.emoo_destroy(self.h)
            self.h = None

    def call(self, name, *args):
        abi.check(getattr(self.L, name)(self.h, *args), name)


def _fields(c, names):
    shape = [v + 3 for v in c["n"]]
    return {k: torch.empty(shape, dtype=torch.float64, pin_memory=True) for k in names}


EB = {"Ex": abi.EX, "Ey": abi.EY, "Ez": abi.EZ, "Bx": abi.BX, "By": abi.BY, "Bz": abi.BZ}


def prepare(case, seed):
    c = _full(case)
    if c["kind"] == "gradient":
        parts = []
        for p in _particles(c, seed):
            arr = [v.cpu().numpy() for v in p]
            parts.append(dict(zip(("x", "y", "z", "vx", "vy", "vz", "gamma"), arr)))
        return {"c": c, "problem": differentiate.Problem(
            _config(c), nsteps=c["steps"], slab=(1, c["nx"] // 2), checkpoint_every=c["every"], parts=parts,
            precision=abi.MIXED if c["precision"] == "mixed" else abi.FP64,
            policy=abi.POLICY_CORRECTED if c["policy"] == "corrected" else abi.POLICY_REFERENCE)}
    if c["kind"] == "multigrid":
        c.update(plasma="langmuir", precision="fp64", policy="reference", rel=False, walls=False, sort=False, dt=0.5,
                 dx=1.0)
        cfg = _config(c, init="poisson")
        info = configs.input_info(cfg)
        info.nparticles_tot = info.nparticles_domain = 0
        src = [t.cpu().pin_memory() for t in _densities(c, seed)]
        return {"c": c, "h": _Handle(c, info, multigrid=True), "src": src, "out": _fields(c, EB)}
    parts = _particles(c, seed)
    info = configs.input_info(_config(c, init="poisson" if c["kind"] == "jacobi" else "constant"))
    h = _Handle(c, info)
    s = {"c": c, "h": h, "counts": (C.c_int64 * 6)()}
    if c["precision"] == "fp64" or c["kind"] == "host":
        parts = [[v.cpu().pin_memory() for v in p] for p in parts]
    torch.cuda.synchronize()
    for si, p in enumerate(parts):
        arr = [_ptr(v) for v in p] + [None] * (7 - len(p))
        h.call("emoo_load_particles", si, p[0].numel(), *arr, None)
    if c["kind"] == "jacobi":
        s["zero"] = torch.zeros([v + 3 for v in c["n"]], dtype=torch.float64, pin_memory=True)
        s["out"] = _fields(c, EB)
        return s
    if c["kind"] == "host":
        for si, p in enumerate(parts):
            h.call("emoo_attach_particles", si, p[0].numel(), *[_ptr(v) for v in p])
        h.call("emoo_init_fields", (C.c_int * 4)())
        h.call("emoo_step", 1, s["counts"])  # the sort and the first push
        s.update(parts=parts, out=_fields(c, EB))
        return s
    s.update(parts=parts, out=_fields(c, dict(EB, rho=abi.RHO)))
    s["back"] = [[torch.empty_like(v, pin_memory=not v.is_cuda) for v in p] for p in parts]
    return s


# ------------------------------------------------------------------------ run

def _read_fields(h, out):
    for k, t in out.items():
        h.call("emoo_get_field", EB.get(k, abi.RHO), _ptr(t))
    return out


def run(state):
    c = state["c"]
    if c["kind"] == "gradient":
        r = state["problem"].gradient()
        return {"objective": r["objective"], "grad_theta": r["grad_theta"], "grad_v": r["grad_v"]}
    h = state["h"]
    if c["kind"] == "multigrid":
        for i, t in zip((abi.RHO, abi.JX, abi.JY, abi.JZ), state["src"]):
            h.call("emoo_set_field", i, _ptr(t))
        h.call("emoo_poisson_init", (C.c_int * 4)())
        return _read_fields(h, state["out"])
    if c["kind"] == "jacobi":
        for i in (abi.PHI1, abi.AX1, abi.AY1, abi.AZ1):  # the solve starts from zero potentials
            h.call("emoo_set_field", i, _ptr(state["zero"]))
        rc = h.L.emoo_init_fields(h.h, (C.c_int * 4)())
        if rc != abi.ERR_NOT_CONVERGED:  # the iteration cap, on even periodic grids
            abi.check(rc, "emoo_init_fields")
        return _read_fields(h, state["out"])
    if c["kind"] == "host":
        h.call("emoo_step", c["steps"], state["counts"])
        return {"particles": state["parts"], "fields": _read_fields(h, state["out"]), "crossings": list(state["counts"])}
    for si, p in enumerate(state["parts"]):
        h.call("emoo_set_particles", si, p[0].numel(), *([_ptr(v) for v in p] + [None] * (7 - len(p))))
    h.call("emoo_init_fields", (C.c_int * 4)())
    h.call("emoo_step", c["steps"], state["counts"])
    got = C.c_int64()
    for si, p in enumerate(state["back"]):
        arr = [_ptr(v) for v in p] + [None] * (8 - len(p))
        h.call("emoo_get_particles", si, p[0].numel(), *arr, C.byref(got))
    return {"particles": state["back"], "fields": _read_fields(h, state["out"]), "crossings": list(state["counts"])}


# ----------------------------------------------------------------------- work

def work(case):
    c = _full(case)
    cells = c["nx"] * c["ny"] * c["nz"]
    if c["kind"] == "multigrid":
        return {"bytes": cells * 8.0 * (4 + 6), "flops": cells * 4 * 100.0}
    npart = 2 * _count(c)
    if c["kind"] == "jacobi":
        # an even side: the iteration runs to its cap; its state fits on chip
        return {"bytes": npart * 48.0 + cells * 80.0, "flops": cells * 4 * 10000.0 * 9}
    io = 2 * npart * 8.0 * (7 if c["rel"] else 6) + cells * 7 * 8.0
    state = npart * (56.0 if c["precision"] == "mixed" else (112.0 if c["rel"] else 96.0))
    grid = cells * 32 * (4.0 if c["precision"] == "mixed" else 8.0)
    flops = npart * c["steps"] * 250.0
    if c["kind"] == "host":
        return {"bytes": c["steps"] * (npart * 112.0 + grid), "flops": flops}
    if c["kind"] == "gradient":
        return {"bytes": npart * 56.0 + npart * 24.0 + 4 * c["steps"] * (state + grid), "flops": 4 * flops}
    return {"bytes": io + c["steps"] * (state + grid), "flops": flops}


# ------------------------------------------------- the same in plain FP64 torch

class _Sim:
    """The time loop in plain FP64 torch operations, differentiable (cells and boundary events held)."""

    def __init__(self, c, sizes):
        self.c, self.n, self.d, self.dt = c, c["n"], c["dx"], c["dt"]
        self.corr, self.rel = c["policy"] == "corrected", c["rel"]
        self.tot = [v + 3 for v in self.n]
        self.sx, self.sy = self.tot[1] * self.tot[2], self.tot[2]
        self.L = [v * self.d for v in self.n]
        self.vol = self.d ** 3
        sp = _species(c)
        w = OMEGA_PE[c["plasma"]] ** 2 * sp[0][1] / (4.0 * math.pi * (c["ppc"] / self.vol) * sp[0][0] ** 2)

        def per(f):
            return torch.cat([torch.full((k,), f(s), dtype=torch.float64, device="cuda") for k, s in zip(sizes, sp)])
        self.qp = per(lambda s: 0.5 * self.dt * s[0] / s[1])
        self.q = per(lambda s: w * s[0])
        self.theta = None
        if c["walls"]:
            self.theta = torch.tensor([_wave(c)[0], 0.0], dtype=torch.float64, device="cuda")
        self.ext = [bool(c["walls"]), False, False]

    def start(self):
        z = lambda: torch.zeros(self.tot, dtype=torch.float64, device="cuda")  # noqa: E731
        return [z() for _ in range(3)], [z() for _ in range(6)], 0

    def cell(self, pos):
        return [torch.floor(p.detach() / self.d) + 1.0 for p in pos]

    def index(self, i):
        return (i[0] * self.sx + i[1] * self.sy + i[2]).long()

    def offsets(self, i):
        """Grid offsets of the four edges of component i and the weights' axes."""
        st = [self.sx, self.sy, 1]
        j, k = (i + 1) % 3, (i + 2) % 3
        return st[j], st[k], st[i], j, k

    def weights(self, pos, cell):
        shift = 1.0 if self.corr else 0.0
        r = [p - self.d * (i - shift) for p, i in zip(pos, cell)]
        return r, [self.d - v for v in r]

    def gather(self, E, B, T, pos):
        cell = self.cell(pos)
        o = self.index(cell)
        r, a = self.weights(pos, cell)
        e, b = [], []
        for i in range(3):
            sj, sk, si, j, k = self.offsets(i)
            f = E[i].reshape(-1)
            e.append((a[j] * a[k] * f[o] + r[j] * a[k] * f[o + sj] + r[j] * r[k] * f[o + sj + sk]
                      + a[j] * r[k] * f[o + sk]) / self.d ** 2)
            g = (0.5 * (B[i] + T[i])).reshape(-1)
            b.append((a[i] * g[o] + r[i] * g[o + si]) / self.d)
        return e, b

    def push(self, e, b, v, gamma):
        q = self.qp
        cross = lambda p, s: [p[1] * s[2] - p[2] * s[1], p[2] * s[0] - p[0] * s[2], p[0] * s[1] - p[1] * s[0]]  # noqa: E731
        if not self.rel:
            t = [q * x for x in b]
            ts = 2.0 / (1.0 + q * q * (b[0] ** 2 + b[1] ** 2 + b[2] ** 2))
            vm = [v[a] + q * e[a] for a in range(3)]
            vi = [x + y for x, y in zip(vm, cross(vm, t))]
            vp = [x + ts * y for x, y in zip(vm, cross(vi, t))]
            return [vp[a] + q * e[a] for a in range(3)], gamma
        vxb = cross(v, b)
        up = [gamma * v[a] + q * (e[a] + vxb[a]) + q * e[a] for a in range(3)]
        tau = [q * x for x in b]
        t2 = tau[0] ** 2 + tau[1] ** 2 + tau[2] ** 2
        sigma = 1.0 + up[0] ** 2 + up[1] ** 2 + up[2] ** 2 - t2
        us = up[0] * tau[0] + up[1] * tau[1] + up[2] * tau[2]
        g = torch.sqrt(0.5 * (sigma + torch.sqrt(sigma * sigma + 4.0 * (t2 + us * us))))
        t = [x / g for x in tau]
        s = 1.0 / (1.0 + t[0] ** 2 + t[1] ** 2 + t[2] ** 2)
        c = cross(up, t)
        return [s * (up[a] + us / g * t[a] + c[a]) / g for a in range(3)], g

    def bounds(self, pos, v):
        pos, v = list(pos), list(v)
        for a in range(3):
            hi = self.L[a]
            if self.ext[a]:
                lo, up = pos[a] < 0.0, pos[a] > hi
                pos[a] = torch.where(lo, -pos[a], torch.where(up, 2.0 * hi - pos[a], pos[a]))
                v[a] = torch.where(lo | up, -v[a], v[a])
            else:
                pos[a] = torch.where(pos[a] < 0.0, pos[a] + hi, torch.where(pos[a] > hi, pos[a] - hi, pos[a]))
        return pos, v

    def zeros(self):
        return torch.zeros(self.tot[0] * self.sx, dtype=torch.float64, device="cuda")

    def current(self, pos, v):
        """The reference policy's current at the new positions, with its x-edge index."""
        cell = self.cell(pos)
        o = self.index(cell)
        r, a = self.weights(pos, cell)
        J = []
        for i in range(3):
            sj, sk, _, j, k = self.offsets(i)
            w = self.q * v[i] / self.vol / self.d ** 2
            f = self.zeros().index_add(0, o, w * a[j] * a[k]).index_add(0, o + sj, w * r[j] * a[k])
            f = f.index_add(0, o + sj + sk, w * r[j] * r[k])
            J.append(f.index_add(0, o + (sj if i == 0 else sk), w * a[j] * r[k]).reshape(self.tot))
        return J

    def path_current(self, p0, p1):
        """Villasenor and Buneman's current of a straight move, split at the faces it crosses."""
        u0, du, t = [x / self.d for x in p0], [], []
        for a in range(3):
            u1 = p1[a] / self.d
            f0, f1 = torch.floor(u0[a].detach()), torch.floor(u1.detach())
            step = u1 - u0[a]
            hit = f0 != f1
            t.append(torch.where(hit, (torch.maximum(f0, f1) - u0[a]) / torch.where(hit, step, torch.ones_like(step)),
                                 torch.ones_like(step)))
            du.append(step)
        t = torch.sort(torch.stack(t), dim=0)[0]
        one = torch.ones_like(t[0])
        ends = [torch.zeros_like(one), t[0], t[1], t[2], one]
        J = [self.zeros() for _ in range(3)]
        for k in range(4):
            ta, tb = ends[k], ends[k + 1]
            m, D, c = [], [], []
            for a in range(3):
                ua, ub = u0[a] + ta * du[a], u0[a] + tb * du[a]
                f = torch.floor(0.5 * (ua + ub).detach())
                m.append(0.5 * (ua + ub) - f)
                D.append(ub - ua)
                c.append(f + 1.0)
            o = self.index(c)
            for a in range(3):
                sj, sk, _, j, l = self.offsets(a)
                w = self.q / self.vol / self.dt * self.d * D[a]
                cr = D[j] * D[l] / 12.0
                J[a] = J[a].index_add(0, o, w * ((1 - m[j]) * (1 - m[l]) + cr))
                J[a] = J[a].index_add(0, o + sj, w * (m[j] * (1 - m[l]) - cr))
                J[a] = J[a].index_add(0, o + sk, w * ((1 - m[j]) * m[l] - cr))
                J[a] = J[a].index_add(0, o + sj + sk, w * (m[j] * m[l] + cr))
        return [f.reshape(self.tot) for f in J]

    def rho(self, pos):
        cell = self.cell(pos)
        o = self.index(cell)
        r, a = self.weights(pos, cell)
        f = self.zeros()
        for b in range(8):
            w, off = self.q / self.vol ** 2, 0
            for ax, st in enumerate((self.sx, self.sy, 1)):
                w, off = (w * r[ax], off + st) if b >> ax & 1 else (w * a[ax], off)
            f = f.index_add(0, o + off, w)
        return self.fold([f.reshape(self.tot)], False)[0]

    def at(self, d, i, full):
        """Plane i of dimension d, over the whole or the physical transverse range."""
        s = [slice(None) if full else slice(1, self.n[a] + 1) for a in range(3)]
        s[d] = i
        return tuple(s)

    def fold(self, F, current=True):
        F = [f.clone() for f in F]
        for d in range(3):
            n = self.n[d]
            if self.ext[d]:
                for right in range(2) if self.corr and current else ():
                    for a in range(3):
                        src = (n + 1 if right else 0) if a == d else (n + 2 if right else 0)
                        dst = (n if right else 1) if a == d else (n if right else 2)
                        s, t = self.at(d, src, True), self.at(d, dst, True)
                        add = F[a][s].clone()
                        F[a][t] += -add if a == d else add
                        F[a][s] = 0.0
                continue
            for a, f in enumerate(F):
                if self.corr:
                    for dst, src in ((n, 0), (1, n + 1), (2, n + 2)):
                        f[self.at(d, dst, True)] += f[self.at(d, src, True)].clone()
                elif not current or a != d:
                    f[self.at(d, 1, False)] += f[self.at(d, n + 1, False)].clone()
        return F

    def copies(self, F):
        for d in range(3):
            if self.ext[d]:
                continue
            n = self.n[d]
            for f in F:
                pairs = ((0, n), (n + 1, 1), (n + 2, 2)) if self.corr else ((0, n), (n + 1, 1))
                for dst, src in pairs:
                    f[self.at(d, dst, self.corr)] = f[self.at(d, src, self.corr)].clone()

    def planes(self, E, Brole, t):
        """The x sides' planes: the pulse at the left, zero elsewhere."""
        _, om, iw, delay = _wave(self.c)
        env = math.exp(-((t - delay) * iw) ** 2)
        amp, phase = self.theta[0], self.theta[1] * math.pi / 180.0
        pulse = lambda shift: amp * torch.cos(om * (t + shift) + phase) * env  # noqa: E731
        n = self.n[0]
        for right in range(2):
            for i in range(3):
                ie = (n if i == 0 else n + 1) if right else 1
                ib = (n + 1 if i == 0 else n) if right else 1
                E[i][ie] = pulse(0.0) if i == 1 and not right else 0.0
                Brole[i][ib] = pulse((self.d - self.dt) / 2.0) if i == 2 and not right else 0.0

    def step(self, pos, v, gamma, E, S, swap, t):
        """One step; S: the six B storage slots, swap: which three hold the current B."""
        n, d, dt = self.n, self.d, self.dt
        B, T = (S[3:], S[:3]) if swap else (S[:3], S[3:])
        e, b = self.gather(E, B, T, pos)
        v, gamma = self.push(e, b, v, gamma)
        moved = [pos[a] + dt * v[a] for a in range(3)]
        J = self.path_current(pos, moved) if self.corr else None
        pos, v = self.bounds(moved, v)
        J = self.fold(J if self.corr else self.current(pos, v))
        E, S, swap = [f.clone() for f in E], [f.clone() for f in S], 1 - swap
        B, T = (S[3:], S[:3]) if swap else (S[:3], S[3:])
        P = tuple(slice(1, k + 1) for k in n)

        def sh(f, a, by):
            s = list(P)
            s[a] = slice(1 + by, n[a] + 1 + by)
            return f[tuple(s)]
        for i in range(3):
            j, k = (i + 1) % 3, (i + 2) % 3
            curl = (T[j][P] - sh(T[j], k, -1)) / d - (T[k][P] - sh(T[k], j, -1)) / d
            E[i][P] = E[i][P] - dt * (curl + 4.0 * math.pi * J[i][P])
        if self.corr:
            self.copies(E)
            if self.c["walls"]:
                self.planes(E, B, t)
        new = []
        for i in range(3):
            j, k = (i + 1) % 3, (i + 2) % 3
            new.append(T[i][P] + dt * ((sh(E[j], k, 1) - E[j][P]) / d - (sh(E[k], j, 1) - E[k][P]) / d))
        for i in range(3):
            B[i][P] = new[i]
        if self.corr:
            self.copies(E + S)
            if self.c["walls"]:
                self.planes(E, B, t)
        else:
            if self.c["walls"]:
                self.planes(E, B, t)
            self.copies(E + S[:3])
        return pos, v, gamma, E, S, swap


def _join(parts):
    return [torch.cat([p[a] for p in parts]) for a in range(len(parts[0]))]


def _sorted(c, parts):
    out = []
    for p in parts:
        key = torch.zeros(p[0].numel(), dtype=torch.int64, device="cuda")
        for a in range(3):
            key = key * c["n"][a] + torch.floor(p[a] / c["dx"]).long()
        order = torch.sort(key, stable=True)[1]
        out.append([v[order] for v in p])
    return out


def _exact_loop(c, seed):
    parts = _particles(c, seed)
    if c["sort"]:
        parts = _sorted(c, parts)
    sizes = [p[0].numel() for p in parts]
    sim = _Sim(c, sizes)
    st = _join(parts)
    pos, v, gamma = st[:3], st[3:6], st[6] if c["rel"] else None
    E, S, swap = sim.start()
    t = 0.0
    for _ in range(c["steps"] + (c["kind"] == "host")):
        pos, v, gamma, E, S, swap = sim.step(pos, v, gamma, E, S, swap, t)
        t += c["dt"]
    whole = pos + v + ([gamma] if c["rel"] else [])
    cut = [torch.split(a, sizes) for a in whole]
    fields = dict(zip(EB, E + S[:3]))
    if c["kind"] == "loop":
        fields["rho"] = sim.rho(pos)
    return {"particles": [[a[si] for a in cut] for si in range(len(sizes))], "fields": fields, "crossings": None}


def _exact_gradient(c, seed):
    from torch.utils.checkpoint import checkpoint
    parts = _particles(c, seed)
    sim = _Sim(c, [p[0].numel() for p in parts])
    st = _join(parts)
    v0 = torch.stack(st[3:6]).requires_grad_(True)
    sim.theta.requires_grad_(True)
    pos, v, gamma = st[:3], list(v0), st[6]
    E, S, swap = sim.start()
    t = 0.0
    for _ in range(c["steps"]):
        pos, v, gamma, E, S, swap = checkpoint(sim.step, pos, v, gamma, E, S, swap, t, use_reentrant=False)
        t += c["dt"]
    B = S[3:] if swap else S[:3]
    sl = (slice(2, c["nx"] // 2 + 1), slice(1, c["ny"] + 1), slice(1, c["nz"] + 1))
    obj = 0.5 * sim.vol * sum((f[sl] ** 2).sum() for f in E + list(B))
    gth, gv = torch.autograd.grad(obj, (sim.theta, v0))
    return {"objective": float(obj.detach()), "grad_theta": gth.cpu(), "grad_v": gv.cpu()}


def _exact_start(c, R, solve):
    """E and B of the field start from the physical densities R and a solver of laplacian(u) = -4 pi R."""
    n = c["n"]
    up = lambda f, a: torch.roll(f, -1, a)  # noqa: E731
    phi, ax, ay, az = [solve(r) for r in R]
    E = [phi - up(phi, a) for a in range(3)]
    B = [up(az, 1) - az + up(az, 2) - ay, up(ax, 2) - ax + up(ax, 0) - az, up(ay, 0) - ay + up(ay, 1) - ax]
    out = {}
    for name, f in zip(EB, E + B):
        g = torch.zeros([k + 3 for k in n], dtype=torch.float64, device="cuda")
        g[1:n[0] + 1, 1:n[1] + 1, 1:n[2] + 1] = f
        for d in range(3):
            for dst, src in ((0, n[d]), (n[d] + 1, 1)):
                s = [slice(1, n[a] + 1) for a in range(3)]
                t = list(s)
                s[d], t[d] = src, dst
                g[tuple(t)] = g[tuple(s)]
        out[name] = g
    return out


def _exact_jacobi(c, seed):
    parts = _particles(c, seed)
    sim = _Sim(c, [p[0].numel() for p in parts])
    st = _join(parts)
    P = tuple(slice(1, k + 1) for k in c["n"])
    J = sim.fold(sim.current(st[:3], st[3:6]))
    R = [f[P].contiguous() for f in [sim.rho(st[:3])] + J]

    def solve(r):
        u = torch.zeros_like(r)
        f = 4.0 * math.pi / 6.0 * r
        last = u  # what the first potential's storage holds: the result of every second sweep
        for it in range(10001):
            w = f.clone()
            for a in range(3):
                w += (torch.roll(u, 1, a) + torch.roll(u, -1, a)) / 6.0
            stop = it % 25 == 24 and (w - u).abs().max().item() < 1e-12
            u = w
            if it % 2:
                last = u
            if stop:
                break
        return last
    return _exact_start(c, R, solve)


def _exact_multigrid(c, seed):
    n = c["n"]
    P = tuple(slice(1, k + 1) for k in n)
    lam = 0.0
    for a in range(3):
        k = torch.arange(n[a], dtype=torch.float64, device="cuda")
        shape = [1, 1, 1]
        shape[a] = n[a]
        lam = lam + (2.0 * torch.cos(2.0 * math.pi * k / n[a]) - 2.0).reshape(shape)
    lam[0, 0, 0] = 1.0

    def solve(r):
        f = torch.fft.fftn(-4.0 * math.pi * (r - r.mean())) / lam
        f[0, 0, 0] = 0.0
        return torch.fft.ifftn(f).real
    return _exact_start(c, [f[P] for f in _densities(c, seed)], solve)


def exact(case, seed):
    c = _full(case)
    if c["kind"] == "multigrid":
        return _exact_multigrid(c, seed)
    if c["kind"] == "jacobi":
        return _exact_jacobi(c, seed)
    if 2 * _count(c) * c["steps"] > 3e8:
        return None  # too long
    return _exact_gradient(c, seed) if c["kind"] == "gradient" else _exact_loop(c, seed)
