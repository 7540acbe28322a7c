"""Handles used by host threads of their own, one a thread, on grids of
different sizes: limits of a kernel that are set for the device (its dynamic
shared memory) must hold for every handle, whoever set them last."""
import threading

import numpy as np
import pytest

from apc_524_project_gb300 import abi, configs
from backends import GpuBackend

pytestmark = pytest.mark.gpu


def _in_threads(work, args):
    """work(arg, start) in a thread each, together; the exceptions that it raised."""
    start, errors = threading.Barrier(len(args)), []

    def run(a):
        try:
            work(a, start)
        except Exception as e:  # noqa: BLE001
            start.abort()
            errors.append((a, e))

    threads = [threading.Thread(target=run, args=(a,)) for a in args]
    for t in threads:
        t.start()
    for t in threads:
        t.join(timeout=120)
        assert not t.is_alive()
    return errors


def test_tiled_jacobi_starts_on_two_grids():
    """Without charge or current every potential is zero from the first sweep
    on: short solves, so that the threads' launches interleave."""
    def work(n, start):
        g = GpuBackend(configs.input_info(configs.tiny("threads", n=n, init="poisson")), 0.4)
        start.wait(60)
        for _ in range(400):
            rc, iters = g.poisson_init()
            assert rc == abi.OK and iters == [0] * 4, (rc, iters)
        g.close()

    assert _in_threads(work, [(64, 64, 64), (6, 5, 4)]) == []


def _multigrid(n):
    """A handle's first solve on a grid of random charge: cycles of the four potentials."""
    g = GpuBackend(configs.input_info(configs.tiny("threads", n=n, init="poisson")), 0.4,
                   poisson_solver=abi.POISSON_MULTIGRID)
    rho = np.zeros(g.shape)
    v = np.random.default_rng(1).normal(0, 1, n)
    rho[1:n[0] + 1, 1:n[1] + 1, 1:n[2] + 1] = v - v.mean()
    g.set_field(abi.RHO, rho)
    rc, cycles = g.poisson_init()
    g.close()
    assert rc == abi.OK, rc
    return cycles


def test_multigrid_set_up_on_four_grids():
    """The 16^3 level's tail takes 80 KB of shared memory, the others' a few, each its own."""
    grids = [(16, 16, 16), (4, 6, 5), (4, 4, 4), (6, 5, 4)]
    alone = {n: _multigrid(n) for n in grids}

    def work(n, start):
        start.wait(60)
        for _ in range(100):
            assert _multigrid(n) == alone[n]

    assert _in_threads(work, grids) == []
