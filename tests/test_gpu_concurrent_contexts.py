"""Contexts and networks of different sizes on several host threads: a kernel's limit
of dynamic shared memory is shared by all of them, so no launch may lower it below
what another thread's launch needs."""
import threading

import numpy as np
import pytest

import cugmres_b200 as cg
from cugmres_b200 import learned, problems

pytestmark = pytest.mark.gpu


def _together(jobs):
    """Runs every job on a thread of its own; the first exception is raised here."""
    failed = []

    def guarded(job):
        try:
            job()
        except Exception as e:  # noqa: BLE001
            failed.append(e)

    threads = [threading.Thread(target=guarded, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if failed:
        raise failed[0]


def _solves(N, restart, precision, repeats, products):
    """Repeated solves and products of one context give the bits of the first ones."""
    pr = problems.helmholtz(N, 3.0, seed=N)
    kw = dict(restart=restart, max_iter=12, tol=1e-12, precision=precision)

    def job():
        with cg.Solver(0) as s:
            s.set_operator(pr["g_block"], pr["chi"], pr["chi_scale"])
            x0, _ = s.solve(pr["b"], **kw)
            y0 = s.matvec(pr["b"])
            for _ in range(repeats):
                x, _ = s.solve(pr["b"], **kw)
                assert np.array_equal(x, x0)
                for _ in range(products):
                    assert np.array_equal(s.matvec(pr["b"]), y0)
    return job


def test_one_kernel_cycles_of_several_sizes(cuda_device):
    cases = [(33, 100, "fp64"), (48, 300, "fp64"), (64, 800, "fp64"), (64, 50, "fp64"), (40, 500, "fp64"),
             (64, 200, "mixed"), (33, 600, "mixed"), (50, 900, "mixed")]
    _together([_solves(*c, repeats=60, products=10) for c in cases])


def test_long_restarts_of_several_lengths(cuda_device):
    # launched cycles whose coefficients take more than 48 KB of a block
    cases = [(20, 4400, "fp64"), (24, 3600, "fp64"), (28, 4000, "mixed"), (70, 3800, "fp64"), (72, 3300, "mixed")]
    _together([_solves(*c, repeats=40, products=1) for c in cases])


def test_networks_of_several_heights(cuda_device):
    def forwards(H, W):
        rng = np.random.default_rng(H)
        chi, k0h = rng.random((1, H, W)).astype(np.float32), np.asarray([0.3], np.float32)
        r = (rng.standard_normal((1, H, W)) + 1j * rng.standard_normal((1, H, W))).astype(np.complex64)

        def job():
            net = learned.FNO(0, seed=0)
            z0 = net.forward(chi, k0h, r)
            for _ in range(100):
                assert np.array_equal(net.forward(chi, k0h, r), z0)
            net.close()
        return job

    _together([forwards(*s) for s in ((32, 32), (512, 32), (64, 64), (1000, 40))])
