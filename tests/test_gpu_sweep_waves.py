"""Buckets of one sweep run side by side, each on its own stream.  A bucket
launches the same kernels on its own arrays whatever runs beside it, so every
system has to come out bit for bit as in a sweep of its grid side alone.  The
sides take in the one-kernel cycles (L = 128), embeddings that change between
buckets and, with max_bucket = 1, more buckets than one wave holds."""
import numpy as np
import pytest

import cugmres_b200 as cg
from cugmres_b200 import problems as P

pytestmark = pytest.mark.gpu

SIDES = (33, 64, 65, 48, 130, 97, 64, 33, 200, 64, 65)


def _systems():
    return [P.helmholtz(N, 2.0 + 0.2 * i, seed=40 + i, cells_per_wavelength=18.0, with_green=False)
            for i, N in enumerate(SIDES)]


@pytest.mark.parametrize("max_bucket", [0, 1])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_waves_match_sweeps_of_one_side(cuda_device, precision, max_bucket):
    systems = _systems()
    kw = dict(device=cuda_device, restart=20, max_iter=60, tol=1e-9, precision=precision, max_bucket=max_bucket)
    xs, infos = cg.solve_batch(systems, **kw)
    for N in sorted(set(SIDES)):
        ids = [i for i, side in enumerate(SIDES) if side == N]
        ys, alone = cg.solve_batch([systems[i] for i in ids], **kw)
        for i, y, info in zip(ids, ys, alone):
            assert infos[i]["iterations"] == info["iterations"] and infos[i]["status"] == info["status"]
            assert np.array_equal(xs[i], y), (N, i)


def test_failing_bucket_ends_the_sweep(cuda_device):
    """A right-hand side with a NaN in the last bucket is refused, and the next sweep runs."""
    systems = _systems()
    bad = dict(systems[0], b=systems[0]["b"].copy())
    bad["b"][3, 5] = np.nan
    with pytest.raises(cg.CugmresError):
        cg.solve_batch([systems[4], bad], device=cuda_device, restart=20, max_iter=60)
    _, infos = cg.solve_batch([systems[4], systems[0]], device=cuda_device, restart=20, max_iter=60, tol=1e-6)
    assert all(i["iterations"] > 0 for i in infos)


def test_seconds_leave_out_the_set_ups_of_other_buckets(cuda_device):
    """One step per system, so a bucket's time is its set-up.  The largest grid's, set up
    first, used to hold the set-ups of the three buckets beside it as well: three times
    its own.  The least of some runs, since allocations take a varying time."""
    systems = [P.helmholtz(N, 2.0, seed=i, with_green=False) for N in (260, 200, 130, 96) for i in range(6)]
    kw = dict(device=cuda_device, restart=20, max_iter=1, tol=1e-10)
    cg.solve_batch(systems, **kw)  # tunes
    alone = min(cg.solve_batch(systems[:6], **kw)[1][0]["seconds"] for _ in range(8))
    beside = min(cg.solve_batch(systems, **kw)[1][0]["seconds"] for _ in range(8))
    assert beside <= 1.8 * alone


def test_time_limit_ends_each_bucket(cuda_device):
    """With a time limit the buckets run one after the other, each against its own clock: the
    limit ends the hard systems at a cycle boundary and leaves the easy one alone.  (The
    limit counts a bucket's set-up, whose allocations have been seen to take a second.)"""
    import ctypes
    lib = cg._lib
    systems = [P.helmholtz(256, 12.0, seed=1, with_green=False), P.helmholtz(200, 12.0, seed=2, with_green=False),
               P.helmholtz(40, 1.5, seed=3, with_green=False)]
    cg.solve_batch(systems, device=cuda_device, restart=20, max_iter=20)  # tunes
    arr, keep = (lib.CgSystem * 3)(), []
    for i, s in enumerate(systems):
        chi, b = np.ascontiguousarray(s["chi"]), np.ascontiguousarray(s["b"], np.complex128)
        x = np.zeros_like(b)
        keep.append((chi, b, x))
        arr[i] = lib.CgSystem(s["N"], None, chi.ctypes.data, s["chi_scale"], b.ctypes.data, x.ctypes.data, s["k0"], s["h"])
    o = lib.CgOpts()
    lib.lib().cugmres_default_opts(ctypes.byref(o))
    o.restart, o.max_iter, o.tol, o.timeout_s = 20, 10 ** 6, 1e-10, 2.5
    res = (lib.CgResult * 3)()
    lib.check(lib.lib().cugmres_solve_buckets(cuda_device, 3, arr, ctypes.byref(o), 0, res), "solve_buckets")
    assert [r.status for r in res] == [lib.CG_ERR_TIMEOUT, lib.CG_ERR_TIMEOUT, lib.CG_OK]
    for r in list(res)[:2]:
        assert 2.5 < r.seconds < 6.0 and r.iterations > 100
    assert res[2].rel_residual_true <= 1e-10
