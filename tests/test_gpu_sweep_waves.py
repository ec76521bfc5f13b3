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
