"""Solves and sweeps where the device memory ends: an allocation that fails is reported
as CG_ERR_OOM and leaves the context and the process usable."""
import numpy as np
import pytest

import cugmres_b200 as cg
from cugmres_b200 import problems

pytestmark = pytest.mark.gpu

N, L = 1024, 2048
UNIT = 16 * N * N  # bytes of an FP64 vector


@pytest.fixture
def little_memory(cuda_device):
    """A device with about 1.3 GB left; yields the bytes that are."""
    import torch
    warm = problems.helmholtz(N, 2.0, seed=0, with_green=False)
    cg.solve_batch([warm], restart=4, max_iter=2)  # tunes and loads what a sweep loads
    torch.cuda.empty_cache()
    hog = torch.empty(max(0, torch.cuda.mem_get_info()[0] - 1300 * 10 ** 6), dtype=torch.uint8, device="cuda")
    yield torch.cuda.mem_get_info()[0]
    del hog
    torch.cuda.empty_cache()


def test_solve_after_one_that_did_not_fit(little_memory, solver):
    pr = problems.helmholtz(N, 2.0, seed=0, with_green=False)
    solver.set_operator_green(N, pr["chi"], pr["chi_scale"], k0=pr["k0"], h=pr["h"])
    kw = dict(max_iter=3, tol=1e-10)
    x, info = solver.solve(pr["b"], restart=8, **kw)
    with pytest.raises(cg.CugmresError) as e:
        solver.solve(pr["b"], restart=little_memory // UNIT + 16, **kw)
    assert e.value.status == cg._lib.CG_ERR_OOM
    y, again = solver.solve(pr["b"], restart=8, **kw)
    assert again["iterations"] == info["iterations"] and np.array_equal(x, y)


def test_sweep_goes_on_after_a_system_that_does_not_fit(little_memory):
    """mode="contexts" reports each system's status; the context of one that failed takes the next."""
    big = problems.helmholtz(N, 2.0, seed=0, with_green=False)
    small = problems.helmholtz(96, 2.0, seed=0, with_green=False)
    with pytest.raises(cg.CugmresError) as e:
        cg.solve_batch([big, small], mode="contexts", workers=1, restart=little_memory // UNIT + 16, max_iter=3)
    assert e.value.status == cg._lib.CG_ERR_OOM
    _, infos = cg.solve_batch([small], restart=8, max_iter=3)
    assert infos[0]["iterations"] == 3


# an operator's arrays in a context: spectra, contrasts, T, three vectors, twiddles
OPERATOR = 24 * (L // 2 + 1) ** 2 + 16 * N * N + 16 * N * L + 3 * UNIT + 24 * 4 * L
SLACK = 48 * 10 ** 6  # workspaces and what the runtime takes; the set-up's temporaries are 92 MB


def test_sweep_has_the_memory_of_its_set_up(little_memory):
    """A bucket that fits beside the operator's arrays, but not beside the temporaries of their set-up."""
    pr = problems.helmholtz(N, 2.0, seed=0, with_green=False)
    bucket = 16 * N * L + 16 * (L // 2 + 1) ** 2 + 8 * N * N + 2 * UNIT
    restart = (little_memory - OPERATOR - bucket - SLACK) // UNIT - 2
    _, infos = cg.solve_batch([pr], restart=int(restart), max_iter=3)
    assert infos[0]["iterations"] == 3


def test_contexts_have_the_memory_of_their_set_up(little_memory):
    big = problems.helmholtz(N, 2.0, seed=0, with_green=False)
    small = problems.helmholtz(16, 2.0, seed=0, with_green=False)
    restart = (little_memory - OPERATOR - SLACK) // UNIT - 2
    _, infos = cg.solve_batch([big, small], mode="contexts", workers=2, restart=int(restart), max_iter=3)
    assert [i["iterations"] for i in infos] == [3, 3]
