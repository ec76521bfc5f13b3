"""The restart cycle's loop graph at its edges: restarts below, at and above the
steps of one loop body, budgets that end inside it, and the context's cached
graphs under new vectors and alternating directions."""
import numpy as np
import pytest

import cugmres_b200 as cg
from cugmres_b200 import problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ortho", ["dcgs2", "cgs2"])
@pytest.mark.parametrize("restart", [1, 2, 3, 4, 5, 9])
def test_restarts_around_the_loop_body(solver, oracle, restart, ortho):
    pr = problems.helmholtz(40, 2.25, seed=3)
    solver.set_operator(pr["g_block"], pr["chi"], pr["chi_scale"])
    x, info = solver.solve(pr["b"], restart=restart, max_iter=11, tol=1e-14, ortho=ortho)
    o = oracle.gmres(oracle.spectrum(pr["g_block"], solver.L), pr["chi"] * pr["chi_scale"], pr["b"], restart=restart,
                     maxiter=11, tol=1e-14)
    assert info["iterations"] == 11
    assert np.linalg.norm(x - o["x"]) <= 1e-10 * np.linalg.norm(o["x"])


def test_cached_graphs_follow_vectors_and_direction(solver, cuda_device):
    import torch
    pr = problems.helmholtz(48, 4.0, seed=5)
    solver.set_operator(pr["g_block"], pr["chi"], pr["chi_scale"])
    rng = np.random.default_rng(0)
    for i in range(6):
        b = rng.standard_normal((48, 48)) + 1j * rng.standard_normal((48, 48))
        kw = dict(restart=20, max_iter=50, tol=1e-12, transpose=bool(i % 2))
        given = torch.from_numpy(b).cuda() if i >= 2 else b
        x, _ = solver.solve(given, **kw)
        with cg.Solver(cuda_device) as fresh:
            fresh.set_operator(pr["g_block"], pr["chi"], pr["chi_scale"])
            y, _ = fresh.solve(b, **kw)
        x = x.cpu().numpy() if i >= 2 else x
        assert np.array_equal(x, y)
