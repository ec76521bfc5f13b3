"""The split Arnoldi passes with several blocks per SM (dot shape 13, axpy shape
11) against the default shapes, and the blocked back-substitution at cycle
lengths around its 32-column blocks against the oracle."""
import numpy as np
import pytest

from cugmres_b200 import problems
from test_gpu_arnoldi_shapes import _compare, _run, default_run  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("env", [{"CUGMRES_DOTS2_SHAPE": "13"}, {"CUGMRES_AXPY2_SHAPE": "11"}])
def test_split_pass_shape(default_run, tmp_path, env):  # noqa: F811
    _compare(_run(tmp_path, "split", env), default_run)


@pytest.mark.parametrize("m", [1, 31, 32, 33, 64, 65, 97])
def test_backsolve_around_its_blocks(solver, oracle, m):
    pr = problems.helmholtz(96, 4.0, seed=9)
    solver.set_operator(pr["g_block"], pr["chi"], pr["chi_scale"])
    x, info = solver.solve(pr["b"], restart=m, max_iter=m, tol=1e-14)
    o = oracle.gmres(oracle.spectrum(pr["g_block"], solver.L), pr["chi"] * pr["chi_scale"], pr["b"], restart=m,
                     maxiter=m, tol=1e-14)
    assert info["iterations"] == m
    assert np.linalg.norm(x - o["x"]) <= 1e-10 * np.linalg.norm(o["x"])
