"""Grids of one thread-block cluster (33 <= N <= 64): the one-kernel restart cycle
and product against the oracle and against the launched kernels, at the sides
where the rows' split over 16 CTAs changes, in both precisions and directions,
with cycles that end by budget, restart and tolerance, and in buckets."""
import os
import subprocess
import sys

import numpy as np
import pytest

import cugmres_b200 as cg
from conftest import ROOT
from cugmres_b200 import problems

pytestmark = pytest.mark.gpu

SIDES = [33, 34, 47, 48, 49, 63, 64]


@pytest.mark.parametrize("N", SIDES)
def test_products_match_oracle(solver, oracle, N):
    pr = problems.helmholtz(N, 4.0, seed=N)
    solver.set_operator(pr["g_block"], pr["chi"], pr["chi_scale"])
    gh, c = oracle.spectrum(pr["g_block"], solver.L), pr["chi"] * pr["chi_scale"]
    rng = np.random.default_rng(N)
    x = rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N))
    for transpose, ref in ((False, oracle.matvec(gh, c, x)), (True, oracle.matvec_transpose(gh, c, x))):
        # the tolerances of the other products: FFT rounding in FP64 and FP32
        y = solver.matvec(x, transpose=transpose)
        assert np.abs(y - ref).max() <= 1e-13 * np.abs(ref).max()
        y = solver.matvec(x.astype(np.complex64), precision="fp32", transpose=transpose)
        assert np.abs(y - ref).max() <= 2e-6 * np.abs(ref).max()


@pytest.mark.parametrize("N", SIDES)
@pytest.mark.parametrize("restart,max_iter", [(1, 3), (7, 20), (60, 25)])
def test_cycles_match_oracle(solver, oracle, N, restart, max_iter):
    pr = problems.helmholtz(N, 3.0, seed=N)
    solver.set_operator(pr["g_block"], pr["chi"], pr["chi_scale"])
    x, info = solver.solve(pr["b"], restart=restart, max_iter=max_iter, tol=1e-12)
    o = oracle.gmres(oracle.spectrum(pr["g_block"], solver.L), pr["chi"] * pr["chi_scale"], pr["b"], restart=restart,
                     maxiter=max_iter, tol=1e-12)
    assert abs(info["iterations"] - o["iterations"]) <= 1  # some sides converge within the budget
    assert np.linalg.norm(x - o["x"]) <= 1e-10 * np.linalg.norm(o["x"])


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("mixed", 1e-10)])
def test_buckets_of_clusters_match_single_solves(cuda_device, precision, tol):
    systems = [problems.helmholtz(N, 2.0 + 0.5 * i, seed=i) for i, N in enumerate([40] * 11 + [64] * 3)]
    xs, infos = cg.solve_batch(systems, restart=50, max_iter=400, tol=tol, precision=precision)
    for pr, x, info in zip(systems, xs, infos):
        with cg.Solver(cuda_device) as s:
            s.set_operator(pr["g_block"], pr["chi"], pr["chi_scale"])
            y, one = s.solve(pr["b"], restart=50, max_iter=400, tol=tol, precision=precision)
        # the same kernel runs alone and in the bucket
        assert (info["status"], info["iterations"]) == (one["status"], one["iterations"]) and np.array_equal(x, y)


SCRIPT = r"""
import sys, numpy as np
sys.path.insert(0, sys.argv[1])
import cugmres_b200 as cg
from cugmres_b200 import problems as P
out = {}
for N in (33, 50, 64):
    pr = P.helmholtz(N, 3.0, seed=N)
    s = cg.Solver(0).set_operator(pr["g_block"], pr["chi"], pr["chi_scale"])
    for tr in (False, True):
        x, info = s.solve(pr["b"], restart=40, max_iter=300, tol=1e-11, transpose=tr)
        out[f"x_{N}_{tr}"], out[f"h_{N}_{tr}"] = x, info["res_hist"]
np.savez(sys.argv[2], **out)
"""


def test_one_kernel_follows_the_launched_cycle(tmp_path, cuda_device):
    got = []
    for on in ("1", "0"):
        f = str(tmp_path / f"s{on}.npz")
        r = subprocess.run([sys.executable, "-c", SCRIPT, ROOT, f], env=dict(os.environ, CUGMRES_SMALL_CYCLE=on),
                           capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        got.append(np.load(f))
    for k in got[0].files:
        # converged solves of the same scheme: only the order of the sums differs
        assert got[0][k].shape == got[1][k].shape, k
        assert np.linalg.norm(got[0][k] - got[1][k]) <= 1e-9 * np.linalg.norm(got[1][k]), k
