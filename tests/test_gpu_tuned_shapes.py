"""Launch shapes differ in rounding, so a system that a sweep solves beside others and
a context solves alone has the same bits only if both take the same ones."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

SCRIPT = r"""
import sys, numpy as np
sys.path.insert(0, sys.argv[1])
import cugmres_b200 as cg
from cugmres_b200 import problems as P
pr = P.helmholtz(int(sys.argv[2]), 3.0, seed=1)
for precision in ("fp64", "mixed"):
    kw = dict(restart=10, max_iter=60, tol=1e-10, precision=precision)
    xs, _ = cg.solve_batch([pr], **kw)
    with cg.Solver(0) as s:
        s.set_operator(pr["g_block"], pr["chi"], pr["chi_scale"])
        y, _ = s.solve(pr["b"], **kw)
    assert np.array_equal(xs[0], y), precision
"""


@pytest.mark.parametrize("N", [33, 64])
def test_small_system_alone_and_in_a_sweep(cuda_device, tmp_path, N):
    """Whatever choices for the two kinds of context the tuner's file holds."""
    import torch
    device = torch.cuda.get_device_name(cuda_device).replace(" ", "_")
    cache = tmp_path / "tune.txt"
    cache.write_text("".join(f"{device}|128|{p}|{v}\n" for p in (0, 1) for v in ("t4 2 2 2", "t4s 0 0 4")))
    r = subprocess.run([sys.executable, "-c", SCRIPT, ROOT, str(N)], env=dict(os.environ, CUGMRES_TUNE_CACHE=str(cache)),
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
