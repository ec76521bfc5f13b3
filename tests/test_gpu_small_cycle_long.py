"""One-kernel cycles of small grids over several hundred steps: accuracy and residual
history against the launched cycles (CUGMRES_SMALL_CYCLE=0)."""
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

FLOORS = r"""
import sys, numpy as np
sys.path.insert(0, sys.argv[1])
import cugmres_b200 as cg
from cugmres_b200 import problems as P
out = []
for seed in range(8):
    pr = P.helmholtz(64, 14.0, seed=seed, cells_per_wavelength=12.0)
    with cg.Solver(0) as s:
        s.set_operator(pr["g_block"], pr["chi"], pr["chi_scale"])
        _, info = s.solve(pr["b"], restart=900, max_iter=900, tol=0.0, precision=sys.argv[3], inner_tol=1e-12)
        out.append(info["rel_residual_true"])
np.save(sys.argv[2], np.asarray(out))
"""


def _both(script, tmp_path, *args):
    got = []
    for on in ("1", "0"):
        f = str(tmp_path / f"s{on}.npy")
        r = subprocess.run([sys.executable, "-c", script, ROOT, f, *args], env=dict(os.environ, CUGMRES_SMALL_CYCLE=on),
                           capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        got.append(np.load(f))
    return got


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_long_cycles_lose_no_more(tmp_path, cuda_device, precision):
    """The residual that rounding leaves after 900 steps.  One system's scatters by a
    factor of 1.4 between runs that round differently, the mean of eight by 1.4^(1/sqrt 8) =
    1.13; sums over all basis vectors in a single chain are 1.5 times off in complex64."""
    one, launched = _both(FLOORS, tmp_path, precision)
    assert np.exp(np.mean(np.log(one / launched))) <= 1.25
