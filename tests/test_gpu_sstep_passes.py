"""Where s-step cycles leave out the second Gram-Schmidt pass: restarts up to 512 follow
the short cycles' rule, longer ones keep the pass unless a block hardly needed it."""
import pytest

from cugmres_b200 import problems

pytestmark = pytest.mark.gpu


def test_second_pass_left_out_up_to_512_steps(solver):
    pr = problems.helmholtz(1024, 4.0, seed=0)
    solver.set_operator(pr["g_block"], pr["chi"], pr["chi_scale"])
    moved, residual = {}, {}
    for restart in (100, 512, 516):
        solver.profile(True)
        _, info = solver.solve(pr["b"], restart=restart, max_iter=60, tol=1e-10, ortho="sstep", sstep=4)
        moved[restart], residual[restart] = solver.profile_read()["dots"]["bytes"], info["rel_residual_true"]
        solver.profile(False)
        assert info["iterations"] == 60
    # the first 60 steps are the same, whatever the restart; two passes read twice the vectors of one
    assert moved[512] == moved[100]
    assert moved[512] <= 0.75 * moved[516]
    assert abs(residual[512] - residual[516]) <= 1e-6 * residual[516]
