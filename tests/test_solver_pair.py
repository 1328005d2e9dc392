"""Several solvers alive at once: what one sets up leaves the others as they were."""
import numpy as np
import pytest

from falcon_gb300 import solver as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("large,small", [
    ((64, 96), (48, 96)),     # clusters of the same kernel
    ((16, 30), (8, 15)),      # single CTAs
])
def test_solver_created_first_solves_after_a_smaller_one_is_created(built_lib, large, small):
    a = S.Solver(S.pfss_spec([large], device=0))
    b = S.Solver(S.pfss_spec([small], device=0))
    fa, fb = a.coarse_form(), b.coarse_form()
    # the coarsest level runs the same kernel in both, with more shared memory in the first
    assert (fa["ctas"] > 1) == (fb["ctas"] > 1) and fa["cells"] == fb["cells"] > 0 and fa["slots"] > fb["slots"]
    for sv in (a, b, a):
        sv.set_smoothing(2, 2, 16)   # drops the captured graphs
        assert sv.solve(tol=1e-9, max_iter=300)["converged"] == 1
        assert (sv.problem_residuals() <= 1e-9).all()
    a.close()
    b.close()
