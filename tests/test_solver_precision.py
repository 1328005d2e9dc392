"""What the solver's inner iteration keeps of its vectors: float-float values."""
import numpy as np
import pytest

from falcon_gb300 import solver as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spec", [
    lambda: S.pfss_spec([(16, 30), (24, 45)], device=0),
    lambda: S.conduction_spec(nr=32, nt=32, np_=96, device=0),
])
def test_plain_cg_searches_along_the_whole_residual(built_lib, spec):
    """The first step of CG without a preconditioner from x0 = 0 is x = alpha b per problem.
    A float-float b keeps 2^-48 of each value and the step rounds four times; an FP32
    direction would be off by up to 2^-25 = 3e-8."""
    sv = S.Solver(spec())
    rng = np.random.default_rng(3)
    b = rng.uniform(0.5, 1.0, sv.rhs().shape)
    sv.set_rhs(b)
    sv.set_guess(np.zeros_like(b))
    sv.solve(tol=1e-12, max_iter=1, precond=S.PRECOND_NONE, check=False)
    x, first = sv.solution(), sv.problem_blocks()
    for q in range(sv.nproblems):
        ratio = x[first[q]:first[q + 1]] / b[first[q]:first[q + 1]]
        assert np.abs(ratio / np.median(ratio) - 1.0).max() <= 16 * 2.0 ** -48
    sv.close()
