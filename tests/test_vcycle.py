"""The V-cycle's forms (sweeps that interpolate their halo on the fly, the coarsest
level's sweeps in one launch of a CTA or a cluster per problem, separate launches for
few of them) as a preconditioner: solves take no more iterations than the CPU's FP64
V-cycle with the same smoothing does, on blocks of powers of two and others, on one and
several problems, and reach the same solution."""
import numpy as np
import pytest

import oracle
from falcon_gb300 import solver as S

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built(built_lib, oracle_lib):
    return built_lib


@pytest.mark.parametrize("sizes,block,nlevels,smoothing", [
    ([(24, 45)], 8, 3, (2, 2, 16)),                        # one CTA on the coarsest level
    ([(24, 45), (16, 30), (33, 60)], 8, 3, (2, 2, 3)),     # uneven problems, the fewest sweeps in one launch
    ([(24, 45), (16, 30)], 8, 3, (1, 1, 2)),               # too few: launches of their own
    ([(24, 48)], 12, 3, (2, 2, 16)),                       # 12, 6 and 3 cells
    ([(18, 36)], 6, 2, (2, 1, 8)),
    ([(24, 45)], 8, 2, (2, 0, 16)),                        # a larger coarsest level, no post-smoothing
])
def test_preconditioned_solve_follows_the_cpu_vcycle(sizes, block, nlevels, smoothing):
    sv = S.Solver(S.pfss_spec(sizes, block=block, nlevels=nlevels, device=0))
    sv.set_smoothing(*smoothing)
    rep = sv.solve(tol=1e-10, max_iter=400)
    assert rep["converged"] == 1 and (sv.problem_residuals() <= 1e-10).all()
    ops = [sv.operator(l) for l in range(sv.nlevels)]
    halos = [sv.halo_map(l) for l in range(sv.nlevels)]
    first = sv.problem_blocks()
    b = sv.rhs()
    bprob = np.repeat(np.arange(sv.nproblems), np.diff(first))
    x, it, rel = oracle.mg_solve(ops, halos, bprob, sv.nproblems, b, np.zeros_like(b), 1e-10, 400, smoothing)
    assert (rel <= 1e-10).all()
    print("iterations: gpu", rep["iterations"], "cpu", it)
    # FP32 V-cycles in FP64-corrected restarts: a restart loses a few iterations
    assert rep["iterations"] <= 1.3 * it + 5
    # both within 1e-10 of their right-hand sides; the operators' condition is below 1e4
    g = sv.solution()
    assert np.linalg.norm(g - x) <= 1e-6 * np.linalg.norm(x)


@pytest.mark.parametrize("precond", [S.PRECOND_NONE, S.PRECOND_MG])
def test_solve_without_and_with_the_vcycle_agree(precond):
    """The solver's FCG iteration in three kernels with either preconditioner."""
    sv = S.Solver(S.pfss_spec([(16, 30), (24, 45)], device=0))
    rep = sv.solve(tol=1e-9, max_iter=3000, precond=precond)
    assert rep["converged"] == 1 and (sv.problem_residuals() <= 1e-9).all()
