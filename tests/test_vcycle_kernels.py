"""The V-cycle's launches value by value: the residual restricted in one pass, the first
sweep from z = 0, the prolongation with a black half sweep and the coarsest level's sweeps,
each as a V-cycle runs it, against the oracle's FP32 operations with FP64 halos.

A half sweep divides a sum of seven products by the diagonal, whose row sum bounds the
off-diagonal ones: some ten roundings of 2^-24 of the largest |z| a half sweep, and errors
do not grow. The ghosts' snapped weights add one."""
import numpy as np
import pytest

import oracle
from falcon_gb300 import solver as S

pytestmark = pytest.mark.gpu
ROUNDINGS = 11 * 2.0 ** -24

SPECS = {
    "m8": dict(sizes=[(24, 45), (16, 30)]),                    # 8, 4, 2 cells
    "m16": dict(sizes=[(32, 60)], block=16, nlevels=4),        # 16, 8, 4, 2
    "m32": dict(sizes=[(32, 64)], block=32, nlevels=5),
    "m12": dict(sizes=[(24, 48)], block=12, nlevels=3),        # 12, 6, 3: a thread per cell
    "m10": dict(sizes=[(40, 80)], block=10, nlevels=2),        # 10 by pairs, 5
    "m24": dict(sizes=[(48, 96)], block=24, nlevels=4),        # 24 by pairs, 12, 6, 3
}


class Level:
    """A level's operator and halo on the CPU."""

    def __init__(self, sv, level):
        self.A = sv.operator(level)
        self.idx, self.wx = sv.halo_map(level)
        self.shape = (sv.nblocks,) + sv.level_shape(level)[::-1]
        self.m = self.shape[1]

    def padded(self, z):
        zp = np.zeros((self.shape[0],) + (self.m + 2,) * 3)
        zp[:, 1:-1, 1:-1, 1:-1] = z
        return oracle.halo_fill(self.m, self.idx, self.wx, zp)

    def half_sweep(self, r, z, colour):
        return oracle.mg_rbgs(self.A, r, self.padded(z).astype(np.float32), colour)[:, 1:-1, 1:-1, 1:-1]

    def residual(self, r, z):
        return r.astype(np.float64) - oracle.spmv(self.m, self.A, self.padded(z))


@pytest.mark.parametrize("spec", sorted(SPECS))
def test_residual_restricted_first_and_prolonged_sweeps(built_lib, oracle_lib, spec):
    sv = S.Solver(S.pfss_spec(device=0, **SPECS[spec]))
    rng = np.random.default_rng(71)
    f32 = lambda shape: rng.normal(size=shape).astype(np.float32)
    for level in range(sv.nlevels):
        L = Level(sv, level)
        A = [np.abs(a).max() for a in L.A]
        z = f32(L.shape)
        r = (f32(L.shape) * A[0]).astype(np.float32)
        # first sweep: red from zero, then black
        first = sv.vcycle_op(S.VCYCLE_FIRST_SWEEP, level, r)
        ref = L.half_sweep(r, L.half_sweep(r, np.zeros(L.shape), 0), 1)
        assert np.abs(first - ref).max() <= 2 * ROUNDINGS * np.abs(ref).max(), level
        if level + 1 == sv.nlevels:
            continue
        C = Level(sv, level + 1)
        # eight residuals, each a sum of eight terms below |r| + 7 max|A| max|z| of its cell
        ref = L.residual(r, z).reshape(L.shape[0], C.m, 2, C.m, 2, C.m, 2).sum(axis=(2, 4, 6))
        bound = 8 * ROUNDINGS * (np.abs(r).max() + sum(A) * 2 * np.abs(z).max())
        assert np.abs(sv.vcycle_op(S.VCYCLE_RESIDUAL_RESTRICT, level, r, z) - ref).max() <= bound, level
        zc = f32(C.shape)
        swept = sv.vcycle_op(S.VCYCLE_PROLONG_SWEEP, level, zc, np.stack([r, z]))
        ref = L.half_sweep(r, oracle.mg_prolong_add(zc, z), 1)
        assert np.abs(swept - ref).max() <= ROUNDINGS * np.abs(ref).max(), level
    sv.close()


@pytest.mark.parametrize("spec,ctas,cells", [
    (dict(sizes=[(16, 30)]), 1, 1),
    (dict(sizes=[(24, 45)]), 1, 2),
    (dict(sizes=[(32, 60)]), 4, 1),
    (dict(sizes=[(24, 45), (16, 30), (33, 60)]), 4, 1),      # problems of uneven size
    (dict(sizes=[(64, 120)]), 16, 2),
    (dict(sizes=[(64, 180)]), 16, 4),
    (dict(sizes=[(24, 45)], nlevels=2), 16, 1),              # four cells a block
    (dict(sizes=[(24, 48)], block=12), 0, 0),                # three: a launch per half sweep
])
@pytest.mark.parametrize("sweeps", [1, 2, 3, 16])
def test_coarsest_sweeps_in_their_forms(built_lib, oracle_lib, spec, ctas, cells, sweeps):
    """Up to two sweeps are launches of their own, more are one launch of a CTA or a cluster
    per problem where the problem fits."""
    sv = S.Solver(S.pfss_spec(device=0, **spec))
    form = sv.coarse_form()
    assert (form["ctas"] > 1, form["cells"]) == (ctas > 1, cells)
    assert (form["ctas"] == 0) == (ctas == 0)
    sv.set_smoothing(2, 2, sweeps)
    level = sv.nlevels - 1
    L = Level(sv, level)
    rng = np.random.default_rng(72)
    r = (rng.normal(size=L.shape) * np.abs(L.A[0]).max()).astype(np.float32)
    z = np.zeros(L.shape)
    for half in range(2 * sweeps):
        z = L.half_sweep(r, z, half & 1)
    g = sv.vcycle_op(S.VCYCLE_COARSE_SWEEPS, level, r)
    err = np.abs(g - z).max() / np.abs(z).max()
    print(form, "sweeps", sweeps, "largest difference %.2e of %.2e" % (err, 2 * sweeps * ROUNDINGS))
    assert err <= 2 * sweeps * ROUNDINGS
    sv.close()


def test_solves_with_and_without_the_vcycle_have_one_solution(built_lib):
    """The same right-hand side with either preconditioner; both residuals are at most
    1e-11 of it and the operators' condition is below 1e5."""
    sv = S.Solver(S.pfss_spec([(24, 45)], device=0))
    x = []
    for precond in (S.PRECOND_NONE, S.PRECOND_MG):
        assert sv.solve(tol=1e-11, max_iter=4000, precond=precond)["converged"] == 1
        assert (sv.problem_residuals() <= 1e-11).all()
        x.append(sv.solution())
    assert np.linalg.norm(x[0] - x[1]) <= 2e-6 * np.linalg.norm(x[1])
    sv.close()
