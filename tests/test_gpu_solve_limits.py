"""Limits of a solve's launches: the bounded grid barrier."""
import numpy as np
import pytest

import immersed_catmull_clark_b200 as icc
from immersed_catmull_clark_b200 import workloads as W

pytestmark = pytest.mark.gpu


def cantilever(nel, seed=21):
    p = W.cantilever(nel, seed=seed)
    sp = icc.SpaceBox(p.bounds, p.nel, 2)
    em = icc.elasticity_element_matrices(sp, *icc.lame(1.0, 0.3))
    return p, sp, icc.MatrixFreeOperator(sp, em, p.scale, p.free_mask, icc.MASK_ZERO)


def test_fp64_grid_barrier_timeout_then_recovery():
    """set_wait_limit bounds the barrier of the FP64 solve as well; the handle solves normally after a time-out."""
    p, sp, op = cantilever((16, 8, 8))
    b = W.rhs_masked(p)
    solver = icc.PcgSolver(20 * sp.ndof, 1e-8, precision=icc.FP64)
    x, its, _ = solver.solve(sp.ndof, b, None, op)
    op.set_wait_limit(0)   # no poll at all: every CTA that is not the last to arrive gives up
    with pytest.raises(icc.IccError) as ei:
        solver.solve(sp.ndof, b, None, op)
    assert ei.value.code == icc.ICC_TIMEOUT
    op.set_wait_limit(1 << 22)
    x2, its2, _ = solver.solve(sp.ndof, b, None, op)
    assert solver.status == icc.ICC_OK and its2 == its and np.array_equal(x2, x)


@pytest.mark.parametrize("check", [1, 4, 16, 32])
def test_iteration_budget_of_a_mixed_solve(check):
    """A mixed solve that leaves its launches early, at residual replacements, still has its whole iteration budget:
    it ends as not converged with every iteration spent, not as a time-out."""
    p, sp, op = cantilever((53, 31, 27))
    solver = icc.PcgSolver(1000, 1e-30, precision=icc.MIXED, check_every=check)
    x, its, res = solver.solve(sp.ndof, W.rhs_masked(p), None, op)
    assert solver.status == icc.ICC_NOT_CONVERGED and its == 1000
