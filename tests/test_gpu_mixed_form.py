"""The form a mixed solve of isotropic elements runs in: the Legendre-mode kernel, or the tensor cores on grids that
its tiles fill badly."""
import numpy as np
import pytest

import immersed_catmull_clark_b200 as icc
from immersed_catmull_clark_b200 import workloads as W
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def cantilever(nel, seed=3):
    p = W.cantilever(nel, seed=seed)
    sp, osp = icc.SpaceBox(p.bounds, p.nel, 2), O.Space(p.bounds, p.nel, 2)
    em = icc.elasticity_element_matrices(sp, *icc.lame(1.0, 0.3))
    op = icc.MatrixFreeOperator(sp, em, p.scale, p.free_mask, icc.MASK_ZERO)
    b = W.rhs_masked(p)

    def residual(x):
        y = O.mf_apply(osp, em.types, em.type_id.astype(np.int64), p.scale, x, p.free_mask, icc.MASK_ZERO)
        return np.linalg.norm(b - y) / np.linalg.norm(b)

    return sp, op, b, residual


@pytest.mark.parametrize("nel,modes", [((33, 52, 49), False), ((65, 65, 65), False), ((132, 66, 66), False),
                                       ((24, 16, 12), True), ((53, 31, 27), True), ((93, 54, 47), True),
                                       ((128, 64, 64), True), ((1000, 17, 17), True)])
def test_single_solves_take_the_sooner_form(nel, modes):
    """Both forms were measured on these grids; the tensor-core form launches two kernels an iteration.  The solve stops
    on the true residual, which the oracle confirms to rounding."""
    tol = 1e-6
    sp, op, b, residual = cantilever(nel)
    solver = icc.PcgSolver(20000, tol, precision=icc.MIXED)
    x, its, _ = solver.solve(sp.ndof, b, None, op)
    assert solver.status == icc.ICC_OK and residual(x) < 1.1 * tol
    assert (op.last_solve_info().kernel_launches < its) == modes
    x2, its2, _ = solver.solve(sp.ndof, b, None, op)
    assert its2 == its and np.array_equal(x2, x)


@pytest.mark.parametrize("sizes", [[(104, 52, 52), (104, 52, 52)], [(65, 65, 65)],
                                   [(120, 60, 60), (104, 52, 52), (16, 8, 8)]])
def test_batches_on_either_side(sizes):
    """Systems above the size from which they may be solved by themselves, some of them sooner together."""
    tol = 1e-6
    inst = [cantilever(nel, seed=i) for i, nel in enumerate(sizes)]
    xs, _, _, st = icc.solve_batched([i[1] for i in inst], [i[2] for i in inst], tol=tol, precision=icc.MIXED)
    assert np.all(st == icc.ICC_OK)
    for x, (_, _, _, residual) in zip(xs, inst):
        assert residual(x) < 1.1 * tol
