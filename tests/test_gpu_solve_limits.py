"""Limits of a solve's launches: the bounded grid barrier, the iteration budget, the length of one launch, device
memory."""
import numpy as np
import pytest
import torch

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


@pytest.mark.parametrize("precision,nel,check", [(icc.FP64, (128, 64, 64), 32), (icc.FP64, (96, 96, 96), 32),
                                                 (icc.FP64, (128, 64, 64), 1000), (icc.MIXED, (96, 96, 96), 1000)])
def test_a_launch_holds_the_chip_for_milliseconds(precision, nel, check):
    """One launch takes every SM, so work on other streams waits for it: launches are cut at about 8 ms (FP64) or 16 ms
    whatever the grid and the check interval.  Half as much again is allowed for the model of an iteration's time."""
    p, sp, op = cantilever(nel)
    solver = icc.PcgSolver(1000, 1e-30, precision=precision, check_every=check, inner_tol=1e-30)
    solver.solve(sp.ndof, W.rhs_masked(p), None, op)
    info = op.last_solve_info()
    assert info.iterations == 1000
    assert info.device_ms / info.kernel_launches < (12.0 if precision == icc.FP64 else 24.0)


def test_launch_cuts_do_not_change_the_solve():
    """The iterations are the same whatever the launches they run in."""
    p, sp, op = cantilever((53, 31, 27))
    b = W.rhs_masked(p)
    for precision in (icc.FP64, icc.MIXED):
        ref = None
        for check in (16, 32, 1 << 30):   # the replacements of the mixed form fall on multiples of the interval
            if precision == icc.MIXED and check != 32:
                continue
            x, its, res = icc.PcgSolver(3000, 1e-8, precision=precision, check_every=check).solve(sp.ndof, b, None, op)
            ref = (x, its, res) if ref is None else ref
            assert its == ref[1] and res == ref[2] and np.array_equal(x, ref[0])


def test_batch_memory():
    """Systems of a batch that run on the tensor-core kernels hold no vectors of the other form."""
    nel = (76, 56, 56)     # below the size from which a system is solved on its own
    for k in range(2):     # the first batch also loads the kernels
        inst = [cantilever(nel, seed=2 * k + i) for i in range(2)]
        sp, ops, bs = inst[0][1], [i[2] for i in inst], [W.rhs_masked(i[0]) for i in inst]
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        icc.solve_batched(ops, bs, tol=1e-3, max_iter=64, precision=icc.MIXED)
        used = free - torch.cuda.mem_get_info()[0]
    n, bricks = sp.ndof, -(-nel[0] // 8) * -(-nel[1] // 4) * -(-nel[2] // 4)
    padded = 3 * ((nel[0] + 2 + 3) // 4 * 4) * (nel[1] + 2) * (nel[2] + 2)
    # FP64: x, r, p, Ap, D^-1, b, diagonal; x, r, y of the mixed form; FP32: load, x, r, p, Ap, D^-1, padded input, brick
    # partial sums, scale.  Allocations are rounded up to 2 MB; the small ones of a handle share two such blocks.
    sizes = [8 * n] * 10 + [4 * n] * 6 + [4 * padded, 4 * bricks * 3 * 360, 4 * sp.nel]
    assert used <= 2 * sum(-(-s // (2 << 20)) for s in sizes) * (2 << 20) + 2 * (4 << 20)
