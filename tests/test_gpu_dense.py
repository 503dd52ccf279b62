"""Element matrices that the Legendre-mode kernels do not take: the dense DMMA and tensor-core kernels.

The elements are of one triclinic material, so every element matrix is the uniform one seen through its
element's B-spline basis (which the tensor-core form asks for), but shear and normal strains couple (which
the mode form excludes).  All results are compared with the oracle's element loop."""
import numpy as np
import pytest

import immersed_catmull_clark_b200 as icc
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def kron3(x, y, z):
    return np.kron(z, np.kron(y, x))


def triclinic_types(bounds, nel, sp):
    """(types, type_id): K[(i, a), (j, b)] = sum_pq C_ipjq int dN_a/dx_p dN_b/dx_q of the uniform B-splines, then
    R K R' per type, R the end elements' B-splines N_0 = 2 B_0, N_1 = B_1 - B_0 in terms of the uniform ones."""
    a = np.random.default_rng(3).standard_normal((6, 6))
    voigt = np.array([[0, 5, 4], [5, 1, 3], [4, 3, 2]])
    c = (np.eye(6) + a @ a.T / 6.0)[voigt][:, :, voigt]           # C[i, p, j, q]
    g, w = np.polynomial.legendre.leggauss(3)
    t, w = 0.5 * (g + 1.0), 0.5 * w
    b0 = np.array([0.5 * (1 - t) ** 2, 0.5 + t - t * t, 0.5 * t * t])
    b1 = np.array([t - 1.0, 1.0 - 2.0 * t, t])
    m = []                                                        # m[d][s][r] = int (d/dx)^s B_a (d/dx)^r B_b dx
    for d in range(3):
        h = (bounds[d][1] - bounds[d][0]) / nel[d]
        v = [b0, b1 / h]
        m.append([[h * np.einsum("aq,bq,q->ab", v[s], v[r], w) for r in range(2)] for s in range(2)])
    ku = np.zeros((3, 27, 3, 27))
    for p in range(3):
        for q in range(3):
            gpq = kron3(*(m[d][int(p == d)][int(q == d)] for d in range(3)))
            ku += np.einsum("ij,ab->iajb", c[:, p, :, q], gpq)
    ku = ku.reshape(81, 81)
    em = icc.elasticity_element_matrices(sp, 1.0, 1.0)
    tid = np.asarray(em.type_id)
    types = np.zeros((len(em.types), 81, 81))
    for k in range(len(types)):
        e = int(np.flatnonzero(tid == k)[0])
        pos = (e % nel[0], e // nel[0] % nel[1], e // (nel[0] * nel[1]))
        r = []
        for d in range(3):
            x = 2.0 if pos[d] == 0 else 1.0
            y = 2.0 if pos[d] == nel[d] - 1 else 1.0
            r.append(np.array([[x, 0.0, 0.0], [1.0 - x, 1.0, 1.0 - y], [0.0, 0.0, y]]))
        rr = np.kron(np.eye(3), kron3(*r))
        types[k] = rr @ ku @ rr.T
    return types, tid


def system(nel, mode, seed=0):
    bounds = ((0.0, 1.0 * nel[0]), (0.0, 0.9 * nel[1]), (0.0, 1.2 * nel[2]))
    sp, osp = icc.SpaceBox(bounds, nel, 2), O.Space(bounds, nel, 2)
    types, tid = triclinic_types(bounds, nel, sp)
    rng = np.random.default_rng(seed)
    s = rng.uniform(0.1, 1.0, sp.nel)
    fm = np.ones(sp.ndof, dtype=np.uint8)
    fm[np.arange(sp.ndof) % (nel[0] + 2) == 0] = 0                # clamped at the first control plane along x
    op = icc.MatrixFreeOperator(sp, icc.ElementMatrices(types, tid), s, None if mode == icc.MASK_NONE else fm, mode)

    def apply(x):
        y = O.mf_apply(osp, types, tid.astype(np.int64), s, x if mode == icc.MASK_NONE else fm * x,
                       np.ones(sp.ndof, dtype=np.uint8), icc.MASK_NONE)
        if mode == icc.MASK_ZERO:
            return fm * y
        return np.where(fm > 0, y, x) if mode == icc.MASK_IDENTITY else y

    return sp, op, fm, apply, rng


@pytest.mark.parametrize("precision", [icc.FP64, icc.MIXED])
@pytest.mark.parametrize("mode", [icc.MASK_ZERO, icc.MASK_IDENTITY])
@pytest.mark.parametrize("nel", [(1, 1, 1), (9, 5, 6), (24, 12, 10)])
def test_solve_twice_on_one_handle(nel, mode, precision):
    """The second solve replays the iterations that the first one captured.  The FP64 recurrence's residual drifts by
    about iterations x eps x |A||x|/|b| < 1e3 x 2e-16 x 1e4; the mixed solve stops on the true one."""
    tol = 1e-8
    sp, op, fm, apply, rng = system(nel, mode)
    b = rng.standard_normal(sp.ndof) * fm
    solver = icc.PcgSolver(5000, tol, precision=precision)
    x, its, res = solver.solve(sp.ndof, b, None, op)
    assert solver.status == icc.ICC_OK and res < tol
    assert np.linalg.norm(b - apply(x)) < 1.1 * tol * np.linalg.norm(b)
    assert op.last_solve_info().kernel_launches > 2 * its         # launches per iteration: not the mode kernel
    x2, its2, _ = solver.solve(sp.ndof, b, None, op)
    assert its2 == its and np.array_equal(x2, x)
    b2 = rng.standard_normal(sp.ndof) * fm                        # another load on the captured iterations
    x3, _, _ = solver.solve(sp.ndof, b2, None, op)
    assert np.linalg.norm(b2 - apply(x3)) < 1.1 * tol * np.linalg.norm(b2)


def extra_term(sp, rng):
    """Triplets of a symmetric, diagonally dominant sparse term."""
    i = rng.permutation(sp.ndof)[: sp.ndof // 8 * 2].reshape(2, -1)
    k = i.shape[1]
    return (np.concatenate([i[0], i[1], i[0], i[1]]), np.concatenate([i[1], i[0], i[0], i[1]]),
            np.concatenate([np.full(2 * k, -0.05), np.full(2 * k, 0.06)]))


@pytest.mark.parametrize("extra", [False, True])
@pytest.mark.parametrize("mode", [icc.MASK_NONE, icc.MASK_ZERO, icc.MASK_IDENTITY])
@pytest.mark.parametrize("nel", [(1, 1, 1), (8, 4, 4), (9, 5, 6), (33, 17, 9)])
def test_applies(nel, mode, extra):
    """Both precisions, at sizes around the bricks of 8x4x4 elements; the repository's parity bars."""
    sp, op, fm, apply, rng = system(nel, mode, seed=1)
    r = c = np.zeros(0, dtype=np.int64)
    v = np.zeros(0)
    if extra:
        r, c, v = extra_term(sp, rng)
        op.set_extra_triplets(r, c, v)
    w = v if mode == icc.MASK_NONE else v * fm[r] * fm[c]
    x = rng.standard_normal(sp.ndof)
    for a, y, tol in ((x, op.matvec(x), 1e-12), (x.astype(np.float32), op.matvec_f32(x.astype(np.float32)), 5e-6)):
        ref = apply(a.astype(np.float64))
        np.add.at(ref, r, w * a.astype(np.float64)[c])
        assert np.linalg.norm(y - ref) < tol * np.linalg.norm(ref)


@pytest.mark.parametrize("precision", [icc.FP64, icc.MIXED])
def test_solve_with_a_sparse_term(precision):
    tol = 1e-8
    sp, op, fm, apply, rng = system((17, 9, 10), icc.MASK_ZERO, seed=2)
    b = rng.standard_normal(sp.ndof) * fm
    solver = icc.PcgSolver(5000, tol, precision=precision)
    solver.solve(sp.ndof, b, None, op)            # the captured iterations are rebuilt when the term is set
    r, c, v = extra_term(sp, rng)
    op.set_extra_triplets(r, c, v)
    x, _, _ = solver.solve(sp.ndof, b, None, op)
    y = apply(x)
    np.add.at(y, r, v * fm[r] * fm[c] * x[c])
    assert solver.status == icc.ICC_OK and np.linalg.norm(b - y) < 1.1 * tol * np.linalg.norm(b)


def test_vector_step_timeout_then_recovery():
    """The grid barrier of the tensor-core form's vector step runs out of polls; the handle solves normally
    afterwards (its iterations were captured with the other limit)."""
    sp, op, fm, apply, rng = system((16, 8, 8), icc.MASK_ZERO, seed=4)
    b = rng.standard_normal(sp.ndof) * fm
    solver = icc.PcgSolver(5000, 1e-8, precision=icc.MIXED)
    op.set_wait_limit(0)   # no poll at all: every CTA that is not the last to arrive gives up
    with pytest.raises(icc.IccError) as ei:
        solver.solve(sp.ndof, b, None, op)
    assert ei.value.code == icc.ICC_TIMEOUT
    op.set_wait_limit(1 << 22)
    x, _, _ = solver.solve(sp.ndof, b, None, op)
    assert solver.status == icc.ICC_OK and np.linalg.norm(b - apply(x)) < 1.1e-8 * np.linalg.norm(b)


def test_batch_of_both_kinds_of_matrices():
    """Systems of the mode form in a batch with others: their elements differ in shape, which a batch refuses; each
    kind alone is solved."""
    sp, op, fm, apply, rng = system((9, 5, 6), icc.MASK_ZERO, seed=5)
    iso = icc.MatrixFreeOperator(sp, icc.elasticity_element_matrices(sp, 1.0, 1.0), None, fm, icc.MASK_ZERO)
    b = rng.standard_normal(sp.ndof) * fm
    with pytest.raises(icc.IccError) as ei:
        icc.solve_batched([op, iso], [b, b], tol=1e-8, precision=icc.MIXED)
    assert ei.value.code == icc.ICC_BAD_ARG
    sp2, op2, fm2, apply2, _ = system((24, 12, 10), icc.MASK_ZERO, seed=6)
    b2 = rng.standard_normal(sp2.ndof) * fm2
    xs, _, _, st = icc.solve_batched([op, op2], [b, b2], tol=1e-8, precision=icc.MIXED)
    assert np.all(st == icc.ICC_OK)
    for x, r, f in ((xs[0], b, apply), (xs[1], b2, apply2)):
        assert np.linalg.norm(r - f(x)) < 1.1e-8 * np.linalg.norm(r)
