"""Which element matrices the Legendre-mode kernels may stand for.

A handle's operator is the one of the matrices given, to the FP64 parity bar of the repository.  Matrices
that are nearly of the mode form must not be replaced by ones that differ by more than that."""
import numpy as np
import pytest

import immersed_catmull_clark_b200 as icc
from oracle import oracle as O

pytestmark = pytest.mark.gpu

APPLY_TOL = 1e-12   # FP64 parity bar of the repository


def near_modal(nel, eps, seed=5):
    """Isotropic element matrices of unit cubes plus symmetric noise of eps times the largest entry of the interior one."""
    bounds = tuple((0.0, float(n)) for n in nel)
    sp, osp = icc.SpaceBox(bounds, nel, 2), O.Space(bounds, nel, 2)
    em = icc.elasticity_element_matrices(sp, *icc.lame(1.0, 0.3))
    cube = icc.SpaceBox(((0.0, 3.0),) * 3, (3, 3, 3), 2)
    mid = icc.elasticity_element_matrices(cube, *icc.lame(1.0, 0.3))
    kmax = np.abs(mid.types[mid.type_id[13]]).max()
    d = np.random.default_rng(seed).uniform(-1.0, 1.0, em.types.shape)
    types = em.types + eps * kmax * np.tril(d) + eps * kmax * np.tril(d, -1).transpose(0, 2, 1)
    return sp, osp, types, em.type_id


# Noise within rounding of long grids' own matrices (2e-16 n) and of end elements' stretched ones, where an
# acceptance by the largest entry lets through several parity bars; a single DOF sees its own column only.
@pytest.mark.parametrize("nel,eps", [((4000, 1, 1), 2e-12), ((2000, 2, 3), 5e-13), ((2, 2, 2), 5e-13), ((1, 1, 1), 1e-12)])
def test_nearly_modal_matrices_are_applied_as_given(nel, eps):
    sp, osp, types, tid = near_modal(nel, eps)
    op = icc.MatrixFreeOperator(sp, icc.ElementMatrices(types, tid))
    rng = np.random.default_rng(1)
    xs = [rng.standard_normal(sp.ndof)]
    for i in rng.integers(0, sp.ndof, 3):
        xs.append((np.arange(sp.ndof) == i).astype(float))
    for x in xs:
        y = O.mf_apply(osp, types, tid.astype(np.int64), np.ones(sp.nel), x, np.ones(sp.ndof, dtype=np.uint8), icc.MASK_NONE)
        assert np.linalg.norm(op.matvec(x) - y) < APPLY_TOL * np.linalg.norm(y)


@pytest.mark.parametrize("nel", [(1, 1, 1), (2, 9, 3), (256, 3, 2), (1500, 2, 2), (6000, 1, 2)])
def test_isotropic_matrices_of_long_grids(nel):
    """The knots i/n round, so a long grid's own matrices are 1e-16 n from the mode form: either path is exact
    to the bar."""
    sp, osp, types, tid = near_modal(nel, 0.0)
    op = icc.MatrixFreeOperator(sp, icc.ElementMatrices(types, tid))
    x = np.random.default_rng(2).standard_normal(sp.ndof)
    y = O.mf_apply(osp, types, tid.astype(np.int64), np.ones(sp.nel), x, np.ones(sp.ndof, dtype=np.uint8), icc.MASK_NONE)
    assert np.linalg.norm(op.matvec(x) - y) < APPLY_TOL * np.linalg.norm(y)
