"""Solves on several handles at the same time, one host thread each: persistent kernels of several systems share the
chip, and every result is bitwise that of the same solve by itself."""
import threading

import numpy as np
import pytest

import immersed_catmull_clark_b200 as icc
from immersed_catmull_clark_b200 import workloads as W

pytestmark = pytest.mark.gpu


def cantilever(nel, seed):
    p = W.cantilever(nel, seed=seed)
    sp = icc.SpaceBox(p.bounds, p.nel, 2)
    em = icc.elasticity_element_matrices(sp, *icc.lame(1.0, 0.3))
    return sp, icc.MatrixFreeOperator(sp, em, p.scale, p.free_mask, icc.MASK_ZERO), W.rhs_masked(p)


@pytest.mark.parametrize("precision", [icc.FP64, icc.MIXED])
# cubes, one a CTA (several systems on an SM); cubes, two a CTA; marches; all of them, and one on the tensor cores
@pytest.mark.parametrize("sizes", [[(24, 16, 12)] * 6, [(33, 16, 17)] * 4, [(53, 31, 27)] * 3,
                                   [(8, 8, 8), (24, 16, 12), (40, 20, 20), (64, 33, 40), (33, 52, 49), (30, 15, 15)]])
def test_concurrent_solves_equal_single_ones(sizes, precision):
    tol = 1e-7
    systems = [cantilever(nel, i) for i, nel in enumerate(sizes)]

    def solve(s):
        return icc.PcgSolver(20000, tol, precision=precision).solve(s[0].ndof, s[2], None, s[1])

    single = [solve(s) for s in systems]
    out = [None] * len(systems)

    def work(i):
        for _ in range(3):
            out[i] = solve(systems[i])

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(systems))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, b in zip(single, out):
        assert b is not None and a[1] == b[1] and a[2] == b[2] and np.array_equal(a[0], b[0])


@pytest.mark.parametrize("precision", [icc.FP64, icc.MIXED])
def test_applies_beside_a_solve(precision):
    """Plain applies, whose marches take tensor memory as the solve's do, while another handle's solve runs."""
    a, b, c = cantilever((64, 33, 40), 1), cantilever((70, 40, 30), 2), cantilever((33, 52, 49), 3)
    x = [np.random.default_rng(i).standard_normal(s[0].ndof) for i, s in enumerate((b, c))]
    ref = [(s[1].matvec(v), s[1].matvec_f32(v.astype(np.float32))) for s, v in zip((b, c), x)]
    one = icc.PcgSolver(20000, 1e-7, precision=precision).solve(a[0].ndof, a[2], None, a[1])
    out, done = [], threading.Event()

    def solve():
        for _ in range(3):
            out.append(icc.PcgSolver(20000, 1e-7, precision=precision).solve(a[0].ndof, a[2], None, a[1]))
        done.set()

    t = threading.Thread(target=solve)
    t.start()
    same, n = True, 0
    while not done.is_set() or n == 0:
        for s, v, r in zip((b, c), x, ref):
            same = same and np.array_equal(s[1].matvec(v), r[0]) and np.array_equal(s[1].matvec_f32(v.astype(np.float32)), r[1])
        n += 1
    t.join()
    assert same and len(out) == 3
    for o in out:
        assert o[1] == one[1] and np.array_equal(o[0], one[0])
