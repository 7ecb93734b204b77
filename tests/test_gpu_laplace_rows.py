"""Rows of the scalar Laplace matrix: several nodes share a warp (six P1 or two
P2 nodes), four incidences are read at a time, and a call that wants the load
alone has a kernel of its own.  Node counts around a warp's and a block's share,
few and many incidences per node, nodes no element refers to.

Tolerance: FP64 throughout; an entry is a sum of at most a few hundred terms of
one sign pattern, so its rounding error is below 1e-13 of the largest entry.
The bound is 1e-12, as for the other Laplace comparisons."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu
TOL = 1e-12


@pytest.fixture(scope="module")
def F():
    import feddlib_gb300 as F
    return F


def fan(n, order, extra, seed):
    """n tetrahedra around one vertex (plus `extra` unreferenced nodes), the
    nodes' numbers permuted."""
    rng = np.random.default_rng(seed)
    el = np.array([[0, 1 + 3 * e, 2 + 3 * e, 3 + 3 * e] for e in range(n)], np.int64)
    nn = 1 + 3 * n
    xyz = np.zeros((nn, 3))
    base = np.array([[1.0, 0.1, 0.0], [0.0, 1.0, 0.2], [0.3, 0.0, 1.0]])
    for e in range(n):
        xyz[1 + 3 * e:4 + 3 * e] = base + 0.1 * rng.standard_normal((3, 3))
    if order == 2:
        pairs = [(0, 1), (1, 2), (0, 2), (0, 3), (1, 3), (2, 3)]
        mid = [(xyz[el[e, a]] + xyz[el[e, b]]) / 2 for e in range(n) for a, b in pairs]
        el = np.hstack([el, nn + np.arange(6 * n).reshape(n, 6)])
        xyz = np.vstack([xyz, mid])
    xyz = np.vstack([xyz, rng.standard_normal((extra, 3))])
    perm = rng.permutation(len(xyz))
    out = np.empty_like(xyz)
    out[perm] = xyz
    return out, perm[el].astype(np.int32)


@pytest.mark.parametrize("order,n,extra", [(1, 1, 0), (1, 1, 2), (1, 2, 0), (1, 7, 1), (1, 8, 25), (1, 63, 3), (1, 64, 0),
                                           (2, 1, 0), (2, 1, 7), (2, 3, 2), (2, 4, 0), (2, 28, 5)])
def test_laplace_rows_and_load(F, order, n, extra):
    xyz, el = fan(n, order, extra, 100 * order + n)
    rule = 1 if order == 1 else 5
    orp, oci, ov = O.assemble_laplace(order, rule, xyz, el)
    ob = O.assemble_rhs(order, rule, xyz, el, 1.5)
    asm = F.Assembler(F.LAPLACE, xyz, el, fe_order=order, source=1.5)
    (v,), b, _ = asm.assemble()
    v, b = v.copy(), b.copy()
    rp, ci, _ = asm.pattern(0)
    np.testing.assert_array_equal(rp, orp)
    np.testing.assert_array_equal(ci, oci)
    assert np.abs(v - ov).max() <= TOL * np.abs(ov).max()
    assert np.abs(b - ob).max() <= TOL * np.abs(ob).max()
    assert (b[np.setdiff1d(np.arange(len(xyz)), el)] == 0.0).all()
    (v1,), _, _ = asm.assemble(residual=False)
    assert np.array_equal(v1, v)
    _, b1, _ = asm.assemble(jacobian=False)
    assert np.array_equal(b1, b)
