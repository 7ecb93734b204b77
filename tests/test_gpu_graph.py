"""The device graph build at the edges of its hash table and incidence lists:
a star of tetrahedra that share one node and nothing else has 9 n + 1
neighbours of the centre, so 28 elements give 253 (the limit is 255) and 29
are rejected; node numbers far apart and element order reversed exercise the
ordering.  Patterns are compared with the oracle's Tpetra-semantics merge."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def F():
    import feddlib_gb300 as F
    return F


def star(n, seed):
    """n P2 tetrahedra around one common vertex, shuffled node numbers (the
    elements may overlap in space: only their connectivity matters here)."""
    rng = np.random.default_rng(seed)
    new = rng.permutation(9 * n + 1).astype(np.int32)
    xyz = np.zeros((9 * n + 1, 3))
    el = np.zeros((n, 10), dtype=np.int32)
    for e in range(n):
        B = np.eye(3) + 0.1 * rng.standard_normal((3, 3))
        v = np.vstack([np.zeros(3), B.T])
        edges = [(0, 1), (1, 2), (0, 2), (0, 3), (1, 3), (2, 3)]
        pts = np.vstack([v, [0.5 * (v[a] + v[b]) for a, b in edges]])
        ids = np.concatenate([[0], 9 * e + 1 + np.arange(9)])
        xyz[new[ids]] = pts
        el[e] = new[ids]
    return xyz, np.ascontiguousarray(el[::-1])


@pytest.mark.parametrize("n", [1, 3, 4, 7, 12, 13, 25, 26, 28])
def test_star_patterns(F, n):
    xyz, el = star(n, n)
    a = F.Assembler(F.LAPLACE, xyz, el, fe_order=2)
    rp, ci, _ = a.pattern(0)
    orp, oci, ov = O.assemble_laplace(2, 5, xyz, el)
    np.testing.assert_array_equal(rp, orp)
    np.testing.assert_array_equal(ci, oci)
    (v,), _, _ = a.assemble(residual=False)
    # FP64 sums of at most 28 contributions in another order than the oracle's
    assert np.linalg.norm(v - ov) <= 1e-13 * np.linalg.norm(ov)
    b = F.Assembler(F.LINEAR_ELASTICITY, xyz, el)
    rp3, ci3, _ = b.pattern(0)
    for d in range(3):
        np.testing.assert_array_equal(np.diff(rp3)[d::3], 3 * np.diff(orp))
    np.testing.assert_array_equal(ci3[::3][:1], 3 * oci[:1])


def test_star_beyond_the_neighbour_limit_is_rejected(F):
    xyz, el = star(29, 0)
    with pytest.raises(F.FeddError) as err:
        F.Assembler(F.LAPLACE, xyz, el, fe_order=2)
    assert "CAPACITY" in str(err.value).upper()
