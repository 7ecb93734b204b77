"""Element matrices of the Laplace operator on stretched tetrahedra, entry by
entry.  A vertex far from the opposite face has a small gradient that is the
difference of large ones, and small entries in its row.

Bound: with edges of at most L and a base of about 1, the cofactors' entries
are differences of two products of size L, wrong by at most 4 eps L, and the
sum of three of them by 16 eps L, of a gradient times volume that is at least
1/2.  An entry (a, b) is a product of two such gradients, so it is within
64 eps L of the geometric mean of the diagonal entries a and b; the P2 entries
are combinations of at most four of these, with weights up to 8 / 5."""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52
EDGES = ((0, 1), (1, 2), (0, 2), (0, 3), (1, 3), (2, 3))


def stretched(L, n, seed):
    """n separate tetrahedra, vertex e % 4 of element e at height L over the others."""
    rng = np.random.default_rng(seed)
    xyz = np.empty((n, 4, 3))
    base = np.array([[0.0, 0.0, 0.0], [1.0, 0.1, 0.0], [0.2, 1.0, 0.1]])
    for e in range(n):
        far = e % 4
        xyz[e, [k for k in range(4) if k != far]] = base + 0.1 * rng.standard_normal((3, 3))
        xyz[e, far] = [0.3, 0.4, L] + 0.1 * rng.standard_normal(3)
    return xyz


def exact_d(x):
    """V grad L_i . grad L_j in exact arithmetic."""
    X = [[Fraction(float(v)) for v in r] for r in x]
    d = [[X[j][k] - X[0][k] for k in range(3)] for j in (1, 2, 3)]
    cross = lambda a, b: [a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]]
    C = [None, cross(d[1], d[2]), cross(d[2], d[0]), cross(d[0], d[1])]
    C[0] = [-(C[1][k] + C[2][k] + C[3][k]) for k in range(3)]
    det = abs(sum(d[0][k] * C[1][k] for k in range(3)))
    return [[sum(C[i][k] * C[j][k] for k in range(3)) / (6 * det) for j in range(4)] for i in range(4)]


def exact_p2(D):
    """int lambda_i lambda_j = V (1 + d_ij) / 20 with phi_i = l_i (2 l_i - 1), phi_ij = 4 l_i l_j."""
    # gradient of a P2 function: sum of (coefficient, barycentric factor or None, gradient index)
    def grad(a):
        if a < 4:
            return [(4, a, a), (-1, None, a)]
        i, j = EDGES[a - 4]
        return [(4, i, j), (4, j, i)]

    def mean(p, q):  # mean over the element of the product of two factors
        if p is None and q is None:
            return Fraction(1)
        if p is None or q is None:
            return Fraction(1, 4)
        return Fraction(2 if p == q else 1, 20)

    return [[sum(c * f * mean(p, q) * D[i][j] for c, p, i in grad(a) for f, q, j in grad(b)) for b in range(10)]
            for a in range(10)]


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("L", [1, 10, 1000])
def test_entries(order, L):
    import feddlib_gb300 as F
    n = 24
    v = stretched(L, n, 7 + L)
    xyz, npe = v, 4
    if order == 2:
        xyz = np.concatenate([v, np.stack([(v[:, a] + v[:, b]) / 2 for a, b in EDGES], axis=1)], axis=1)
        npe = 10
    el = np.arange(n * npe, dtype=np.int32).reshape(n, npe)
    a = F.Assembler(F.LAPLACE, np.ascontiguousarray(xyz.reshape(-1, 3)), el, fe_order=order)
    K, _ = a.element_matrices()
    (vals,), _, _ = a.assemble()  # separate elements: the rows are the elements' rows
    assert np.array_equal(vals.reshape(n, npe, npe), K)
    # D's geometric means that enter an entry, for the bound
    for e in range(n):
        D = exact_d(v[e])
        ex = D if order == 1 else exact_p2(D)
        d = [float(D[i][i]) ** 0.5 for i in range(4)]
        of = [(i,) for i in range(4)] + list(EDGES)
        for i in range(npe):
            for j in range(npe):
                size = max(d[p] * d[q] for p in of[i] for q in of[j])
                bound = (1.0 if order == 1 else 8.0) * 64 * EPS * L * size
                assert abs(float(Fraction(float(K[e, i, j])) - ex[i][j])) <= bound, (e, i, j)
