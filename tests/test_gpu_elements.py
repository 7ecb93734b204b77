"""The hyperelastic element stage takes a warp's elements two at a time, in
batches whose size follows the mesh: odd and single elements, the ends of
batches, every law, with and without displacements, four and five points.

Bounds as for the other element matrices (FP32 integrals against FP64): 2e-6 of
the matrix, 1e-5 of the residual, whose stresses cancel."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def F():
    import feddlib_gb300 as F
    return F


def rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


E, NU = 32.0 / 11.0, 5.0 / 11.0
LAWS = {
    "LINEAR_ELASTICITY": (O.law_from_E_nu(O.LAW_SKR1, E, NU), 4, {}),
    "NONLINEAR_ELASTICITY": (O.law_from_E_nu(O.LAW_SKR2, E, NU), 5, {}),
    "NONLINEAR_ELASTICITY2": (O.law_from_E_nu(O.LAW_SKR3, E, NU), 5, {}),
    "ANISO_FIBER": (O.LawSpec(O.LAW_ANISO, mu=1.0, lam=10.0, k1=2.0, k2=1.0, angle_deg=40.0), 4,
                    dict(k1=2.0, k2=1.0, fiber_angle_deg=40.0)),
}


@pytest.mark.parametrize("problem", list(LAWS))
@pytest.mark.parametrize("M,n,field", [(1, 1, True), (1, 2, True), (1, 3, True), (2, 33, False), (11, 7985, True)])
def test_elements_of_every_batch(F, problem, M, n, field):
    law, npts, extra = LAWS[problem]
    field = field or problem != "LINEAR_ELASTICITY"  # the other laws want displacements
    xyz, el = F.structured_mesh(M, 2, seed=50 + M)
    el = np.ascontiguousarray(el[:n])
    u = F.fourier_field(xyz, seed=50, kmin=1, kmax=2, scale=0.004) if field else None
    a = F.Assembler(getattr(F, problem), xyz, el, E=E, poisson_ratio=NU, **extra)
    K, r = a.element_matrices(u=u)
    zero = np.zeros(30)
    for e in sorted({0, 1, 2, 31, 32, 63, n // 2, n - 3, n - 2, n - 1} & set(range(n))):
        Ko, ro = O.elem_hyper(law, npts, xyz[el[e]], u.reshape(-1, 3)[el[e]].ravel() if field else zero)
        assert rel(K[e], Ko) < 2e-6, e
        if field:
            assert rel(r[e], ro) < 1e-5, e
    # each element is computed for itself: the ends of a shorter list are the same bits
    if n > 3:
        b = F.Assembler(getattr(F, problem), xyz, np.ascontiguousarray(el[1:n // 2]), E=E, poisson_ratio=NU, **extra)
        Kb, rb = b.element_matrices(u=u)
        assert np.array_equal(Kb, K[1:n // 2]) and np.array_equal(rb, r[1:n // 2])


@pytest.mark.parametrize("M,n,newton", [(1, 1, True), (1, 5, False), (8, 3071, True), (8, 3071, False)])
def test_generalized_newtonian_elements_of_every_batch(F, M, n, newton):
    """The viscous element stage works in batches that follow the mesh too."""
    xyz2, el2 = F.structured_mesh(M, 2, seed=60 + M)
    xyz1, el1 = F.structured_mesh(M, 1, seed=60 + M)
    el2, el1 = np.ascontiguousarray(el2[:n]), np.ascontiguousarray(el1[:n])
    u, p = 0.5 * F.fourier_field(xyz2, seed=60), F.uniform_field(60, xyz1.shape[0])
    prm = [1.902, 0.22, 0.056, 0.00345, 1.25]
    L = O.visc_law(0, prm, 1e-12)

    def matrices(lo, hi):
        a = F.Assembler(F.NAVIER_STOKES, xyz2, el2[lo:hi], elements_p=el1[lo:hi], num_nodes_p=xyz1.shape[0],
                        viscosity=0.01, density=1.0, newton=newton)
        a.set_viscosity_law(0, prm, gamma_min=1e-12)
        return a.element_matrices(u=u, p=p)

    K, r = matrices(0, n)
    for e in sorted({0, 1, 2, 3, n // 2, n - 2, n - 1} & set(range(n))):
        Jo, ro = O.elem_gn(xyz2[el2[e]], u.reshape(-1, 3)[el2[e]].ravel(), p[el1[e]], L, 1.0, newton)
        assert rel(K[e], Jo) < 2e-6 and rel(r[e], ro) < 2e-6, e
    if n > 2:
        Kb, rb = matrices(1, n // 2)
        assert np.array_equal(Kb, K[1:n // 2]) and np.array_equal(rb, r[1:n // 2])
