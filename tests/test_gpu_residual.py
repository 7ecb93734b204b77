"""The residual alone (no Jacobian) takes kernels of its own, with the same
operations in the same order as the call that assembles both: its values are
compared bit for bit with that call's, and with the oracle at the parity
tests' bounds."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOL_NS, TOL_HYPER = 1e-6, 1e-5
LAWS = [(0, [1.902, 0.22, 0.056, 0.00345, 1.25]), (1, [0.017, 0.708, 0.056, 0.00345]),
        (2, [1.902, 0.22, 1.0, 0.0616, 0.056])]


@pytest.fixture(scope="module")
def F():
    import feddlib_gb300 as F
    return F


def rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def same(a, b):
    return np.array_equal(a.view(np.uint64), b.view(np.uint64))


def ns(F, M, seed, shuffle=False, swap=False, **kw):
    xyz2, el2 = F.structured_mesh(M, 2, seed=seed)
    xyz1, el1 = F.structured_mesh(M, 1, seed=seed)
    if shuffle:
        perm = np.random.default_rng(seed).permutation(el2.shape[0])
        el2, el1 = np.ascontiguousarray(el2[perm]), np.ascontiguousarray(el1[perm])
    if swap:  # no vertex map: the pressure nodes are summed by a pass of their own
        el1 = np.ascontiguousarray(el1[:, [1, 0, 2, 3]])
    a = F.Assembler(F.NAVIER_STOKES, xyz2, el2, elements_p=el1, num_nodes_p=xyz1.shape[0], viscosity=0.01,
                    density=1.3, newton=kw.pop("newton", True), **kw)
    return a, xyz2, el2, el1, xyz1.shape[0], F.fourier_field(xyz2, seed=seed), F.uniform_field(seed, xyz1.shape[0])


@pytest.mark.parametrize("M,shuffle,swap,newton", [(1, False, False, True), (2, True, False, False),
                                                   (3, False, True, True), (5, True, False, True)])
def test_navier_stokes(F, M, shuffle, swap, newton):
    a, xyz2, el2, el1, n1, u, p = ns(F, M, 40 + M, shuffle, swap, newton=newton)
    _, ru, rp = a.assemble(u=u, p=p, jacobian=False)
    _, (ou, op) = O.assemble_ns(xyz2, el2, el1, n1, u, p, 0.01, 1.3, newton, blocks=(0,))
    assert rel(ru, ou) < TOL_NS and rel(rp, op) < TOL_NS
    _, ju, jp = a.assemble(u=u, p=p)
    assert same(ru, ju) and same(rp, jp)
    # without a pressure, and with block factors
    _, ru0, rp0 = a.assemble(u=u, jacobian=False)
    _, ju0, jp0 = a.assemble(u=u)
    assert same(ru0, ju0) and same(rp0, jp0)
    a.set_coeff([[0.5, -2.0], [3.0, 1.0]])
    _, ru1, rp1 = a.assemble(u=u, p=p, jacobian=False)
    _, ju1, jp1 = a.assemble(u=u, p=p)
    assert same(ru1, ju1) and same(rp1, jp1)


@pytest.mark.parametrize("law", range(3))
def test_generalized_newtonian_with_outflow(F, law):
    a, xyz2, el2, el1, n1, u, p = ns(F, 3, 50)
    u = 0.5 * u
    a.set_viscosity_law(*LAWS[law], gamma_min=1e-12)
    faces = [[int(el2[e, i]) for i in f] for e in range(el2.shape[0])
             for f in ((0, 1, 2), (0, 1, 3), (0, 2, 3), (1, 2, 3))
             if all(abs(xyz2[el2[e, i], 0] - 1.0) < 1e-12 for i in f)]
    for fc in ([], faces):
        a.set_outflow_faces(np.array(fc, dtype=np.int32).reshape(-1, 3))
        for coeff in ([[1.0, 1.0], [1.0, 1.0]], [[0.5, -2.0], [3.0, 1.0]]):
            a.set_coeff(coeff)
            _, ru, rp = a.assemble(u=u, p=p, jacobian=False)
            _, ju, jp = a.assemble(u=u, p=p)
            assert same(ru, ju) and same(rp, jp)


@pytest.mark.parametrize("problem,nq", [("LINEAR_ELASTICITY", 4), ("NONLINEAR_ELASTICITY", 5),
                                        ("NONLINEAR_ELASTICITY2", 5), ("ANISO_FIBER", 4), ("LINEAR_ELASTICITY", 5),
                                        ("NONLINEAR_ELASTICITY", 4)])
@pytest.mark.parametrize("M", [1, 4])
def test_elasticity(F, problem, nq, M):
    xyz, el = F.structured_mesh(M, 2, seed=60)
    el = np.ascontiguousarray(el[np.random.default_rng(60).permutation(el.shape[0])])
    u = F.fourier_field(xyz, seed=60, kmin=1, kmax=2, scale=0.004)
    a = F.Assembler(getattr(F, problem), xyz, el, E=32.0 / 11.0, poisson_ratio=5.0 / 11.0, quad_points=nq)
    _, r, _ = a.assemble(u=u, jacobian=False)
    _, j, _ = a.assemble(u=u)
    assert same(r, j)
    if problem != "ANISO_FIBER":
        a.set_element_moduli(np.random.default_rng(61).uniform(0.5, 4.0, el.shape[0]))
        _, r, _ = a.assemble(u=u, jacobian=False)
        _, j, _ = a.assemble(u=u)
        assert same(r, j)


def test_elasticity_against_the_oracle_and_at_rest(F):
    xyz, el = F.structured_mesh(3, 2, seed=62)
    u = F.fourier_field(xyz, seed=62, kmin=1, kmax=2, scale=0.004)  # det F in [0.73, 1.24]
    for problem, law, npts in (("LINEAR_ELASTICITY", O.LAW_SKR1, 4), ("NONLINEAR_ELASTICITY2", O.LAW_SKR3, 5)):
        a = F.Assembler(getattr(F, problem), xyz, el, E=32.0 / 11.0, poisson_ratio=5.0 / 11.0)
        _, r, _ = a.assemble(u=u, jacobian=False)
        _, ores = O.assemble_vec(1, O.law_from_E_nu(law, 32.0 / 11.0, 5.0 / 11.0), npts, xyz, el, u)
        assert rel(r, ores) < TOL_HYPER
    a = F.Assembler(F.LINEAR_ELASTICITY, xyz, el)
    _, r, _ = a.assemble(u=None, jacobian=False)
    assert not r.any()


def test_surrogate_with_fallback_points(F):
    xyz, el = F.structured_mesh(4, 2, seed=63)
    u = F.fourier_field(xyz, seed=63, kmin=1, kmax=2, scale=0.004)
    rng = np.random.default_rng(63)
    model = {"W1": 0.5 * rng.standard_normal((64, 4)), "b1": 0.1 * rng.standard_normal(64),
             "W2": rng.standard_normal((64, 64)) / 8.0, "b2": 0.1 * rng.standard_normal(64),
             "w3": 0.1 * rng.standard_normal(64), "b3": 0.0, "out_scale": 0.01,
             "in_shift": [0.0, 0.0, 1.0, 1.0], "in_scale": [0.0, 0.0, 20.0, 20.0]}
    a = F.Assembler(F.ANISO_FIBER, xyz, el, surrogate=True, E=32.0 / 11.0, poisson_ratio=5.0 / 11.0)
    a.set_surrogate(model, inv_lo=(-1e30, -1e30, 0.99, 0.99), inv_hi=(1e30, 1e30, 1.01, 1.01))
    _, r, _ = a.assemble(u=u, jacobian=False)
    fb = a.surrogate_fallbacks()
    _, j, _ = a.assemble(u=u)
    assert fb == a.surrogate_fallbacks() and 0 < fb[0] < fb[1]
    assert same(r, j)


def test_errors_are_reported(F):
    xyz, el = F.structured_mesh(2, 2, seed=64)
    u = F.fourier_field(xyz, seed=64, kmin=1, kmax=2, scale=0.5)  # det F <= 0 somewhere
    a = F.Assembler(F.NONLINEAR_ELASTICITY, xyz, el)
    for jac in (True, False):
        with pytest.raises(F.FeddError) as err:
            a.assemble(u=u, jacobian=jac)
        assert err.value.code == 4  # FEDD_ERR_NONFINITE
    flat = xyz.copy()
    flat[el[5, :4]] = flat[el[5, 0]]
    b = F.Assembler(F.LINEAR_ELASTICITY, flat, el)
    with pytest.raises(F.FeddError):
        b.assemble(u=0 * u, jacobian=False)
