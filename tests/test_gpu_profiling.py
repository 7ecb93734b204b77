"""Stage times of calls whose stages differ: a call for the residual alone has
kernels of its own, fewer than the matrix call's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def elasticity(F):
    xyz, el = F.structured_mesh(3, 2, seed=31)
    return F.Assembler(F.NONLINEAR_ELASTICITY, xyz, el), dict(u=F.fourier_field(xyz, seed=31, kmin=1, kmax=2, scale=0.004))


def navier_stokes(F):
    """Without a vertex map: the pressure rows are a stage of their own."""
    xyz2, el2 = F.structured_mesh(3, 2, seed=32)
    xyz1, el1 = F.structured_mesh(3, 1, seed=32)
    a = F.Assembler(F.NAVIER_STOKES, xyz2, el2, elements_p=np.ascontiguousarray(el1[:, [1, 0, 2, 3]]),
                    num_nodes_p=xyz1.shape[0], viscosity=0.01)
    return a, dict(u=F.fourier_field(xyz2, seed=32), p=F.uniform_field(32, xyz1.shape[0]))


@pytest.mark.parametrize("make,both,alone", [
    (elasticity, {"hyper_elem", "hyper_rows"}, {"hyper_residual"}),
    (navier_stokes, {"ns_record", "ns_vel_rows", "ns_pres_rows"}, {"ns_record", "ns_residual"})])
def test_matrix_and_residual_calls_in_one_session(make, both, alone):
    import feddlib_gb300 as F
    a, fields = make(F)
    want, r, _ = a.assemble(**fields)
    a.set_profiling(True)
    a.assemble(**fields)
    a.assemble(**fields, jacobian=False)
    times = a.stage_times()
    assert set(times) == both | alone
    assert all(ms > 0.0 and calls == 2 for ms, calls in times.values())
    # a later session's stages are its own
    a.assemble(**fields, jacobian=False)
    assert set(a.stage_times()) == alone
    a.set_profiling(True)
    assert a.stage_times() == {}
    a.assemble(**fields)
    assert set(a.stage_times()) == both
    a.set_profiling(False)
    again, r2, _ = a.assemble(**fields)
    assert all(np.array_equal(v, w) for v, w in zip(again, want)) and np.array_equal(r, r2)


def test_a_call_that_fails_leaves_no_stage():
    """The surrogate's call without a network is refused; the next session's
    first stage is the first one again."""
    import feddlib_gb300 as F
    xyz, el = F.structured_mesh(2, 2, seed=33)
    a = F.Assembler(F.ANISO_FIBER, xyz, el, surrogate=True, k1=2.0, k2=1.0, fiber_angle_deg=40.0)
    a.set_profiling(True)
    with pytest.raises(F.FeddError):
        a.assemble(u=np.zeros(xyz.size))
    assert a.stage_times() == {}
