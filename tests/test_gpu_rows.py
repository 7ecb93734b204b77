"""The elasticity rows' write-out: a node's 9 K values start at any multiple of
8 bytes, so the pairs of values that go out as 16-byte stores start at the
first or the second one.  Value arrays at even and odd offsets of a larger
buffer give the same values, and nothing around them is written."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 2, 5])
def test_value_arrays_at_any_offset(M):
    import torch
    import feddlib_gb300 as F
    xyz, el = F.structured_mesh(M, 2, seed=70 + M)
    # two nodes that no element references: rows without values
    xyz = np.vstack([xyz[:3], xyz[:1], xyz[3:], xyz[:1]])
    el = np.where(el >= 3, el + 1, el).astype(np.int32)
    u = F.fourier_field(xyz, seed=70, kmin=1, kmax=2, scale=0.004)
    a = F.Assembler(F.NONLINEAR_ELASTICITY, xyz, el)
    nnz = a.block_info(0)[2]
    (v,), r, _ = a.assemble(u=u)
    assert np.isfinite(v).all() and not r.reshape(-1, 3)[[3, -1]].any()
    du = torch.from_numpy(u).cuda()
    for offset in range(4):
        buf = torch.full((nnz + 8,), -7.0, dtype=torch.float64, device="cuda")
        res = torch.full((a.n_u + 4,), -7.0, dtype=torch.float64, device="cuda")
        a.assemble_device(du.data_ptr(), None, [buf.data_ptr() + 8 * offset], res.data_ptr() + 8 * (offset & 1), None)
        torch.cuda.synchronize()
        b, x = buf.cpu().numpy(), res.cpu().numpy()
        assert np.array_equal(b[offset:offset + nnz], v) and np.array_equal(x[offset & 1:][:a.n_u], r)
        assert (b[:offset] == -7.0).all() and (b[offset + nnz:] == -7.0).all()


@pytest.mark.parametrize("newton,gn", [(True, False), (False, False), (True, True)])
@pytest.mark.parametrize("M", [1, 3])
def test_navier_stokes_blocks_at_any_offset(M, newton, gn):
    """The three blocks' runs of a node are written the same way; odd node
    counts leave half of the last pair of nodes empty."""
    import torch
    import feddlib_gb300 as F
    xyz2, el2 = F.structured_mesh(M, 2, seed=80 + M)
    xyz1, el1 = F.structured_mesh(M, 1, seed=80 + M)
    u, p = 0.5 * F.fourier_field(xyz2, seed=80), F.uniform_field(80, xyz1.shape[0])
    a = F.Assembler(F.NAVIER_STOKES, xyz2, el2, elements_p=el1, num_nodes_p=xyz1.shape[0], viscosity=0.01, density=1.3,
                    newton=newton)
    if gn:
        a.set_viscosity_law(0, [1.902, 0.22, 0.056, 0.00345, 1.25], gamma_min=1e-12)
    want, ru, rp = a.assemble(u=u, p=p)
    du, dp = torch.from_numpy(u).cuda(), torch.from_numpy(p).cuda()
    for offset in range(4):
        offs = [offset & 1, offset >> 1, (offset + 1) & 1]
        bufs = [torch.full((w.size + 4,), -7.0, dtype=torch.float64, device="cuda") for w in want]
        dru = torch.zeros(a.n_u, dtype=torch.float64, device="cuda")
        drp = torch.zeros(a.n_p, dtype=torch.float64, device="cuda")
        a.assemble_device(du.data_ptr(), dp.data_ptr(), [b.data_ptr() + 8 * o for b, o in zip(bufs, offs)],
                          dru.data_ptr(), drp.data_ptr())
        torch.cuda.synchronize()
        for b, o, w in zip(bufs, offs, want):
            x = b.cpu().numpy()
            assert np.array_equal(x[o:o + w.size], w) and (x[:o] == -7.0).all() and (x[o + w.size:] == -7.0).all()
        assert np.array_equal(dru.cpu().numpy(), ru) and np.array_equal(drp.cpu().numpy(), rp)


@pytest.mark.parametrize("M,newton,gn", [(12, True, False), (12, False, True), (14, True, True), (14, False, False),
                                         (29, True, False)])
def test_navier_stokes_rows_of_every_mesh_size(M, newton, gn):
    """How the velocity rows' nodes are given to the warps depends on their
    number: one node per warp (15,625 nodes), pairs of groups of four (24,389)
    or of eight (205,379).  The host-buffer call works in node ranges, which
    take another of these forms than the whole mesh: the same values."""
    import torch
    import feddlib_gb300 as F
    xyz2, el2 = F.structured_mesh(M, 2, seed=90 + M)
    xyz1, el1 = F.structured_mesh(M, 1, seed=90 + M)
    u, p = 0.5 * F.fourier_field(xyz2, seed=90), F.uniform_field(90, xyz1.shape[0])
    a = F.Assembler(F.NAVIER_STOKES, xyz2, el2, elements_p=el1, num_nodes_p=xyz1.shape[0], viscosity=0.01, density=1.3,
                    newton=newton)
    if gn:
        a.set_viscosity_law(0, [1.902, 0.22, 0.056, 0.00345, 1.25], gamma_min=1e-12)
    want, ru, rp = a.assemble(u=u, p=p)
    du, dp = torch.from_numpy(u).cuda(), torch.from_numpy(p).cuda()
    bufs = [torch.empty(w.size, dtype=torch.float64, device="cuda") for w in want]
    dru = torch.empty(a.n_u, dtype=torch.float64, device="cuda")
    drp = torch.empty(a.n_p, dtype=torch.float64, device="cuda")
    a.assemble_device(du.data_ptr(), dp.data_ptr(), [b.data_ptr() for b in bufs], dru.data_ptr(), drp.data_ptr())
    torch.cuda.synchronize()
    for b, w in zip(bufs, want):
        assert w.any() and np.array_equal(b.cpu().numpy(), w)
    assert np.array_equal(dru.cpu().numpy(), ru) and np.array_equal(drp.cpu().numpy(), rp)


@pytest.mark.parametrize("newton,gn", [(True, False), (False, False), (True, True), (False, True)])
@pytest.mark.parametrize("M", [2, 15])
def test_navier_stokes_matrix_alone(M, newton, gn):
    """A call for the matrix alone stages less of each record and sums no
    residual; the values are those of the call for both."""
    import feddlib_gb300 as F
    xyz2, el2 = F.structured_mesh(M, 2, seed=40 + M)
    xyz1, el1 = F.structured_mesh(M, 1, seed=40 + M)
    u, p = 0.5 * F.fourier_field(xyz2, seed=40), F.uniform_field(40, xyz1.shape[0])
    a = F.Assembler(F.NAVIER_STOKES, xyz2, el2, elements_p=el1, num_nodes_p=xyz1.shape[0], viscosity=0.01, density=1.3,
                    newton=newton)
    if gn:
        a.set_viscosity_law(0, [1.902, 0.22, 0.056, 0.00345, 1.25], gamma_min=1e-12)
    both, ru, _ = a.assemble(u=u, p=p)
    both = [b.copy() for b in both]
    alone, none, _ = a.assemble(u=u, p=p, residual=False)
    assert none is None and ru.any()
    for b, v in zip(both, alone):
        assert b.any() and np.array_equal(b, v)
