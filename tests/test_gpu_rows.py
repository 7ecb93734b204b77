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
