"""The velocity rows of meshes above the size from which a warp takes two nodes
at a time (some 22,000 nodes on 152 SMs): special nodes next to a lattice of
14^3 cubes (pairs from groups of four nodes) or 25^3 (of eight), all nodes'
numbers permuted, so that they meet lattice nodes in a warp.  A fan of 60 elements around one node (its list of incidences takes four
windows of 16 lanes), in its variant `wide` 28 elements that share one node
alone (253 neighbours: rows so long that a CTA holds fewer than four warps'
pairs and takes an SM's whole shared memory), and nodes no element refers to;
with and without the vertex map.

The patches do not touch the lattice, so their rows and residuals are the sums
of the oracle's element matrices over the patches' elements; the lattice's
residuals and block norms follow from the oracle's whole assembly in the
Newtonian cases of the smaller one without factors.  Bounds: 1e-6, as for the other FP32 rows."""
import functools

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

TOL = 1e-6
PRM = [1.902, 0.22, 0.056, 0.00345, 1.25]


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a) - np.asarray(b)) / max(np.linalg.norm(b), 1e-300))


def fan(shift):
    """60 elements around the origin: the hull of 32 points of the sphere."""
    spatial = pytest.importorskip("scipy.spatial")
    k = np.arange(32) + 0.5
    phi, z = np.pi * (1 + 5 ** 0.5) * k, 1 - 2 * k / 32
    pts = np.stack([np.sqrt(1 - z * z) * np.cos(phi), np.sqrt(1 - z * z) * np.sin(phi), z], axis=1)
    tri = spatial.ConvexHull(pts).simplices
    assert len(tri) == 60
    xyz = np.vstack([[0.02, -0.03, 0.01], pts])
    el = np.hstack([np.zeros((60, 1), int), tri + 1])
    # the middle node at every local place in turn
    el = np.array([np.roll(t, e % 4) for e, t in enumerate(el)])
    return 0.5 * xyz + shift, el


def wide(shift):
    """28 elements that share one node."""
    rng = np.random.default_rng(5)
    base = np.array([[1.0, 0.1, 0.0], [0.0, 1.0, 0.2], [0.3, 0.0, 1.0]])
    xyz = np.vstack([np.zeros((1, 3))] + [base + 0.1 * rng.standard_normal((3, 3)) for _ in range(28)])
    el = np.array([[0, 3 * e + 1, 3 * e + 2, 3 * e + 3] for e in range(28)])
    return 0.5 * xyz + shift, el


def refine(xyz, el):
    """P2 nodes and elements of a P1 mesh (det B > 0)."""
    d = xyz[el[:, 1:]] - xyz[el[:, :1]]
    flip = np.linalg.det(d) < 0
    el = el.copy()
    el[flip, 2], el[flip, 3] = el[flip, 3].copy(), el[flip, 2].copy()
    edges, mid = {}, []
    el2 = np.empty((len(el), 10), int)
    el2[:, :4] = el
    for e, t in enumerate(el):
        for k, (a, b) in enumerate(((0, 1), (1, 2), (0, 2), (0, 3), (1, 3), (2, 3))):
            key = tuple(sorted((int(t[a]), int(t[b]))))
            if key not in edges:
                edges[key] = len(xyz) + len(mid)
                mid.append((xyz[t[a]] + xyz[t[b]]) / 2)
            el2[e, 4 + k] = edges[key]
    return np.vstack([xyz, mid]), el2, el


@functools.lru_cache(maxsize=None)
def mesh(M, with_wide):
    """(xyz2, el2, el1, number of P1 nodes, patch elements)"""
    import feddlib_gb300 as F
    xyz2, el2 = F.structured_mesh(M, 2, seed=21)
    xyz1, el1 = F.structured_mesh(M, 1, seed=21)
    n1, lattice = xyz1.shape[0], len(el2)
    for patch in [fan] + ([wide] if with_wide else []):
        px, pe2, pe1 = refine(*patch(np.array([3.0 + 2.0 * (patch is wide), 0.0, 0.0])))
        el2 = np.vstack([el2, pe2 + len(xyz2)])
        el1 = np.vstack([el1, pe1 + n1])
        xyz2, n1 = np.vstack([xyz2, px]), n1 + pe1.max() + 1
    xyz2 = np.vstack([xyz2, [[9.0, 9.0, 9.0], [8.0, 9.0, 9.0], [9.0, 8.0, 9.0]]])  # no element refers to these
    rng = np.random.default_rng(22)
    p2, p1 = rng.permutation(len(xyz2)), rng.permutation(n1)
    x = np.empty_like(xyz2)
    x[p2] = xyz2
    order = rng.permutation(len(el2))
    e2, e1 = p2[el2[order]].astype(np.int32), p1[el1[order]].astype(np.int32)
    return x, np.ascontiguousarray(e2), np.ascontiguousarray(e1), int(n1), np.flatnonzero(order >= lattice)


def dense_rows(a, block, vals, rows, cols):
    """The rows of a block as a dense matrix over the columns; other columns are empty."""
    rp, ci, (_, nc) = a.pattern(block)
    at = np.full(nc, -1)
    at[cols] = np.arange(len(cols))
    out = np.zeros((len(rows), len(cols)))
    for k, r in enumerate(rows):
        c = at[ci[rp[r]:rp[r + 1]]]
        assert (c >= 0).all()
        out[k, c] = vals[rp[r]:rp[r + 1]]
    return out


FORMS = [(True, False, None), (False, False, None), (True, False, (1.5, -0.5, 2.0, 1.0)), (True, True, None),
         (False, True, None)]  # newton, viscosity law, residual factors


@pytest.mark.parametrize("M,with_wide,vertex_map,newton,gn,coeff",
                         [(14, w, v, *f) for w in (False, True) for v in (True, False) for f in FORMS] +
                         [(25, False, True, *FORMS[0]), (25, False, False, *FORMS[3])])
def test_special_nodes_in_pairs(M, with_wide, vertex_map, newton, gn, coeff):
    import feddlib_gb300 as F
    xyz2, el2, el1, n1, patch = mesh(M, with_wide)
    if not vertex_map:
        el1 = np.ascontiguousarray(el1[:, [1, 0, 2, 3]])
    u, p = 0.5 * F.fourier_field(xyz2, seed=23), F.uniform_field(23, n1)
    visc, dens = 0.01, 1.3
    a = F.Assembler(F.NAVIER_STOKES, xyz2, el2, elements_p=el1, num_nodes_p=n1, viscosity=visc, density=dens,
                    newton=newton)
    law = O.visc_law(0, PRM, 1e-12)
    faces = None
    if gn:
        a.set_viscosity_law(0, PRM, gamma_min=1e-12)
        # outflow through some of the fan's outer faces, opposite the node all of its elements have
        count = np.bincount(el2[patch][:, :4].ravel())
        mid = int(np.flatnonzero(count == 60)[0])
        faces = [[int(v) for v in el2[e, :4] if v != mid] for e in patch if mid in el2[e, :4]][:20]
        a.set_outflow_faces(faces)
    if coeff is not None:
        a.set_coeff(coeff)
    # device buffers: the whole mesh in one launch
    import torch
    du, dp = torch.from_numpy(u).cuda(), torch.from_numpy(p).cuda()
    bufs = [torch.full((a.block_info(b)[2],), np.nan, dtype=torch.float64, device="cuda") for b in range(3)]
    dru = torch.full((a.n_u,), np.nan, dtype=torch.float64, device="cuda")
    drp = torch.full((a.n_p,), np.nan, dtype=torch.float64, device="cuda")
    a.assemble_device(du.data_ptr(), dp.data_ptr(), [b.data_ptr() for b in bufs], dru.data_ptr(), drp.data_ptr())
    torch.cuda.synchronize()
    a.check()
    vals, ru, rp = [b.cpu().numpy() for b in bufs], dru.cpu().numpy(), drp.cpu().numpy()
    if with_wide:
        nbr = np.diff(a.pattern(0)[0])[::3] // 3
        assert nbr.max() == 253
    # the patches against the oracle's elements
    n2 = len(xyz2)
    nodes, nodes_p = np.unique(el2[patch]), np.unique(el1[patch])
    dofs = (3 * nodes[:, None] + np.arange(3)).ravel()
    at = np.full(3 * n2, -1)
    at[dofs] = np.arange(len(dofs))
    atp = np.full(n1, -1)
    atp[nodes_p] = np.arange(len(nodes_p))
    J = [np.zeros((len(dofs), len(dofs))), np.zeros((len(dofs), len(nodes_p))), np.zeros((len(nodes_p), len(dofs)))]
    oru, orp = np.zeros(len(dofs)), np.zeros(len(nodes_p))
    taken = O.outflow_owners(el2, faces)[1] if faces else {}
    for e in patch:
        ue = u.reshape(-1, 3)[el2[e]].ravel()
        if gn:
            Je, re = O.elem_gn(xyz2[el2[e]], ue, p[el1[e]], law, dens, newton)
            if e in taken:
                re = re.copy()
                re[:30] += O.gn_outflow(xyz2[el2[e]], xyz2[faces[taken[e]]], ue, law) @ ue
        else:
            Je, re = O.elem_ns(xyz2[el2[e]], ue, p[el1[e]], visc, dens, newton, coeff=coeff or (1, 1, 1, 1))
        d, q = at[(3 * el2[e][:, None] + np.arange(3)).ravel()], atp[el1[e]]
        J[0][np.ix_(d, d)] += Je[:30, :30]
        J[1][np.ix_(d, q)] += Je[:30, 30:]
        J[2][np.ix_(q, d)] += Je[30:, :30]
        oru[d] += re[:30]
        orp[q] += re[30:]
    assert rel(dense_rows(a, 0, vals[0], dofs, dofs), J[0]) < TOL
    assert rel(dense_rows(a, 1, vals[1], dofs, nodes_p), J[1]) < TOL
    assert rel(dense_rows(a, 2, vals[2], nodes_p, dofs), J[2]) < TOL
    assert rel(ru[dofs], oru) < TOL and rel(rp[nodes_p], orp) < TOL
    free = np.setdiff1d(np.arange(n2), el2)
    assert len(free) == 3 and not ru.reshape(-1, 3)[free].any()
    # the lattice around them, and the node ranges of the host-buffer call
    hv, hru, hrp = a.assemble(u=u, p=p)
    assert all(np.array_equal(x, y) for x, y in zip(vals, hv)) and np.array_equal(ru, hru) and np.array_equal(rp, hrp)
    if M == 14 and not gn and coeff is None:
        blocks, (ou, op) = O.assemble_ns(xyz2, el2, el1, n1, u, p, visc, dens, newton, blocks=(0, 1, 2))
        for b in range(3):
            np.testing.assert_array_equal(a.pattern(b)[1], blocks[b][1])
            assert rel(vals[b], blocks[b][2]) < TOL
        assert rel(ru, ou) < TOL and rel(rp, op) < TOL
