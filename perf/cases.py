"""The work that users of the engine have it do, as cases that can be timed.

A case names one call of a simulation: the Jacobian and/or residual of a problem on a tetrahedral mesh, written
into device CSR values and vectors that the caller owns (the call of a Newton step), one short training run of
the strain-energy surrogate, or the set-up of an assembler on a new mesh.  The mesh is a box of nx x ny x nz
hexahedra, six tetrahedra each, interior vertices moved by up to 0.1 h, and is numbered in one of two ways:

  lattice   P2 nodes in lattice order (x fastest), elements hexahedron by hexahedron: FEDDLib's structured meshes
  shuffled  vertices and elements in random order, P2 nodes as vertices first and then the edges by their
            (min, max) vertex pair: a mesh file as a mesh generator leaves it, refined to P2

Meshes, fields and the 64-bit values of `exact` are made here with torch and numpy alone.
"""
import math

import numpy as np
import torch

import feddlib_gb300 as F

DEV = "cuda"
F64 = torch.float64

# edges of the P2 element at local nodes 4..9
_EDGES = ((0, 1), (1, 2), (0, 2), (0, 3), (1, 3), (2, 3))
# Carreau-Yasuda with FEDDLib's blood parameters (lambda, n, eta0, etaInf, a)
_BLOOD = (1.902, 0.22, 0.056, 0.00345, 1.25)
# the neo-Hooke matrix mu = 1, lambda = 10 and the two fibre families at +-40 degrees
_SOFT = dict(E=32.0 / 11.0, nu=5.0 / 11.0)
_FIBRE = dict(k1=2.0, k2=1.0, angle=40.0)
_STEEL = dict(E=1000.0, nu=0.3)


# ---------------------------------------------------------------- cases ------
def _box(name, kind, n, numbering="lattice", **opt):
    nx, ny, nz = (n, n, n) if isinstance(n, int) else n
    return dict(name=name, kind=kind, nx=nx, ny=ny, nz=nz, numbering=numbering, **opt)


def listed():
    return [
        # the smallest call of all: P1 Poisson stiffness and load on a coarse mesh, FP64 (launch latency)
        _box("laplace_p1_16", "laplace", 16, order=1, jacobian=True, residual=True),
        # a coarse fluid problem, as in a convergence study or a coarse level: launches and latency count
        _box("ns_newton_6", "ns", 6, newton=True, jacobian=True, residual=True),
        # the Newton step of a flow solver: Jacobian and residual of P2-P1 Navier-Stokes (the headline size)
        _box("ns_newton_48", "ns", 48, newton=True, jacobian=True, residual=True),
        # the Picard matrix on a mesh read from a file, box sides that fit no tile
        _box("ns_picard_file", "ns", (27, 19, 33), "shuffled", newton=False, jacobian=True, residual=False),
        # the residual alone: FEDDLib assembles "Rhs" in a call of its own, and line searches need only it
        _box("ns_residual_40", "ns", 40, newton=True, jacobian=False, residual=True),
        # a Newton step of a generalized-Newtonian (blood) flow
        _box("gn_newton_32", "gn", 32, newton=True, jacobian=True, residual=True),
        # linear elasticity: the stiffness matrix at rest, assembled once per problem
        _box("elasticity_32", "hyper", 32, law="neo1", field=False, moduli=False, jacobian=True, residual=False),
        # the Newton step of compressible neo-Hooke hyperelasticity: the largest call
        _box("neo_hooke_64", "hyper", 64, law="neo1", field=True, moduli=False, jacobian=True, residual=True),
        # the hyperelastic residual alone (5-point law, a modulus per element) on a mesh from a file
        _box("neo_hooke_residual_file", "hyper", (41, 29, 35), "shuffled", law="neo2", field=True, moduli=True,
             jacobian=False, residual=True),
        # the Newton step of the two-fibre law through its network
        _box("fibre_network_40", "hyper", 40, law="net", field=True, moduli=False, jacobian=True, residual=True),
        # training of that network: some mini-batch steps on samples of the law
        dict(name="train_65536", kind="train", samples=200_000, batch=65_536, steps=8),
        # a new mesh: connectivity, CSR patterns and maps of a Navier-Stokes assembler
        _box("setup_ns_24", "setup", 24, "shuffled"),
    ]


def draw(rng):
    kind = rng.choice(["laplace", "ns", "ns", "gn", "hyper", "hyper", "hyper", "train", "setup"])
    if kind == "train":
        batch = int(round(math.exp(rng.uniform(math.log(2_000), math.log(65_536)))))
        return dict(kind=kind, samples=batch + rng.randrange(1, 134_465), batch=batch, steps=rng.randrange(2, 9))
    top = {"laplace": 64, "ns": 48, "gn": 32, "hyper": 56, "setup": 24}[kind]
    mean = math.exp(rng.uniform(math.log(4), math.log(top)))
    a, b = math.exp(rng.uniform(-0.3, 0.3)), math.exp(rng.uniform(-0.3, 0.3))
    n = [max(2, int(round(mean * s))) for s in (a, b, 1.0 / (a * b))]
    while n[0] * n[1] * n[2] > top ** 3:
        n[n.index(max(n))] -= 1
    case = dict(kind=kind, nx=n[0], ny=n[1], nz=n[2], numbering=rng.choice(["lattice", "lattice", "shuffled"]))
    mode = rng.choice([(True, True), (True, False), (False, True)])
    if kind != "setup":
        case.update(jacobian=mode[0], residual=mode[1])
    if kind == "laplace":
        case.update(order=rng.choice([1, 2]))
    elif kind in ("ns", "gn"):
        case.update(newton=rng.choice([True, False]))
    elif kind == "hyper":
        law = rng.choice(["neo1", "neo2", "fibre", "net"])
        case.update(law=law, field=True, moduli=law.startswith("neo") and rng.random() < 0.3)
    return case


# ----------------------------------------------------------------- meshes ----
def _generator(seed, stream):
    return torch.Generator().manual_seed(1_000_003 * seed + stream)


def _mesh(case, seed):
    """(vertices, P1 elements, P2 nodes, P2 elements) on the device."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    h = 1.0 / max(nx, ny, nz)
    g = _generator(seed, 1)
    k, j, i = torch.meshgrid(torch.arange(nz + 1), torch.arange(ny + 1), torch.arange(nx + 1), indexing="ij")
    ijk = torch.stack([i, j, k], -1).reshape(-1, 3)
    size = torch.tensor([nx, ny, nz])
    inner = ((ijk > 0) & (ijk < size)).all(1, keepdim=True)
    move = (2.0 * torch.rand(ijk.shape, generator=g, dtype=F64) - 1.0) * 0.1
    x1 = ((ijk.to(F64) + move * inner) * h).to(DEV)
    # six tetrahedra of every hexahedron: the paths from its first to its last corner along the axes
    kc, jc, ic = torch.meshgrid(torch.arange(nz), torch.arange(ny), torch.arange(nx), indexing="ij")
    corner = torch.stack([ic, jc, kc], -1).reshape(-1, 1, 1, 3)
    paths = []
    for axes, even in (((0, 1, 2), 1), ((1, 2, 0), 1), ((2, 0, 1), 1), ((0, 2, 1), 0), ((2, 1, 0), 0), ((1, 0, 2), 0)):
        p = [[0, 0, 0]]
        for a in axes:
            p.append([p[-1][d] + (d == a) for d in range(3)])
        if not even:  # positive orientation
            p[1], p[2] = p[2], p[1]
        paths.append(p)
    v = (corner + torch.tensor(paths)[None]).reshape(-1, 4, 3).to(DEV)  # lattice positions of every element
    e1 = v[..., 0] + (nx + 1) * (v[..., 1] + (ny + 1) * v[..., 2])
    n1 = x1.shape[0]
    if case["numbering"] == "shuffled":
        old = torch.randperm(n1, generator=g).to(DEV)  # new number -> old number
        new = torch.empty_like(old)
        new[old] = torch.arange(n1, device=DEV)
        x1 = x1[old].contiguous()
        e1 = new[e1][torch.randperm(e1.shape[0], generator=g).to(DEV)]
        ends = torch.stack([e1[:, list(e)] for e in _EDGES], 1)  # (ne, 6, 2)
        key = ends.min(-1).values * n1 + ends.max(-1).values
        uniq, edge = torch.unique(key, return_inverse=True)
        x2 = torch.cat([x1, 0.5 * (x1[uniq // n1] + x1[uniq % n1])])
        e2 = torch.cat([e1, n1 + edge], 1)
    else:
        fine = torch.cat([2 * v, torch.stack([v[:, a] + v[:, b] for a, b in _EDGES], 1)], 1)
        e2 = fine[..., 0] + (2 * nx + 1) * (fine[..., 1] + (2 * ny + 1) * fine[..., 2])
        x2 = torch.empty(((2 * nx + 1) * (2 * ny + 1) * (2 * nz + 1), 3), dtype=F64, device=DEV)
        x2[e2[:, :4]] = x1[e1]
        for t, (a, b) in enumerate(_EDGES):
            x2[e2[:, 4 + t]] = 0.5 * (x1[e1[:, a]] + x1[e1[:, b]])
    return x1.contiguous(), e1.to(torch.int32).contiguous(), x2.contiguous(), e2.to(torch.int32).contiguous()


def _modes(x, seed, kmax, scale):
    """Sum of 8 Fourier modes with wave numbers 1..kmax and unit amplitude vectors, times scale."""
    g = _generator(seed, 2)
    u = torch.zeros_like(x)
    for _ in range(8):
        k = torch.randint(1, kmax + 1, (3,), generator=g).to(F64)
        a = torch.randn(3, generator=g, dtype=F64)
        phase = 2.0 * math.pi * torch.rand(1, generator=g, dtype=F64)
        a = (a / a.norm() * scale).to(x.device)
        u += torch.sin(2.0 * math.pi * (x @ k.to(x.device)) + phase.to(x.device))[:, None] * a
    return u


def _inputs(case, seed):
    """What the call is made on: mesh, nodal fields, moduli."""
    x1, e1, x2, e2 = _mesh(case, seed)
    kind = case["kind"]
    d = dict(x1=x1, e1=e1, x2=x2, e2=e2, u=None, p=None, moduli=None)
    if kind in ("ns", "gn", "setup"):
        d["u"] = _modes(x2, seed, 4, 1.0)
        d["p"] = (2.0 * torch.rand(x1.shape[0], generator=_generator(seed, 3), dtype=F64) - 1.0).to(DEV)
    elif kind == "hyper" and case["field"]:
        # det F stays within about [0.65, 1.35]
        d["u"] = _modes(x2, seed, 2, 0.004)
        if case["moduli"]:
            t = torch.rand(e2.shape[0], generator=_generator(seed, 4), dtype=F64)
            d["moduli"] = _material(case)["E"] * torch.exp(2.0 * t - 1.0)
    return d


def _material(case):
    return _SOFT if case["field"] else _STEEL


def _network(seed):
    """A 4-64-64-1 network as training leaves it: frozen I1 and J, the fibre invariants as max(I4 - 1, 0)^2."""
    r = np.random.default_rng(1_000_003 * seed + 5)
    f = lambda *s: r.standard_normal(s).astype(np.float32)
    return dict(W1=f(64, 4) * np.float32(0.5), b1=f(64) * np.float32(0.1), W2=f(64, 64) * np.float32(0.125),
                b2=f(64) * np.float32(0.1), w3=f(64) * np.float32(0.125), b3=0.25, out_scale=0.0625, in_clamp=12,
                in_shift=(3.0, 1.0, 1.0, 1.0), in_scale=(0.0, 0.0, 32.0, 32.0))


def _samples(case, seed):
    """Training samples: normalised fibre invariants, energy and its gradient."""
    r = np.random.default_rng(1_000_003 * seed + 6)
    e = np.maximum(r.normal(0.05, 0.08, (case["samples"], 2)), 0.0)
    z = e * e
    s = 1.0 / np.sqrt((z * z).mean())
    ex = np.exp(_FIBRE["k2"] * z)
    psi = (_FIBRE["k1"] / (2.0 * _FIBRE["k2"]) * (ex - 1.0)).sum(1)
    top = psi.max()
    x, tg = np.zeros((case["samples"], 4)), np.zeros((case["samples"], 4))
    x[:, 2:] = z * s
    tg[:, 2:] = 0.5 * _FIBRE["k1"] * ex / (s * top)
    par = dict(W1=0.5 * r.standard_normal((64, 4)), b1=np.zeros(64), W2=r.standard_normal((64, 64)) / 8.0,
               b2=np.zeros(64), w3=r.standard_normal(64) / 8.0, b3=0.0)
    f = lambda a: np.asarray(a, dtype=np.float32)
    return f(x), f(psi / top), f(tg), {k: f(v) if k != "b3" else 0.0 for k, v in par.items()}


# ------------------------------------------------------------ prepare, run ---
def _assembler(case, d):
    kind, order = case["kind"], case.get("order", 2)
    if kind == "laplace":
        x, e = (d["x1"], d["e1"]) if order == 1 else (d["x2"], d["e2"])
        return F.Assembler(F.LAPLACE, x, e, fe_order=order, source=1.0)
    if kind in ("ns", "gn", "setup"):
        asm = F.Assembler(F.NAVIER_STOKES, d["x2"], d["e2"], elements_p=d["e1"], num_nodes_p=d["x1"].shape[0],
                          viscosity=0.01, density=1.0, newton=case.get("newton", True))
        if kind == "gn":
            asm.set_viscosity_law(asm.CARREAU_YASUDA, _BLOOD, gamma_min=1e-12)
        return asm
    m = _material(case)
    problem = {"neo1": F.LINEAR_ELASTICITY, "neo2": F.NONLINEAR_ELASTICITY}.get(case["law"], F.ANISO_FIBER)
    asm = F.Assembler(problem, d["x2"], d["e2"], E=m["E"], poisson_ratio=m["nu"], surrogate=case["law"] == "net",
                      k1=_FIBRE["k1"], k2=_FIBRE["k2"], fiber_angle_deg=_FIBRE["angle"])
    if d["moduli"] is not None:
        asm.set_element_moduli(d["moduli"].numpy())
    return asm


def prepare(case, seed):
    if case["kind"] == "train":
        x, ty, tg, par = _samples(case, seed)
        return dict(case=case, x=x, ty=ty, tg=tg, par=par, seed=seed)
    d = _inputs(case, seed)
    torch.cuda.synchronize()
    if case["kind"] == "setup":
        return dict(case=case, d=d)
    asm = _assembler(case, d)
    if case.get("law") == "net":
        asm.set_surrogate(_network(seed))
    empty = lambda n: torch.empty(n, dtype=F64, device=DEV)
    vals = [empty(asm.block_info(b)[2]) for b in range(asm.nblocks)] if case["jacobian"] else []
    ru = empty(asm.n_u) if case["residual"] else None
    rp = empty(asm.n_p) if case["residual"] and asm.n_p else None
    st = dict(case=case, asm=asm, vals=vals, ru=ru, rp=rp, u=None, p=None)
    if case["kind"] != "laplace":
        st.update(u=d["u"], p=d["p"])
    torch.cuda.synchronize()
    return st


class _View:
    """A device array of the engine, for torch.as_tensor."""

    def __init__(self, ptr, n, typestr):
        self.__cuda_array_interface__ = dict(shape=(n,), typestr=typestr, data=(ptr, False), version=2)


def _pattern(asm, block):
    rows, _, nnz = asm.block_info(block)
    rp, ci = asm.device_pattern(block)
    out = [torch.as_tensor(_View(rp, rows + 1, "<i8"), device=DEV).clone()]
    if nnz:
        out.append(torch.as_tensor(_View(ci, nnz, "<i4"), device=DEV).clone())
    return out


def run(state):
    case = state["case"]
    if case["kind"] == "train":
        tr = F.Trainer(64, state["x"], state["ty"], state["tg"])
        tr.set_params(state["par"])
        loss = tr.run(case["steps"], case["batch"], 3e-3, seed=state["seed"])
        out = tr.get_params()
        tr.close()
        return dict(loss=loss, **out)
    if case["kind"] == "setup":
        asm = _assembler(case, state["d"])
        out = [_pattern(asm, b) for b in range(4)]
        torch.cuda.current_stream().synchronize()  # the copies are done before the handle frees its patterns
        asm.close()
        return out
    ptr = lambda t: None if t is None else t.data_ptr()
    state["asm"].assemble_device(ptr(state["u"]), ptr(state["p"]), [t.data_ptr() for t in state["vals"]],
                                 ptr(state["ru"]), ptr(state["rp"]), jacobian=case["jacobian"],
                                 residual=case["residual"], stream=torch.cuda.current_stream().cuda_stream)
    out = {"vals%d" % b: t for b, t in enumerate(state["vals"])}
    if case["residual"]:
        out["res_u"] = state["ru"]
        if state["rp"] is not None:
            out["res_p"] = state["rp"]
    return out


def work(case):
    """Mesh and fields read once, CSR values and residuals written once; the multiplications and additions of the
    element integrals as the weak form has them for affine elements."""
    if case["kind"] == "train":
        n = case["steps"] * case["batch"]
        return {"bytes": n * (9 * 4 + 8) + 8 * 4 * 4609, "flops": n * 3 * 5 * 64 * 64 * 2}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    v, t = (nx + 1) * (ny + 1) * (nz + 1), 6 * nx * ny * nz
    f = (4 * t + 4 * (nx * ny + ny * nz + nz * nx)) // 2
    e = v + f - t - 1
    uu = v + e + 2 * (3 * e + 6 * f + 3 * t)  # pairs of P2 nodes that share an element
    up = v + 4 * e + 3 * f                    # a P2 node and a vertex
    kind = case["kind"]
    if kind == "setup":
        nnz = 9 * uu + 2 * 3 * up
        return {"bytes": 24 * (v + e) + 56 * t + 4 * nnz + 8 * (3 * 2 * (v + e) + 2 * v), "flops": 0}
    jac, res = case["jacobian"], case["residual"]
    if kind == "laplace":
        n, npe, nnz = (v, 4, v + 2 * e) if case["order"] == 1 else (v + e, 10, uu)
        return {"bytes": 4 * npe * t + 24 * v + 8 * (nnz * jac + n * res),
                "flops": t * (100 + (npe * (npe + 1) * 6 if jac else 0) + 2 * npe * res)}
    n = 3 * (v + e)
    if kind in ("ns", "gn"):
        newton = case["newton"]
        flops = jac * 2 * (3600 + 3600 * newton + 360) + res * 2 * (900 + 240)
        if kind == "gn":
            flops += jac * 2 * (5 * 900 + 15 * 900 * newton) + res * 2 * 5 * 180
        return {"bytes": 56 * t + 24 * v + 8 * (n + v) + jac * 8 * (9 * uu + 6 * up) + res * 8 * (n + v),
                "flops": t * flops}
    q = 5 if case["law"] == "neo2" else 4
    flops = q * (jac * 55 * 54 + 10 * 36 + res * 10 * 12)
    if case["law"] in ("fibre", "net"):
        flops += q * jac * 55 * 24
    if case["law"] == "net":
        flops += q * 4 * 64 * 64 * 2
    return {"bytes": 40 * t + 24 * v + 8 * n * case["field"] + 4 * t * case["moduli"] + jac * 8 * 9 * uu + res * 8 * n,
            "flops": t * flops}


# ------------------------------------------------------------------ exact ----
_Q4A, _Q4B = 0.585410196624968454, 0.138196601125010515
_RULE4 = ([[_Q4A, _Q4B, _Q4B], [_Q4B, _Q4A, _Q4B], [_Q4B, _Q4B, _Q4A], [_Q4B, _Q4B, _Q4B]], [1.0 / 24] * 4)
_RULE5 = ([[0.25] * 3, [1 / 6] * 3, [1 / 6, 1 / 6, 0.5], [1 / 6, 0.5, 1 / 6], [0.5, 1 / 6, 1 / 6]],
          [-2.0 / 15] + [3.0 / 40] * 4)


def _rule15():
    s = math.sqrt(15.0)
    pts, w = [[0.25] * 3], [8.0 / 405]
    for sg in (1.0, -1.0):
        b, c = (7 + sg * s) / 34, (13 - 3 * sg * s) / 34
        pts += [[b, b, b], [b, b, c], [b, c, b], [c, b, b]]
        w += [(2665 - sg * 14 * s) / 226800] * 4
    d, e = (5 - s) / 20, (5 + s) / 20
    pts += [[d, d, e], [d, e, d], [e, d, d], [d, e, e], [e, d, e], [e, e, d]]
    return pts, w + [5.0 / 567] * 6


def _basis(pts):
    """P2 values (q, 10) and reference gradients (q, 10, 3), P1 values (q, 4)."""
    p = torch.tensor(pts, dtype=F64, device=DEV)
    lam = torch.cat([1.0 - p.sum(1, keepdim=True), p], 1)
    dl = torch.tensor([[-1.0, -1, -1], [1, 0, 0], [0, 1, 0], [0, 0, 1]], dtype=F64, device=DEV)
    phi = [lam[:, a] * (2 * lam[:, a] - 1) for a in range(4)] + [4 * lam[:, a] * lam[:, b] for a, b in _EDGES]
    dphi = [(4 * lam[:, a:a + 1] - 1) * dl[a] for a in range(4)]
    dphi += [4 * (lam[:, a:a + 1] * dl[b] + lam[:, b:b + 1] * dl[a]) for a, b in _EDGES]
    return torch.stack(phi, 1), torch.stack(dphi, 1), lam


def _geometry(x, e):
    v = x[e[:, :4]]
    B = (v[:, 1:] - v[:, :1]).transpose(1, 2)  # columns x_k - x_0
    return torch.linalg.inv(B), torch.linalg.det(B)


class _Csr:
    """Sums element blocks (ne, nr, nc, dr, dc) into CSR values with node-wise dofs."""

    def __init__(self, rows, cols, nrow, ncol, dr, dc):
        self.rows, self.cols, self.ncol, self.dr, self.dc = rows.long(), cols.long(), ncol, dr, dc
        self.key = torch.unique((self.rows[:, :, None] * ncol + self.cols[:, None, :]).reshape(-1))
        row = self.key // ncol
        self.count = torch.bincount(row, minlength=nrow)
        self.start = torch.cumsum(self.count, 0) - self.count
        self.acc = torch.zeros(self.key.numel(), dr * dc, dtype=F64, device=DEV)

    def add(self, lo, hi, blocks):
        k = self.rows[lo:hi, :, None] * self.ncol + self.cols[lo:hi, None, :]
        self.acc.index_add_(0, torch.searchsorted(self.key, k.reshape(-1)), blocks.reshape(-1, self.dr * self.dc))

    def values(self):
        out = torch.empty(self.acc.numel(), dtype=F64, device=DEV)
        for lo in range(0, self.key.numel(), 1 << 24):
            row = self.key[lo:lo + (1 << 24)] // self.ncol
            a0, n = self.start[row], self.count[row]
            slot = torch.arange(lo, lo + row.numel(), device=DEV) - a0
            for i in range(self.dr):
                for j in range(self.dc):
                    out[self.dr * self.dc * a0 + i * self.dc * n + self.dc * slot + j] = \
                        self.acc[lo:lo + row.numel(), i * self.dc + j]
        return out


def _chunks(ne, step=1 << 15):
    return [(lo, min(ne, lo + step)) for lo in range(0, ne, step)]


def _exact_laplace(case, d):
    x, e = (d["x1"], d["e1"].long()) if case["order"] == 1 else (d["x2"], d["e2"].long())
    pts, w = ([[0.25] * 3], [1.0 / 6]) if case["order"] == 1 else _rule15()
    w = torch.tensor(w, dtype=F64, device=DEV)
    phi, dphi, lam = _basis(pts)
    if case["order"] == 1:
        phi, dphi = lam, torch.tensor([[[-1.0, -1, -1], [1, 0, 0], [0, 1, 0], [0, 0, 1]]], dtype=F64, device=DEV)
    stiff = torch.einsum("q,qac,qbd->cdab", w, dphi, dphi).reshape(9, -1)
    load = torch.einsum("q,qa->a", w, phi)
    n, npe = x.shape[0], e.shape[1]
    K = _Csr(e, e, n, n, 1, 1) if case["jacobian"] else None
    r = torch.zeros(n, dtype=F64, device=DEV)
    for lo, hi in _chunks(e.shape[0]):
        Bi, det = _geometry(x, e[lo:hi])
        if K:
            G = det.abs()[:, None, None] * (Bi @ Bi.transpose(1, 2))
            K.add(lo, hi, G.reshape(-1, 9) @ stiff)
        r.index_add_(0, e[lo:hi].reshape(-1), (det.abs()[:, None] * load).reshape(-1))
    return ([K.values()] if K else []), r, None


def _exact_ns(case, d):
    x, e, e1, u, p = d["x2"], d["e2"].long(), d["e1"].long(), d["u"], d["p"]
    n, n1, gn, newton = x.shape[0], d["x1"].shape[0], case["kind"] == "gn", case["newton"]
    visc = 0.0 if gn else 0.01  # times the density 1
    pts, w = _rule15()
    w = torch.tensor(w, dtype=F64, device=DEV)
    phi, dphi, lam = _basis(pts)
    lap = torch.einsum("q,qac,qbd->cdab", w, dphi, dphi).reshape(9, 100)
    adv = torch.einsum("q,qa,qk,qbc->ckab", w, phi, phi, dphi).reshape(30, 100)
    new = torch.einsum("q,qa,qb,qkc->kcab", w, phi, phi, dphi).reshape(30, 100)
    div = torch.einsum("q,qp,qbc->cbp", w, lam, dphi).reshape(3, 40)
    jac = case["jacobian"]
    K00 = _Csr(e, e, n, n, 3, 3) if jac else None
    K01 = _Csr(e, e1, n, n1, 3, 1) if jac else None
    K10 = _Csr(e1, e, n1, n, 1, 3) if jac else None
    ru, rp = torch.zeros(n, 3, dtype=F64, device=DEV), torch.zeros(n1, dtype=F64, device=DEV)
    eye = torch.eye(3, dtype=F64, device=DEV)
    for lo, hi in _chunks(e.shape[0]):
        c, c1 = e[lo:hi], e1[lo:hi]
        m = hi - lo
        Bi, det = _geometry(x, c)
        ad = det.abs()[:, None, None]
        ue, pe = u[c], p[c1]
        na = (visc * ad * (Bi @ Bi.transpose(1, 2))).reshape(m, 9) @ lap
        na += (ad * (Bi @ ue.transpose(1, 2))).reshape(m, 30) @ adv
        J = na.reshape(m, 10, 10, 1, 1) * eye
        B = -torch.einsum("ecd,cx->exd", ad * Bi, div).reshape(m, 10, 4, 3)  # (b, p, d)
        if gn:
            S, D = _viscous(Bi, ad, ue, newton)
            J = J + S
        r = torch.einsum("eabij,ebj->eai", J, ue) + torch.einsum("ebpd,ep->ebd", B, pe)
        ru.index_add_(0, c.reshape(-1), r.reshape(-1, 3))
        rp.index_add_(0, c1.reshape(-1), torch.einsum("ebpd,ebd->ep", B, ue).reshape(-1))
        if jac:
            if newton:
                g = torch.einsum("eki,ecj->eijkc", ue, ad * Bi).reshape(m, 9, 30)
                J = J + (g @ new).reshape(m, 3, 3, 10, 10).permute(0, 3, 4, 1, 2)
                if gn:
                    J = J + D
            K00.add(lo, hi, J)
            K01.add(lo, hi, B)
            K10.add(lo, hi, B.transpose(1, 2))
    return ([K00.values(), K01.values(), K10.values()] if jac else []), ru.reshape(-1), rp


def _viscous(Bi, ad, ue, newton):
    """Stress-divergence blocks (a, b, k, l) of the Carreau-Yasuda fluid and their derivative."""
    lam, nn, eta0, inf, a = _BLOOD
    m = ue.shape[0]

    def point(rule):
        w = torch.tensor(rule[1], dtype=F64, device=DEV)
        g = torch.einsum("qac,ecj->eqaj", _basis(rule[0])[1], Bi)
        du = torch.einsum("eai,eqaj->eqij", ue, g)
        sym = 0.5 * (du + du.transpose(2, 3))
        rate = torch.sqrt(2.0 * (sym * sym).sum((2, 3)))
        return w, g, sym, 1.0 + (lam * rate) ** a

    w, g, _, base = point(_RULE5)
    eta = inf + (eta0 - inf) * base ** ((nn - 1.0) / a)
    gw = g * (w * eta * ad[:, 0])[:, :, None, None]
    S = torch.einsum("eqac,eqbc->eab", gw, g)[:, :, :, None, None] * torch.eye(3, dtype=F64, device=DEV)
    S = S + torch.einsum("eqal,eqbk->eabkl", gw, g)
    if not newton:
        return S, None
    w, g, sym, base = point(_rule15())
    # FEDDLib takes the a = 2 form of the derivative for every a in (1, 3)
    der = -2.0 * (eta0 - inf) * (nn - 1.0) * lam ** a * base ** ((nn - 1.0 - a) / a)
    fa = torch.einsum("eqac,eqck->eqak", g, sym)
    gb = fa.clone()
    gb[..., 2] = g[..., 2] * sym[:, :, None, 0, 2] + g[..., 1] * sym[:, :, None, 1, 2] + g[..., 2] * sym[:, :, None, 2, 2]
    fa = fa * (-2.0 * der * w * ad[:, 0])[:, :, None, None]
    D = fa.reshape(m, 15, 30).transpose(1, 2) @ gb.reshape(m, 15, 30)
    return S, D.reshape(m, 10, 3, 10, 3).permute(0, 1, 3, 2, 4)


def _round_bf16(a):
    return torch.tensor(a).to(torch.bfloat16).to(F64).to(DEV)


def _fibre_net(net, inv4):
    """First and second derivatives of the network's energy with respect to (I4a, I4b): (n, 2), (n, 2, 2)."""
    W1, W2, w3 = (_round_bf16(net[k]) for k in ("W1", "W2", "w3"))
    b1, b2 = (torch.tensor(net[k]).to(F64).to(DEV) for k in ("b1", "b2"))
    W1 = W1[:, 2:]
    e = (inv4 - 1.0).clamp_min(0.0)
    s = net["in_scale"][2]
    x, dx, d2x = e * e * s, 2.0 * e * s, 2.0 * s * (e > 0)
    s1 = torch.sigmoid(x @ W1.T + b1)
    t1 = s1 * (1.0 - s1)
    z2 = torch.nn.functional.softplus(x @ W1.T + b1, threshold=1e9) @ W2.T + b2
    s2 = torch.sigmoid(z2)
    D = torch.stack([(s1 * W1[:, k]) @ W2.T for k in range(2)], -1)  # (n, 64, 2)
    g = torch.einsum("nj,njk->nk", w3 * s2, D)
    h = torch.einsum("nj,njk,njl->nkl", w3 * s2 * (1.0 - s2), D, D)
    beta = (w3 * s2) @ W2
    h = h + torch.einsum("ni,ik,il->nkl", beta * t1, W1, W1)
    d1 = net["out_scale"] * g * dx
    d2 = net["out_scale"] * (h * dx[:, :, None] * dx[:, None, :] + torch.diag_embed(g * d2x))
    return d1, d2


def _exact_hyper(case, d, seed):
    x, e, u = d["x2"], d["e2"].long(), d["u"]
    n, law = x.shape[0], case["law"]
    m = _material(case)
    mu = m["E"] / (2.0 * (1.0 + m["nu"]))
    la = m["nu"] * 2.0 * mu / (1.0 - 2.0 * m["nu"])
    pts, w = _RULE5 if law == "neo2" else _RULE4
    nq, w = len(w), torch.tensor(w, dtype=F64, device=DEV)
    dphi = _basis(pts)[1]
    ang = math.radians(_FIBRE["angle"])
    fib = torch.tensor([[math.cos(ang), math.sin(ang), 0.0], [math.cos(ang), -math.sin(ang), 0.0]], dtype=F64, device=DEV)
    fibres = law in ("fibre", "net")
    net = _network(seed) if law == "net" else None
    K = _Csr(e, e, n, n, 3, 3) if case["jacobian"] else None
    res = torch.zeros(n, 3, dtype=F64, device=DEV)
    eye = torch.eye(3, dtype=F64, device=DEV)
    for lo, hi in _chunks(e.shape[0]):
        c = e[lo:hi]
        Bi, det = _geometry(x, c)
        if d["moduli"] is not None:
            det = det * d["moduli"][lo:hi].to(DEV) / m["E"]
        G = torch.einsum("qac,ecj->eqaj", dphi, Bi)
        Fg = eye.expand(hi - lo, nq, 3, 3)
        if u is not None:
            Fg = Fg + torch.einsum("eai,eqaj->eqij", u[c], G)
        J = torch.linalg.det(Fg)
        cof = J[..., None, None] * torch.linalg.inv(Fg).transpose(2, 3)
        s = w * det[:, None]
        if law == "neo2":
            pj, pjj = (la * J.log() - mu) / J, (mu + la - la * J.log()) / J ** 2
        else:
            pj, pjj = -mu / J + 0.5 * la * (J - 1.0 / J), mu / J ** 2 + 0.5 * la * (1.0 + 1.0 / J ** 2)
        cv = torch.einsum("eqij,eqaj->eqai", cof, G)
        P = mu * torch.einsum("eqij,eqaj->eqai", Fg, G) + pj[..., None, None] * cv
        if fibres:
            Fa = torch.einsum("eqij,fj->eqfi", Fg, fib)
            I4 = (Fa * Fa).sum(-1)
            ag = torch.einsum("fj,eqaj->eqfa", fib, G)
            if law == "net":
                d1, d2 = _fibre_net(net, I4.reshape(-1, 2))
                d1, d2 = d1.reshape(I4.shape), d2.reshape(*I4.shape, 2)
            else:
                ep = (I4 - 1.0).clamp_min(0.0)
                ex = _FIBRE["k1"] * torch.exp(_FIBRE["k2"] * ep * ep)
                d1, d2 = ep * ex, torch.diag_embed(ex * (1.0 + 2.0 * _FIBRE["k2"] * ep * ep) * (I4 > 1.0))
            D4 = 2.0 * torch.einsum("eqfa,eqfi->eqfai", ag, Fa)
            P = P + torch.einsum("eqf,eqfai->eqai", d1, D4)
        if case["residual"]:
            res.index_add_(0, c.reshape(-1), -torch.einsum("eq,eqai->eai", s, P).reshape(-1, 3))
        if K:
            k = hi - lo
            pair = lambda wt, a, b: (a * wt[..., None, None]).reshape(k, nq, 30).transpose(1, 2) @ b.reshape(k, nq, 30)
            blocks = lambda t: t.reshape(k, 10, 3, 10, 3).permute(0, 1, 3, 2, 4)
            M = blocks(pair(s * (pjj + pj / J), cv, cv))
            M = M - blocks(pair(s * pj / J, cv, cv)).transpose(3, 4)
            gg = torch.einsum("eq,eqai,eqbi->eab", s * mu, G, G)
            if fibres:
                gg = gg + torch.einsum("eqf,eqfa,eqfb->eab", 2.0 * d1 * s[..., None], ag, ag)
                for f in range(2):
                    for h in range(2):
                        M = M + blocks(pair(s * d2[..., f, h], D4[:, :, f], D4[:, :, h]))
            K.add(lo, hi, M + gg[..., None, None] * eye)
    return ([K.values()] if K else []), res.reshape(-1), None


def _shuffled(n, seed, step, perm):
    """The trainer's seeded Fisher-Yates shuffle before step `step`."""
    mask = (1 << 64) - 1
    s = seed ^ (0x5851F42D4C957F2D * (step + 1) & mask)
    for i in range(n - 1, 0, -1):
        s = (s + 0x9E3779B97F4A7C15) & mask
        z = ((s ^ (s >> 30)) * 0xBF58476D1CE4E5B9) & mask
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
        j = (z ^ (z >> 31)) % (i + 1)
        perm[i], perm[j] = perm[j], perm[i]


def _exact_train(case, seed):
    x, ty, tg, par = _samples(case, seed)
    x, ty, tg = (torch.tensor(a).to(F64).to(DEV) for a in (x, ty, tg))
    P = {k: torch.tensor(v, dtype=torch.float32).to(F64).to(DEV).requires_grad_() for k, v in par.items()}
    m1, m2 = ({k: torch.zeros_like(v) for k, v in P.items()} for _ in range(2))
    n, batch = case["samples"], case["batch"]
    perm, cursor, loss = list(range(n)), n, 0.0
    f32 = lambda v: float(np.float32(v))
    lr, b1, b2 = f32(3e-3), f32(0.9), f32(0.999)
    for step in range(case["steps"]):
        if cursor + batch > n:
            _shuffled(n, seed, step, perm)
            cursor = 0
        idx = torch.tensor(perm[cursor:cursor + batch], device=DEV)
        cursor += batch
        z1 = x[idx] @ P["W1"].T + P["b1"]
        s1 = torch.sigmoid(z1)
        z2 = torch.nn.functional.softplus(z1, threshold=1e9) @ P["W2"].T + P["b2"]
        s2 = torch.sigmoid(z2)
        y = torch.nn.functional.softplus(z2, threshold=1e9) @ P["w3"] + P["b3"]
        g = (((P["w3"] * s2) @ P["W2"]) * s1) @ P["W1"]
        total = ((y - ty[idx]) ** 2).mean() + ((g - tg[idx]) ** 2).sum(1).mean()
        loss = float(total.detach())
        grads = torch.autograd.grad(total, list(P.values()))
        with torch.no_grad():
            for (k, v), gr in zip(P.items(), grads):
                m1[k].mul_(b1).add_(gr, alpha=1.0 - b1)
                m2[k].mul_(b2).add_(gr * gr, alpha=1.0 - b2)
                v -= lr * (m1[k] / (1.0 - b1 ** (step + 1))) / ((m2[k] / (1.0 - b2 ** (step + 1))).sqrt() + 1e-8)
    out = {k: v.detach().cpu().numpy() for k, v in P.items()}
    out["b3"] = float(out["b3"])
    return dict(loss=loss, **out)


def exact(case, seed):
    if case["kind"] == "setup":
        return None  # whole numbers
    if case["kind"] == "train":
        return _exact_train(case, seed)
    d = _inputs(case, seed)
    if case["kind"] == "laplace":
        vals, ru, rp = _exact_laplace(case, d)
    elif case["kind"] == "hyper":
        vals, ru, rp = _exact_hyper(case, d, seed)
    else:
        vals, ru, rp = _exact_ns(case, d)
    out = {"vals%d" % b: t for b, t in enumerate(vals)}
    if case["residual"]:
        out["res_u"] = ru
        if rp is not None:
            out["res_p"] = rp
    return out
