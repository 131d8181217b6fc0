"""The work that programs on this framework have it do, as cases that can be timed and checked.

Each case is one pass through the public entry points (the Feel++-style front end of ``feelpp_gb300.fe`` and
the C-ABI under it) on a mesh, a space and the handles that such a program keeps between calls. The meshes
are the seeded Kuhn boxes, hexahedral boxes and curved boxes of ``feelpp_gb300.meshgen``; the sizes follow the
framework's named configurations (P1 on 16^3, P2 and P3 on 64^3 and below, the elasticity beam, uneven batches
of 8 to 40 cells a side, the P2 heat step, matrix-free P3) and ragged boxes around them.

``exact`` restates every result in binary64 torch on its own: first-encounter dof numbering, Lagrange bases by
Vandermonde solves, Gauss quadrature, entries summed per (row, column), conjugate gradients for the solves.
"""
import ctypes
import math

import numpy as np
import torch

import feelpp_gb300 as fpp
from feelpp_gb300 import _ffi, meshgen

_env = None


def env():
    """The one context of the process, as a program has it."""
    global _env
    if _env is None:
        _env = fpp.Environment(device=0)
    return _env


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------


def listed():
    return [
        # reassembly of a small P1 problem (config 1's range and below): launches and host time count
        dict(name="assemble_p1_10x9x11", kind="assemble", order=1, nx=10, ny=9, nz=11, dtype="f64"),
        # the headline: P2 Laplace + mass with a lognormal coefficient per element, 64^3 cells
        dict(name="assemble_p2_64", kind="assemble", order=2, nx=64, ny=64, nz=64, dtype="f64"),
        # P3 on a ragged box, binary64
        dict(name="assemble_p3_41x37x40", kind="assemble", order=3, nx=41, ny=37, nz=40, dtype="f64"),
        # binary32 matrices, as the mixed solvers take them
        dict(name="assemble_p2_f32_47x50x49", kind="assemble", order=2, nx=47, ny=50, nz=49, dtype="f32"),
        # the vector P2 elasticity beam [0,4]x[0,1]^2
        dict(name="elasticity_p2_36x28x30", kind="elasticity", order=2, nx=36, ny=28, nz=30, dtype="f64"),
        # curved (P2-geometry) tetrahedra: element matrices by quadrature
        dict(name="curved_p2_32", kind="curved", order=2, nx=32, ny=32, nz=32, dtype="f64"),
        # Q2 hexahedra: element matrices by quadrature
        dict(name="hex_q2_31x32x33", kind="hex", order=2, nx=31, ny=32, nz=33, dtype="f64"),
        # one backward-Euler step's reassembly, replayed from a captured graph: A(t), b = M u, Dirichlet rows
        dict(name="heat_step_p2_48", kind="heat", order=2, nx=48, ny=48, nz=48, dtype="f64"),
        # a whole small Poisson problem: matrix, load, on(), CG + Jacobi
        dict(name="poisson_p1_16_jacobi", kind="poisson", order=1, nx=16, ny=16, nz=16, dtype="f64", method="jacobi"),
        # a whole large Poisson problem: matrix, load, on(), AMG set-up, CG + AMG
        dict(name="poisson_p2_48_gamg", kind="poisson", order=2, nx=48, ny=48, nz=48, dtype="f64", method="gamg"),
        # matrix-free P3 Poisson: double-float operator outside, binary32 CG + p-multigrid inside
        dict(name="matfree_p3_36x40x38", kind="matfree", order=3, nx=36, ny=40, nz=38, dtype="df64", method="pmg"),
        # uneven independent problems assembled together (order and size of each from `shape`)
        dict(name="batch_16", kind="batch", count=16, shape=4321, lo=8, hi=32, dtype="f64"),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, lo, hi):
    """Three cell counts, one logarithmic size with up to a fifth more or less along each axis."""
    n = _logint(rng, lo, hi)
    near = lambda: max(2, min(hi, int(round(n * rng.uniform(0.8, 1.2)))))  # noqa: E731
    return dict(nx=near(), ny=near(), nz=near())


def draw(rng):
    kind = rng.choice(["assemble", "assemble", "assemble", "elasticity", "curved", "hex", "heat", "poisson", "poisson",
                       "matfree", "batch"])
    real = rng.choice(["f64", "f64", "f32"])
    if kind == "assemble":
        order = rng.choice([1, 2, 2, 3])
        return dict(kind=kind, order=order, dtype=real, **_box(rng, 6, {1: 64, 2: 60, 3: 40}[order]))
    if kind == "elasticity":
        order = rng.choice([1, 2, 2])
        return dict(kind=kind, order=order, dtype=real, **_box(rng, 6, {1: 48, 2: 31}[order]))
    if kind == "curved":
        return dict(kind=kind, order=2, dtype=real, **_box(rng, 6, 32))
    if kind == "hex":
        order = rng.choice([1, 2, 2])
        return dict(kind=kind, order=order, dtype=real, **_box(rng, 6, {1: 40, 2: 32}[order]))
    if kind == "heat":
        return dict(kind=kind, order=rng.choice([1, 2, 2]), dtype="f64", **_box(rng, 8, 48))
    if kind == "poisson":
        order = rng.choice([1, 2, 2, 3])
        method = rng.choice(["jacobi", "mixed", "cheb_jacobi", "gamg", "gamg", "gmres_gamg"])
        return dict(kind=kind, order=order, dtype="f64", method=method, **_box(rng, 6, {1: 48, 2: 36, 3: 24}[order]))
    if kind == "matfree":
        order = rng.choice([2, 3, 3])
        method = rng.choice(["pmg", "pmg", "jacobi"])
        return dict(kind=kind, order=order, dtype="df64", method=method, **_box(rng, 8, {2: 48, 3: 36}[order]))
    lo = rng.randint(4, 12)
    return dict(kind=kind, count=rng.randint(3, 16), shape=rng.randrange(1 << 20), lo=lo, hi=lo + rng.randint(4, 20), dtype=real)


# ---------------------------------------------------------------------------
# what a program has in hand before the call
# ---------------------------------------------------------------------------


class _Device:
    """A device buffer of the library seen through the CUDA array interface; a tensor made from it holds it, and with
    it the object that owns the buffer."""

    def __init__(self, owner, ptr, n, kind):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (int(n),), "typestr": kind, "data": (int(ptr), False), "version": 2}


def _values(form):
    """The CSR values of a form as a tensor on its own buffer."""
    d = ctypes.c_void_p()
    form.env.check(form.env.lib.fgpu_matrix_values_device(form.h, ctypes.byref(d)))
    return torch.as_tensor(_Device(form, d.value, form.nnz, "<f8" if form.precision == _ffi.F64 else "<f4"), device="cuda")


def _vector(v):
    return torch.as_tensor(_Device(v, v.device_ptr().value, v.n, "<f8"), device="cuda")


def _tets(case, seed):
    """(vertices, tetrahedra) of a case: the perturbed Kuhn box; the elasticity beam is [0,4]x[0,1]^2."""
    lengths = (4.0, 1.0, 1.0) if case["kind"] == "elasticity" else (1.0, 1.0, 1.0)
    return meshgen.kuhn_box(case["nx"], case["ny"], case["nz"], lengths=lengths, perturb=0.15, seed=1234 + seed)


def _curved(case, seed):
    """A curved box with its own cell count along each axis (meshgen.curved_box takes one)."""
    xyz0, tets = meshgen.kuhn_box(case["nx"], case["ny"], case["nz"], perturb=0.1, seed=1234 + seed)
    mids = np.stack([0.5 * (xyz0[tets[:, a]] + xyz0[tets[:, b]]) for a, b in meshgen.EDGE_VERTS], axis=1)
    return meshgen.bulge_map(xyz0, 0.1), tets, meshgen.bulge_map(mids, 0.1)


def _hexes(case, seed):
    return meshgen.hex_box(case["nx"], case["ny"], case["nz"], perturb=0.15, seed=1234 + seed)


def _kappa(nt, seed):
    return meshgen.lognormal_kappa(nt, seed=5678 + seed)


def _problems(case):
    """(order, nx, ny, nz) of the problems of a batch; the shapes belong to the case, the values to the seed."""
    r = np.random.default_rng(case["shape"])
    out = []
    for _ in range(case["count"]):
        n = int(r.integers(case["lo"], case["hi"] + 1))
        out.append((int(r.integers(1, 4)), n, n, n))
    return out


def _laplace_mass(V, kappa=1.0, mass=1.0):
    u, v = V.element(), V.element()
    return fpp.integrate(fpp.elements(V.mesh), kappa * fpp.inner(fpp.gradt(u), fpp.grad(v)) + mass * (fpp.idt(u) * fpp.id(v)))


def prepare(case, seed):
    e = env()
    kind = case["kind"]
    if kind == "batch":
        forms, integrals = [], []
        for k, (order, nx, ny, nz) in enumerate(_problems(case)):
            xyz, tets = meshgen.kuhn_box(nx, ny, nz, perturb=0.15, seed=1234 + 1000 * seed + k)
            V = fpp.Pch(fpp.Mesh(xyz, tets, env=e), order)
            forms.append(fpp.form2(test=V, precision=case["dtype"]))
            integrals.append(_laplace_mass(V, _kappa(len(tets), 1000 * seed + k)))
        return dict(kind=kind, batch=fpp.Batch(forms, integrals), out=[_values(f) for f in forms], keep=forms)
    if kind == "curved":
        xyz, tets, ho = _curved(case, seed)
        M = fpp.Mesh(xyz, tets, env=e, ho=ho)
    elif kind == "hex":
        xyz, tets = _hexes(case, seed)
        M = fpp.Mesh(xyz, tets, env=e)
    else:
        xyz, tets = _tets(case, seed)
        M = fpp.Mesh(xyz, tets, env=e)
    if kind == "elasticity":
        V = fpp.Pchv(M, case["order"])
        u, v = V.element(), V.element()
        lam, mu = _lame(seed)
        a = fpp.form2(test=V, precision=case["dtype"])
        return dict(kind=kind, a=a, form=fpp.integrate(fpp.elements(M), fpp.inner(fpp.stress(u, lam, mu), fpp.grad(v))),
                    out=_values(a))
    V = fpp.Pch(M, case["order"])
    if kind in ("assemble", "curved", "hex"):
        # the coefficient lives on the device: the C-ABI takes its pointer
        a = fpp.form2(test=V, precision=case["dtype"])
        k = fpp.DeviceVector(e, len(tets))
        k.upload(_kappa(len(tets), seed))
        desc, _ = a._desc(_laplace_mass(V))
        return dict(kind=kind, a=a, desc=desc, kappa=k, out=_values(a), keep=V)
    if kind == "heat":
        dt, kappa_t = _heat(seed)
        kt = fpp.DeviceScalar(e, kappa_t)
        u, v = V.element(), V.element()
        A, Mm = fpp.form2(test=V), fpp.form2(test=V)
        Mm.assign(fpp.integrate(fpp.elements(M), fpp.idt(u) * fpp.id(v)))
        form = fpp.integrate(fpp.elements(M), fpp.idt(u) * fpp.id(v) + dt * kt * fpp.inner(fpp.gradt(u), fpp.grad(v)))
        b = fpp.DeviceVector(e, V.ndof)
        u.upload(_field(V.ndof, seed))
        bc = fpp.DirichletBC(V, V.boundary_dofs())
        A.assign(form)
        Mm.mult(u, b)
        A.apply_bc(bc, b)
        with fpp.capture(e) as g:
            A.assign(form)
            Mm.mult(u, b)
            A.apply_bc(bc, b)
        return dict(kind=kind, kt=kt, value=kappa_t, graph=g, out=[_values(A), _vector(b)], keep=(A, Mm, u, b, bc, V, form))
    if kind == "poisson":
        u, v = V.element(), V.element()
        a, l = fpp.form2(test=V), fpp.form1(test=V)
        return dict(kind=kind, a=a, l=l, u=u, mesh=M, method=case["method"],
                    form=fpp.integrate(fpp.elements(M), fpp.inner(fpp.gradt(u), fpp.grad(v))),
                    load=fpp.integrate(fpp.elements(M), fpp.cst(1.0) * fpp.id(v)), out=[_vector(u), _values(a), _vector(l.vec)])
    if kind == "matfree":
        u, v = V.element(), V.element()
        bd = V.boundary_dofs()
        form = fpp.integrate(fpp.elements(M), fpp.inner(fpp.gradt(u), fpp.grad(v)))
        op, inner = fpp.operator(V, form, precision="df64"), fpp.operator(V, form, precision="f32")
        op.set_dirichlet(bd)
        inner.set_dirichlet(bd)
        l = fpp.form1(test=V)
        l.assign(fpp.integrate(fpp.elements(M), fpp.cst(1.0) * fpp.id(v)))
        rhs = l.to_numpy()
        rhs[bd] = 0.0
        l.vec.upload(rhs)
        s = dict(kind=kind, op=op, inner=inner, l=l, u=u, method=case["method"], out=_vector(u), keep=V)
        if case["method"] == "pmg":
            P = fpp.Pch(M, 1)
            up, vp = P.element(), P.element()
            c, lc = fpp.form2(test=P), fpp.form1(test=P)
            c.assign(fpp.integrate(fpp.elements(M), fpp.inner(fpp.gradt(up), fpp.grad(vp))))
            c += fpp.on(fpp.boundaryfaces(M), rhs=lc, element=up, expr=0.0, type="elimination_symmetric")
            s.update(coarse=c, keep=(V, P, lc, up))
        return s
    raise ValueError("unknown kind %r" % kind)


def _lame(seed):
    r = np.random.default_rng(97 + seed)
    return 1.0 + 0.25 * r.random(), 0.5 + 0.25 * r.random()


def _heat(seed):
    """The step length and kappa(t) = 1 + sin(t) / 2 at the step's time."""
    r = np.random.default_rng(31 + seed)
    return 0.01, 1.0 + 0.5 * math.sin(6.0 * r.random())


def _field(n, seed):
    return np.random.default_rng(77 + seed).standard_normal(n)


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------


def run(s):
    kind = s["kind"]
    if kind in ("assemble", "curved", "hex"):
        a, e = s["a"], s["a"].env
        e.check(e.lib.fgpu_assemble_matrix_dev(e.h, a.h, s["desc"], s["kappa"].device_ptr(), 0))
    elif kind == "elasticity":
        s["a"].assign(s["form"])
    elif kind == "heat":
        s["kt"].set(s["value"])
        s["graph"].launch()
    elif kind == "poisson":
        a, l, u, m = s["a"], s["l"], s["u"], s["method"]
        a.assign(s["form"])
        l.assign(s["load"])
        nonsymmetric = m.startswith("gmres")
        a += fpp.on(fpp.boundaryfaces(s["mesh"]), rhs=l, element=u, expr=0.0,
                    type="elimination" if nonsymmetric else "elimination_symmetric")
        u.zero()
        if nonsymmetric:
            a.solve(l, u, rtol=1e-10, pc="gamg", ksp="gmres")
        elif m == "mixed":
            a.solve(l, u, rtol=1e-10, pc="jacobi", mixed=True)
        else:
            a.solve(l, u, rtol=1e-10, pc=m)
    elif kind == "matfree":
        s["u"].zero()
        if s["method"] == "pmg":
            s["op"].solve(s["l"], s["u"], rtol=1e-10, pc="pmg", inner=s["inner"], coarse=s["coarse"])
        else:
            s["op"].solve(s["l"], s["u"], rtol=1e-10, pc="jacobi", inner=s["inner"])
    else:
        s["batch"].assemble()
    return s["out"]


# ---------------------------------------------------------------------------
# bytes and operations that a pass cannot do without
# ---------------------------------------------------------------------------

# ordered pairs of nodes whose smallest common simplex is a vertex, an edge, a triangle, a tetrahedron
_PAIRS = {1: (1, 2, 0, 0), 2: (1, 7, 12, 6), 3: (1, 14, 55, 92)}
_NLOC = {1: 4, 2: 10, 3: 20}


def _counts(nx, ny, nz, order):
    """(vertices, tetrahedra, nodes, pattern entries) of the Kuhn box."""
    V = (nx + 1) * (ny + 1) * (nz + 1)
    E = nx * (ny + 1) * (nz + 1) + (nx + 1) * ny * (nz + 1) + (nx + 1) * (ny + 1) * nz
    E += nx * ny * (nz + 1) + nx * (ny + 1) * nz + (nx + 1) * ny * nz + nx * ny * nz
    T = 6 * nx * ny * nz
    F = 1 + T + E - V
    nodes = V + (order - 1) * E + (F if order == 3 else 0)
    return V, T, nodes, sum(a * b for a, b in zip(_PAIRS[order], (V, E, F, T)))


def _assembly_work(nx, ny, nz, order, size, kappa=8):
    """Coordinates, elements, dof table, coefficient and pattern read once, values written once; an entry of an
    element matrix is a sum of seven products."""
    V, T, N, nnz = _counts(nx, ny, nz, order)
    n = _NLOC[order]
    return nnz * (size + 4) + (N + 1) * 4 + V * 24 + T * (4 * n + kappa), T * (n * (n + 1) // 2) * 14


def work(case):
    kind = case["kind"]
    size = 4 if case["dtype"] == "f32" else 8
    if kind == "batch":
        each = [_assembly_work(nx, ny, nz, order, size) for order, nx, ny, nz in _problems(case)]
        return {"bytes": sum(b for b, _ in each), "flops": sum(f for _, f in each)}
    nx, ny, nz, order = case["nx"], case["ny"], case["nz"], case["order"]
    if kind == "hex":
        n1 = [order * k + 1 for k in (nx, ny, nz)]
        nnz = math.prod((3 * k + 1) if order == 1 else (8 * k + 1) for k in (nx, ny, nz))
        cells, n, q = nx * ny * nz, (order + 1) ** 3, (order + 1) ** 3
        return {"bytes": nnz * (size + 4) + (math.prod(n1) + 1) * 4 + (nx + 1) * (ny + 1) * (nz + 1) * 24 + cells * (4 * n + 8),
                "flops": cells * q * (n * (n + 1) // 2) * 8}
    V, T, N, nnz = _counts(nx, ny, nz, order)
    n = _NLOC[order]
    if kind == "elasticity":
        return {"bytes": 9 * nnz * (size + 4) + (3 * N + 1) * 4 + V * 24 + T * 4 * n, "flops": T * (n * (n + 1) // 2) * 9 * 18}
    if kind == "curved":
        q = 24
        return {"bytes": nnz * (size + 4) + (N + 1) * 4 + V * 24 + T * (4 * n + 8 + 144), "flops": T * q * (n * (n + 1) // 2) * 8}
    b, f = _assembly_work(nx, ny, nz, order, size, 8 if kind == "assemble" else 0)
    if kind == "assemble":
        return {"bytes": b, "flops": f}
    if kind == "heat":      # the assembly, M u, and the Dirichlet rows in the values just written
        return {"bytes": b + nnz * 12 + N * 25, "flops": f + 2 * nnz}
    if kind == "poisson":   # the assembly, one look at the matrix, load and solution
        return {"bytes": b + nnz * 12 + N * 24, "flops": f + 2 * nnz}
    return {"bytes": V * 24 + T * 4 * n + N * 24, "flops": T * n * n * 2}


# ---------------------------------------------------------------------------
# the results in binary64, without the framework
# ---------------------------------------------------------------------------

_EDGES = [(1, 2), (2, 0), (0, 1), (0, 3), (1, 3), (2, 3)]
_FACES = [(1, 2, 3), (0, 2, 3), (0, 1, 3), (0, 1, 2)]
_HEX_EDGES = [(0, 1), (1, 2), (2, 3), (3, 0), (1, 5), (5, 4), (4, 0), (2, 6), (6, 5), (3, 7), (7, 6), (4, 7)]
_HEX_FACES = [(0, 1, 2, 3), (0, 1, 5, 4), (1, 2, 6, 5), (2, 3, 7, 6), (3, 0, 4, 7), (4, 5, 6, 7)]
_HEX_VERTS = np.array([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1], [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]], float)


def _number(keys):
    """Ids of the entries of keys (elements x local dofs), numbered by first encounter."""
    flat = keys.reshape(-1)
    u, inv = torch.unique(flat, return_inverse=True)
    first = torch.full((len(u),), len(flat), dtype=torch.int64, device=flat.device)
    first.scatter_reduce_(0, inv, torch.arange(len(flat), device=flat.device), "amin")
    rank = torch.empty_like(first)
    rank[torch.argsort(first)] = torch.arange(len(u), device=flat.device)
    return rank[inv].reshape(keys.shape), len(u)


def _entity(c, verts):
    """A key for the entity of the given local vertices, the same in all its elements."""
    v = torch.sort(torch.stack([c[:, k] for k in verts], 1), 1).values
    key = v[:, 0]
    for k in range(1, 3 if len(verts) > 2 else len(verts)):    # three vertices name a triangle or a quadrilateral
        key = key * (1 << 20) + v[:, k]
    return key


def _dofs(cells, order):
    """(dof table, dof count): vertices, edges, faces, the interior, first encounter over (element, local dof)."""
    c = torch.as_tensor(cells, device="cuda").long()
    cols = [c[:, k] for k in range(c.shape[1])]
    hexes = c.shape[1] == 8
    if order > 1:
        edges = torch.unique(torch.stack([_entity(c, e) for e in (_HEX_EDGES if hexes else _EDGES)]), return_inverse=True)[1]
        for (a, b), ids in zip(_HEX_EDGES if hexes else _EDGES, edges):
            for l in range(order - 1):
                slot = torch.where(c[:, a] > c[:, b], order - 2 - l, l)
                cols.append((1 << 40) + ids * (order - 1) + slot)
    if order == 3 or (hexes and order == 2):
        faces = torch.unique(torch.stack([_entity(c, f) for f in (_HEX_FACES if hexes else _FACES)]), return_inverse=True)[1]
        cols += [(1 << 50) + ids for ids in faces]
    if hexes and order == 2:
        cols.append((1 << 60) + torch.arange(len(c), device="cuda"))
    return _number(torch.stack(cols, 1))


def _monomials(x, order, grad):
    """Monomials up to a degree at points x (q x 3); with grad their derivatives (q x 3 x m)."""
    p = [(a, b, s - a - b) for s in range(order + 1) for a in range(s + 1) for b in range(s + 1 - a)]
    P = lambda t, k: t ** k if k >= 0 else np.zeros_like(t)  # noqa: E731
    X, Y, Z = x.T
    if not grad:
        return np.stack([P(X, a) * P(Y, b) * P(Z, c) for a, b, c in p], 1)
    return np.stack([np.stack([a * P(X, a - 1) * P(Y, b) * P(Z, c), b * P(X, a) * P(Y, b - 1) * P(Z, c),
                               c * P(X, a) * P(Y, b) * P(Z, c - 1)], 1) for a, b, c in p], 2)


def _nodes(order):
    """Nodes of the unit tetrahedron: vertices, edge points (Gauss-Lobatto at order 3), face centroids."""
    v = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1]], float)
    t = {1: [], 2: [0.5], 3: [0.5 - 0.5 / math.sqrt(5), 0.5 + 0.5 / math.sqrt(5)]}[order]
    pts = list(v) + [v[a] + s * (v[b] - v[a]) for a, b in _EDGES for s in t]
    if order == 3:
        pts += [v[list(f)].mean(0) for f in _FACES]
    return np.array(pts)


def _basis(order, x):
    """Lagrange functions and gradients on the unit tetrahedron: (q x n), (q x 3 x n)."""
    C = np.linalg.inv(_monomials(_nodes(order), order, False))
    return _monomials(x, order, False) @ C, _monomials(x, order, True) @ C


def _duffy(k):
    """Collapsed Gauss rule of the unit tetrahedron, exact to degree 2k - 3."""
    g, w = np.polynomial.legendre.leggauss(k)
    g, w = (g + 1) / 2, w / 2
    pts, ws = [], []
    for a, wa in zip(g, w):
        for b, wb in zip(g, w):
            for c, wc in zip(g, w):
                pts.append((a, b * (1 - a), c * (1 - a) * (1 - b)))
                ws.append(wa * wb * wc * (1 - a) ** 2 * (1 - b))
    return np.array(pts), np.array(ws)


def _rule24():
    """The symmetric 24-point rule of degree 6 (three vertex orbits and one of twelve points), the rule of the
    curved P2 form; weights sum to the volume 1/6."""
    pts, w = [], []
    for a, wt in ((0.214602871259152, 0.053230333677557), (0.0406739585346115, 0.013436281407094),
                  (0.3223378901422755, 0.073809575391540)):
        for k in range(4):
            L = [a] * 4
            L[k] = 1 - 3 * a
            pts.append(L[1:])
            w.append(wt)
    a, b = 0.0636610018750175, 0.269672331458316
    for i in range(4):
        for j in range(4):
            if i != j:
                L = [a] * 4
                L[i], L[j] = b, 1 - 2 * a - b
                pts.append(L[1:])
                w.append(27 / 420)
    w = np.array(w)
    return np.array(pts), w / w.sum() / 6


def _gpu(x):
    return torch.as_tensor(np.ascontiguousarray(x), dtype=torch.float64, device="cuda")


def _frames(xyz, cells):
    """Inverse-transposed Jacobian (T x 3 x 3: B[e, physical, reference]) and |det| of the affine map from the unit
    tetrahedron, by cofactors."""
    X = _gpu(xyz)
    c = torch.as_tensor(cells, device="cuda").long()
    K = torch.stack([X[c[:, k]] - X[c[:, 0]] for k in (1, 2, 3)], 2)
    return _inverse_t(K)


def _inverse_t(K):
    k0, k1, k2 = K[..., 0], K[..., 1], K[..., 2]
    B = torch.stack([torch.linalg.cross(k1, k2), torch.linalg.cross(k2, k0), torch.linalg.cross(k0, k1)], -1)
    det = (k0 * B[..., 0]).sum(-1)
    return B / det[..., None, None], det.abs()


def _sum_entries(rows, cols, N, blocks):
    """CSR values and pattern: `blocks()` yields (element slice, T x n x n matrices); entries sorted by (row, column)."""
    n = rows.shape[1]
    key = (rows[:, :, None] * N + cols[:, None, :]).reshape(-1)
    u, inv = torch.unique(key, return_inverse=True)
    del key
    val = torch.zeros(len(u), dtype=torch.float64, device="cuda")
    for sl, K in blocks():
        val.index_add_(0, inv[sl.start * n * n:sl.stop * n * n], K.reshape(-1))
    return val, u // N, u % N


def _slices(T, step):
    return [slice(a, min(T, a + step)) for a in range(0, T, step)]


def _scalar(order, xyz, tets, l2g, N, kappa, mass):
    """Values, rows, columns of kappa grad.grad + mass on affine tetrahedra."""
    q, w = _duffy(order + 2)
    phi, dphi = _basis(order, q)
    S = _gpu(np.einsum("q,qai,qbj->abij", w, dphi, dphi))
    M = _gpu(np.einsum("q,qi,qj->ij", w, phi, phi))
    B, J = _frames(xyz, tets)
    k = J * (_gpu(kappa) if isinstance(kappa, np.ndarray) else kappa)

    def blocks():
        for sl in _slices(len(tets), 1 << 18):
            G = torch.einsum("eda,edb->eab", B[sl], B[sl]) * k[sl, None, None]
            yield sl, torch.einsum("eab,abij->eij", G, S) + mass * J[sl, None, None] * M

    return _sum_entries(l2g, l2g, N, blocks)


def _quadrature(l2g, N, X, geo, dgeo, w, phi, dphi, kappa):
    """Values of kappa grad.grad + mass on mapped cells: X (cells x g x 3), the map's functions at the points."""
    geo_, dg, W, p, dp = _gpu(geo), _gpu(dgeo), _gpu(w), _gpu(phi), _gpu(dphi)

    def blocks():
        for sl in _slices(len(X), 1 << 14):
            K = torch.einsum("egd,qag->eqda", X[sl], dg)
            B, J = _inverse_t(K)
            J = J * W
            D = torch.einsum("eqda,qai->eqdi", B, dp)
            A = torch.einsum("eqdi,eqdj->eij", D * (J * kappa[sl, None])[..., None, None], D)
            yield sl, A + torch.einsum("eq,qi,qj->eij", J, p, p)

    return _sum_entries(l2g, l2g, N, blocks)


def _boundary(cells, l2g, order):
    """Dofs on the boundary faces of a tetrahedral mesh."""
    c = torch.as_tensor(cells, device="cuda").long()
    keys = torch.stack([_entity(c, f) for f in _FACES], 1)
    _, inv, cnt = torch.unique(keys.reshape(-1), return_inverse=True, return_counts=True)
    lone = (cnt[inv] == 1).reshape(-1, 4)
    x = _nodes(order)
    bary = np.concatenate([1 - x.sum(1, keepdims=True), x], 1)
    on = torch.zeros(int(l2g.max()) + 1, dtype=torch.bool, device="cuda")
    for f in range(4):
        local = [i for i in range(len(x)) if abs(bary[i, f]) < 1e-12]      # face f lies opposite vertex f
        on[l2g[lone[:, f]][:, local].reshape(-1)] = True
    return on


def _load(order, xyz, tets, l2g, N):
    """Load vector of f = 1."""
    q, w = _duffy(order + 2)
    phi, _ = _basis(order, q)
    _, J = _frames(xyz, tets)
    out = torch.zeros(N, dtype=torch.float64, device="cuda")
    return out.index_add_(0, l2g.reshape(-1), (J[:, None] * _gpu(w @ phi)).reshape(-1))


def _solve(val, row, col, b, free):
    """Jacobi-preconditioned conjugate gradients on the free dofs (zero elsewhere), to the binary64 floor."""
    N = len(b)
    keep = free[row] & free[col]
    r_, c_, v_ = row[keep], col[keep], val[keep]
    ptr = torch.zeros(N + 1, dtype=torch.int64, device="cuda")
    ptr[1:] = torch.cumsum(torch.bincount(r_, minlength=N), 0)
    A = torch.sparse_csr_tensor(ptr, c_, v_, (N, N))
    d = torch.ones(N, dtype=torch.float64, device="cuda")
    on = r_ == c_
    d[r_[on]] = v_[on]
    x = torch.zeros_like(b)
    b = torch.where(free, b, torch.zeros_like(b))
    for _ in range(3):                          # restarted from the true residual
        r = b - A @ x
        z = r / d
        p, rz, stop = z.clone(), torch.dot(r, z), 1e-13 * float(b.norm())
        for it in range(4000):
            q = A @ p
            alpha = rz / torch.dot(p, q)
            x += alpha * p
            r -= alpha * q
            z = r / d
            new = torch.dot(r, z)
            p = z + (new / rz) * p
            rz = new
            if it % 25 == 24 and float(r.norm()) <= stop:
                break
    return x


def exact(case, seed):
    kind, order = case["kind"], case.get("order")
    if kind == "batch":
        out = []
        for k, (order, nx, ny, nz) in enumerate(_problems(case)):
            xyz, tets = meshgen.kuhn_box(nx, ny, nz, perturb=0.15, seed=1234 + 1000 * seed + k)
            l2g, N = _dofs(tets, order)
            out.append(_scalar(order, xyz, tets, l2g, N, _kappa(len(tets), 1000 * seed + k), 1.0)[0])
        return out
    if kind == "curved":
        xyz, tets, ho = _curved(case, seed)
        l2g, N = _dofs(tets, order)
        X = torch.cat([_gpu(xyz)[torch.as_tensor(tets, device="cuda").long()], _gpu(ho)], 1)
        q, w = _rule24()
        geo, dgeo = _basis(2, q)
        return _quadrature(l2g, N, X, geo, dgeo, w, *_basis(order, q), _gpu(_kappa(len(tets), seed)))[0]
    if kind == "hex":
        xyz, cells = _hexes(case, seed)
        l2g, N = _dofs(cells, order)
        g, w1 = np.polynomial.legendre.leggauss(order + 1)
        q = np.array([(a, b, c) for a in g for b in g for c in g])
        w = np.array([a * b * c for a in w1 for b in w1 for c in w1])
        v = _HEX_VERTS
        mids = [v[list(e)].mean(0) for e in _HEX_EDGES] + [v[list(f)].mean(0) for f in _HEX_FACES] + [np.zeros(3)]
        nodes = v if order == 1 else np.concatenate([v, mids])
        return _quadrature(l2g, N, _gpu(xyz)[torch.as_tensor(cells, device="cuda").long()], *_tensor(v, 1, q), w,
                           *_tensor(nodes, order, q), _gpu(_kappa(len(cells), seed)))[0]
    xyz, tets = _tets(case, seed)
    l2g, N = _dofs(tets, order)
    if kind == "assemble":
        return _scalar(order, xyz, tets, l2g, N, _kappa(len(tets), seed), 1.0)[0]
    if kind == "elasticity":
        return _elasticity(order, xyz, tets, l2g, N, *_lame(seed))
    on = _boundary(tets, l2g, order)
    if kind == "heat":
        dt, kt = _heat(seed)
        val, row, col = _scalar(order, xyz, tets, l2g, N, dt * kt, 1.0)
        mval = _scalar(order, xyz, tets, l2g, N, 0.0, 1.0)[0]
        b = torch.zeros(N, dtype=torch.float64, device="cuda").index_add_(0, row, mval * _gpu(_field(N, seed))[col])
        gone = on[row] | on[col]
        val[gone] = 0.0
        val[(row == col) & on[row]] = 1.0
        b[on] = 0.0
        return [val, b]
    val, row, col = _scalar(order, xyz, tets, l2g, N, 1.0, 0.0)
    b = _load(order, xyz, tets, l2g, N)
    x = _solve(val, row, col, b, ~on)
    if kind == "matfree":
        return x
    b[on] = 0.0
    val[on[row] if case["method"].startswith("gmres") else on[row] | on[col]] = 0.0
    val[(row == col) & on[row]] = 1.0
    return [x, val, b]


def _tensor(nodes, order, q):
    """Tensor Lagrange functions of the nodes in [-1, 1]^3 at the points: (q x n), (q x 3 x n)."""
    def one(a, t):
        if order == 1:
            return 0.5 * (1 + a * t), 0.5 * a + 0 * t
        return {-1: (0.5 * t * (t - 1), t - 0.5), 0: (1 - t * t, -2 * t), 1: (0.5 * t * (t + 1), t + 0.5)}[int(round(a))]
    phi, dphi = [], []
    for p in nodes:
        (f, df), (g, dg), (h, dh) = (one(p[k], q[:, k]) for k in range(3))
        phi.append(f * g * h)
        dphi.append(np.stack([df * g * h, f * dg * h, f * g * dh], 1))
    return np.stack(phi, 1), np.stack(dphi, 2)


def _elasticity(order, xyz, tets, l2g, N, lam, mu):
    """Values of lambda div u div v + 2 mu eps(u):eps(v), dof 3 node + component."""
    q, w = _duffy(order + 2)
    _, dphi = _basis(order, q)
    S = _gpu(np.einsum("q,qai,qbj->abij", w, dphi, dphi))
    B, J = _frames(xyz, tets)
    eye = torch.eye(3, dtype=torch.float64, device="cuda")
    n = l2g.shape[1]
    rows = (3 * l2g[:, :, None] + torch.arange(3, device="cuda")).reshape(len(tets), 3 * n)

    def blocks():
        for sl in _slices(len(tets), 1 << 15):
            Y = torch.einsum("eca,edb,abij->eicjd", B[sl], B[sl], S) * J[sl, None, None, None, None]
            tr = torch.einsum("eicjc->eij", Y)
            K = lam * Y + mu * Y.transpose(2, 4) + mu * tr[:, :, None, :, None] * eye[None, None, :, None, :]
            yield sl, K.reshape(-1, 3 * n, 3 * n)

    return _sum_entries(rows, rows, 3 * N, blocks)[0]
