"""Performance cases of the FEM path: what a program that uses this library has
it do, through its public entry points, from the smallest model to the largest.

listed() and draw(rng) give cases (dicts of plain values), prepare(case, seed)
what a program has in hand before the call, run(state) one pass with its
outputs, work(case) the bytes and operations one pass cannot do without, and
exact(case, seed) the outputs computed in FP64 with plain torch.

Kinds of case:
  solve     FemSystem.solve_mixed / solve_fast: the linear solve of an
            assembled system, the main cost of every analysis
  dropin    nb_sparse_solve_CG_precond_Jacobi called as nbots calls it, host
            vectors, on a matrix that the program keeps
  multiply  nb_sparse_multiply_vector, the same
  assemble  FemSystem.assemble + apply_bcs: K and F of a new material field
  entry     nb_fem_compute_2D_Solid_Mechanics, nbots' whole FEM call
  gradient  SimpProblem.evaluate, one step of a topology optimisation
  batch     Batch.launch and its results: many uneven designs side by side
  post      strain, stress and principal stresses of a solution
"""
import ctypes
import math

import numpy as np
import torch

from nbots_gb300 import _lib as L
from nbots_gb300 import dropin
from nbots_gb300 import workloads as W
from nbots_gb300.batch import Batch
from nbots_gb300.fem import FemSystem
from nbots_gb300.simp import SimpProblem

NU = 0.3


# ------------------------------------------------------------------- cases
def listed():
    return [
        # the smallest solve: a coarse jittered model, where launches and
        # grid-wide waits are all of the time
        dict(name="solve_64x32_mixed", kind="solve", mesh="q4", nx=64, ny=32, field="uniform",
             jitter=0.2, method="mixed", tol=1e-10, budget=0),
        # a small heterogeneous model in FP64, odd width
        dict(name="solve_127x64_fp64", kind="solve", mesh="q4", nx=127, ny=64, field="lognormal",
             jitter=0.0, method="fp64", tol=1e-10, budget=0),
        # an ordinary design model (SIMP densities), mixed precision
        dict(name="solve_512x256_mixed", kind="solve", mesh="q4", nx=512, ny=256, field="simp",
             jitter=0.0, method="mixed", tol=1e-10, budget=0),
        # the headline model: 1M dof, lognormal moduli, relative residual 1e-8
        dict(name="solve_1024x512_mixed", kind="solve", mesh="q4", nx=1024, ny=512,
             field="lognormal", jitter=0.0, method="mixed", tol=1e-8, budget=0),
        # the largest: a 2.6M-dof triangle mesh too large to keep on chip,
        # with the iteration budget a design loop gives an inexact solve
        dict(name="solve_t3_1601x802_budget", kind="solve", mesh="t3", nx=1601, ny=802,
             field="lognormal", jitter=0.2, method="mixed", tol=1e-10, budget=500),
        # nbots' own solver call on a triangle mesh, host vectors
        dict(name="dropin_cg_t3_301x150", kind="dropin", mesh="t3", nx=301, ny=150,
             field="lognormal", jitter=0.2, tol=1e-10),
        # nbots' matrix-vector product, host vectors
        dict(name="dropin_multiply_701x350", kind="multiply", mesh="q4", nx=701, ny=350,
             field="lognormal", jitter=0.1),
        # a new material field on the headline mesh: element stiffness,
        # gather, boundary conditions
        dict(name="assemble_1024x512", kind="assemble", mesh="q4", nx=1024, ny=512,
             field="lognormal", jitter=0.1),
        # nbots' FEM entry on a small model, everything in one call
        dict(name="entry_96x48", kind="entry", mesh="q4", nx=96, ny=48, jitter=0.2),
        # one optimisation step: objective and gradient of new densities
        dict(name="gradient_255x128", kind="gradient", nx=255, ny=128, method="mixed", tol=1e-10),
        # many designs of uneven size in one launch
        dict(name="batch_24", kind="batch", count=24, small=64, large=512, tol=1e-10),
        # post-processing of a solution
        dict(name="post_512x256", kind="post", mesh="q4", nx=512, ny=256, field="lognormal",
             jitter=0.1),
    ]


def _grid(rng, lo, hi):
    """A model about twice as long as high with lo to hi nodes, sizes spread
    over their logarithm; the length odd or even, the height even (the point
    load sits on its middle node)."""
    nodes = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    aspect = rng.uniform(1.2, 3.0)
    ny = max(8, 2 * int(math.sqrt(nodes / aspect) / 2))
    nx = max(12, int(nodes / (ny + 1)) - 1)
    return nx, ny


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "solve", "dropin", "multiply", "assemble",
                       "entry", "gradient", "batch", "post"])
    mesh = rng.choice(["q4", "q4", "t3"])
    field = rng.choice(["uniform", "lognormal", "simp"])
    jitter = round(rng.uniform(0.05, 0.2), 3)
    if kind == "solve":
        method = rng.choice(["mixed", "mixed", "fp64"])
        nx, ny = _grid(rng, 600, 500_000 if method == "mixed" else 150_000)
        return dict(kind=kind, mesh=mesh, nx=nx, ny=ny, field=field, jitter=jitter,
                    method=method, tol=1e-10, budget=0)
    if kind == "dropin":
        nx, ny = _grid(rng, 600, 100_000)
        return dict(kind=kind, mesh=mesh, nx=nx, ny=ny, field=field, jitter=jitter, tol=1e-10)
    if kind in ("multiply", "assemble", "post"):
        nx, ny = _grid(rng, 2_000, 500_000)
        return dict(kind=kind, mesh=mesh, nx=nx, ny=ny, field=field, jitter=jitter)
    if kind == "entry":
        nx, ny = _grid(rng, 600, 30_000)
        return dict(kind=kind, mesh=mesh, nx=nx, ny=ny, jitter=jitter)
    if kind == "gradient":
        nx, ny = _grid(rng, 2_000, 130_000)
        return dict(kind=kind, nx=nx, ny=ny, method=rng.choice(["mixed", "fp64"]), tol=1e-10)
    small = rng.choice([48, 64, 96])
    return dict(kind=kind, count=rng.randint(6, 24), small=small,
                large=rng.choice([2, 4]) * small, tol=1e-10)


# ------------------------------------------------------------------ inputs
def _field(field, n, seed):
    if field == "uniform":
        return np.ones(n)
    if field == "lognormal":
        return W.lognormal_E(n, 0.5, seed)
    rho = np.random.Generator(np.random.PCG64(seed)).uniform(0.3, 0.7, size=n)
    return W.simp_E(rho)


def _problem(case, seed):
    """A clamped plate with a point load and a top traction whose sizes come
    from the seed; triangles: every quadrilateral cut along one diagonal,
    the direction alternating."""
    r = np.random.Generator(np.random.PCG64([seed, 7]))
    nx, ny = case["nx"], case["ny"]
    p = W.cantilever_q4(nx, ny, jitter=case.get("jitter", 0.0), seed=seed, nu=NU,
                        point_load=-float(r.uniform(0.8, 1.2)),
                        top_traction=float(r.uniform(0.008, 0.012)))
    if case.get("mesh") == "t3":
        c = p.conn.astype(np.int64)
        i, j = np.meshgrid(np.arange(nx), np.arange(ny))
        up = ((i + j) % 2 == 0).ravel()[:, None]
        a = np.where(up, c[:, [0, 1, 2]], c[:, [0, 1, 3]])
        b = np.where(up, c[:, [0, 2, 3]], c[:, [1, 2, 3]])
        d = np.where(up, c[:, [0, 2]], c[:, [1, 3]])
        p.elem = "t3"
        p.conn = np.stack([a, b], 1).reshape(-1, 3).astype(np.uint32)
        p.edges = np.concatenate([p.edges, d.astype(np.uint32)])
    p.E = _field(case.get("field", "uniform"), p.n_elems, seed)
    return p


def _designs(case, seed):
    """Independent clamped plates of uneven size (small, 2 small, ... large
    elements long), random densities, one to four point loads."""
    r = np.random.Generator(np.random.PCG64([seed, 5]))
    sizes = np.random.Generator(np.random.PCG64([case["count"], case["small"]]))
    lengths = [case["small"]]
    while 2 * lengths[-1] <= case["large"]:
        lengths.append(2 * lengths[-1])
    out, rho = [], []
    for _ in range(case["count"]):
        nx = int(lengths[int(sizes.integers(0, len(lengths)))])
        ny = nx // 2
        p = W.cantilever_q4(nx, ny, point_load=0.0, nu=NU)
        p.bcs = [p.bcs[0]]
        n = int(r.integers(1, 5))
        at = r.choice(np.arange(1, ny + 1) * (nx + 1) + nx, size=n, replace=False)
        base = len(p.vtx)
        p.vtx = np.concatenate([p.vtx, at.astype(np.uint32)])
        for q in range(n):
            f = r.uniform(-1.0, 1.0, size=2)
            p.bcs.append(W.BC(W.NEUMANN, W.ON_POINT, base + q, (1, 1),
                              (float(f[0]), float(f[1]))))
        out.append(p)
        rho.append(r.uniform(0.2, 1.0, size=p.n_elems))
    return out, rho


class _View:
    """A device array of a FemSystem as a torch tensor, without a copy; it
    keeps the system, and so the memory, alive."""

    def __init__(self, system, ptr, n):
        self.system = system
        self.__cuda_array_interface__ = dict(shape=(n,), typestr="<f8", data=(ptr, False),
                                             version=2)


def _tensor(s, what):
    view = _View(s, s.dptr(what), s.lib.nbg_fem_bytes(s.handle, what) // 8)
    t = torch.as_tensor(view, device="cuda")
    t.system = s
    return t


class _Matrix:
    """An nbots matrix that a program keeps, destroyed with its owner."""

    def __init__(self, p):
        s = FemSystem(p)
        L.check(s.assemble(), "assemble")
        s.apply_bcs()
        self.F = s.get(L.FEM_F)
        self.A, self.keep = dropin.sparse_from_csr(p, s.get(L.FEM_K))
        s.close()

    def __del__(self):
        dropin.libs()[0].nb_sparse_destroy(self.A)


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case)
    if kind == "batch":
        probs, rho = _designs(case, seed)
        b = Batch(probs)
        b.assemble_simp(rho, NU)
        b.setup(max_iter=40000, tol=case["tol"])
        st["batch"] = b
        return st
    p = _problem(case, seed)
    if kind == "entry":
        st["objects"] = dropin.NbotsObjects(p)
    elif kind == "gradient":
        st["rho"] = np.random.Generator(np.random.PCG64(seed)).uniform(0.3, 0.7, size=p.n_elems)
        method = L.METHOD_MIXED if case["method"] == "mixed" else L.METHOD_FP64
        st["simp"] = SimpProblem(p, method=method, tol=case["tol"])
    elif kind in ("dropin", "multiply"):
        st["matrix"] = m = _Matrix(p)
        n = m.F.shape[0]
        r = np.random.Generator(np.random.PCG64([seed, 9]))
        st["in"] = r.standard_normal(n) if kind == "multiply" else m.F
        st["out"] = np.zeros(n)
    else:
        st["system"] = s = FemSystem(p)
        if kind == "post":
            L.check(s.assemble(), "assemble")
            r = np.random.Generator(np.random.PCG64([seed, 9]))
            s.put(L.FEM_U, 1e-3 * r.standard_normal(s.N))
        elif kind == "solve":
            L.check(s.assemble(), "assemble")
            s.apply_bcs()
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "solve":
        s = st["system"]
        solve = s.solve_mixed if case["method"] == "mixed" else s.solve_fast
        solve(max_iter=case["budget"] or None, tol=case["tol"])
        return s.get(L.FEM_U)
    if kind == "dropin":
        G = dropin.libs()[0]
        x = st["out"]
        x[:] = 0.0
        n = x.shape[0]
        it, reached = ctypes.c_uint32(), ctypes.c_double()
        G.nb_sparse_solve_CG_precond_Jacobi(st["matrix"].A, st["in"].ctypes.data, x.ctypes.data,
                                            n, case["tol"], ctypes.byref(it),
                                            ctypes.byref(reached), 1)
        return x
    if kind == "multiply":
        G = dropin.libs()[0]
        G.nb_sparse_multiply_vector(st["matrix"].A, st["in"].ctypes.data, st["out"].ctypes.data, 1)
        return st["out"]
    if kind == "assemble":
        s = st["system"]
        L.check(s.assemble(), "assemble")
        s.apply_bcs()
        return {"K": _tensor(s, L.FEM_K), "F": _tensor(s, L.FEM_F)}
    if kind == "entry":
        _, u, strain = st["objects"].fem()
        return {"u": u, "strain": strain}
    if kind == "gradient":
        J, dJ, _ = st["simp"].evaluate(st["rho"])
        return {"J": J, "dJ": dJ}
    if kind == "batch":
        b = st["batch"]
        b.launch()
        _, J = b.results()
        return {"J": J, "u": np.concatenate(b.displacements()),
                "dJ": np.concatenate(b.sensitivities())}
    s = st["system"]
    # the device arrays, as a program that goes on with them there takes them
    lib = s.lib
    L.check(lib.nbg_fem_strain(s.handle), "strain")
    L.check(lib.nbg_fem_stress(s.handle), "stress")
    L.check(lib.nbg_fem_main_stress(s.handle), "main_stress")
    return {"strain": _tensor(s, L.FEM_STRAIN), "stress": _tensor(s, L.FEM_STRESS),
            "main": _tensor(s, L.FEM_MAIN_STRESS)}


# -------------------------------------------------------------------- work
def work(case):
    """Bytes: matrix, mesh and vectors once.  Operations of a solve: those of
    the iterations that Jacobi-preconditioned CG takes on such a plate, in
    proportion to its length in elements."""
    kind = case["kind"]

    def solve(nx, ny, t3, per_length, budget=0):
        n = 2 * (nx + 1) * (ny + 1)
        nnz = n * (14 if t3 else 18)
        its = min(per_length * nx, budget or 1e18)
        return 8 * nnz + 4 * nnz // 4 + 16 * n, its * (2 * nnz + 12 * n)

    if kind == "batch":
        sizes = np.random.Generator(np.random.PCG64([case["count"], case["small"]]))
        lengths = [case["small"]]
        while 2 * lengths[-1] <= case["large"]:
            lengths.append(2 * lengths[-1])
        pick = [int(lengths[int(sizes.integers(0, len(lengths)))]) for _ in range(case["count"])]
        w = [solve(nx, nx // 2, False, 9) for nx in pick]
        return {"bytes": sum(x[0] for x in w), "flops": sum(x[1] for x in w)}
    nx, ny, t3 = case["nx"], case["ny"], case.get("mesh") == "t3"
    nodes, quads = (nx + 1) * (ny + 1), nx * ny
    n, nnz = 2 * nodes, 2 * nodes * (14 if t3 else 18)
    elems, nen, ngp = (2 * quads, 3, 1) if t3 else (quads, 4, 4)
    mesh = 16 * nodes + 4 * nen * elems + 8 * elems
    if kind in ("solve", "dropin"):
        b, f = solve(nx, ny, t3, 8, case.get("budget", 0))
        return {"bytes": b, "flops": f}
    if kind == "multiply":
        return {"bytes": 12 * nnz + 20 * n, "flops": 2 * nnz}
    if kind == "assemble":
        return {"bytes": mesh + 4 * nnz + 8 * nnz + 12 * n, "flops": elems * ngp * (8 if t3 else 400)}
    if kind == "post":
        return {"bytes": mesh + 8 * n + 8 * (3 + 3 + 2) * ngp * elems, "flops": elems * ngp * 90}
    b, f = solve(nx, ny, t3, 8)
    if kind == "entry":
        return {"bytes": mesh + b + 24 * ngp * elems, "flops": f}
    return {"bytes": mesh + b + 16 * elems, "flops": f}


# ------------------------------------------------------------------- exact
# nbots' shape-function derivatives at the Gauss points, 12 digits: they
# define the discrete problem
_D, _E = 0.394337567297, 0.105662432703
_PSI4 = [[-_D, -_D, -_E, -_E], [_D, _D, _E, _E], [_E, _E, _D, _D], [-_E, -_E, -_D, -_D]]
_ETA4 = [[-_D, -_E, -_E, -_D], [-_E, -_D, -_D, -_E], [_E, _D, _D, _E], [_D, _E, _E, _D]]


def _b_matrices(p):
    """(dx, dy, detJ * weight) per element and Gauss point: derivatives
    [e, node, gp], in FP64 on the GPU."""
    nod = torch.from_numpy(np.ascontiguousarray(p.nod)).cuda()
    conn = torch.from_numpy(p.conn.astype(np.int64)).cuda()
    if conn.shape[1] == 4:
        ps = torch.tensor(_PSI4, dtype=torch.float64, device="cuda")
        et = torch.tensor(_ETA4, dtype=torch.float64, device="cuda")
        w = 1.0
    else:
        ps = torch.tensor([[-1.0], [1.0], [0.0]], dtype=torch.float64, device="cuda")
        et = torch.tensor([[-1.0], [0.0], [1.0]], dtype=torch.float64, device="cuda")
        w = 0.5
    x, y = nod[conn, 0], nod[conn, 1]
    xp, xe, yp, ye = x @ ps, x @ et, y @ ps, y @ et
    det = xp * ye - yp * xe
    dx = (ye[:, None] * ps - yp[:, None] * et) / det[:, None]
    dy = (-xe[:, None] * ps + xp[:, None] * et) / det[:, None]
    return conn, dx, dy, det * w * p.thickness


def _elasticity(E):
    d0 = E / (1.0 - NU * NU)
    return d0, NU * d0, E / (2.0 * (1.0 + NU))


def _element_stiffness(p, E):
    """[e, 2 nen, 2 nen] for moduli E."""
    conn, dx, dy, w = _b_matrices(p)
    d0, d1, d3 = (v[:, None, None] for v in _elasticity(E))
    xx = torch.einsum("eig,ejg,eg->eij", dx, dx, w)
    yy = torch.einsum("eig,ejg,eg->eij", dy, dy, w)
    xy = torch.einsum("eig,ejg,eg->eij", dx, dy, w)
    nen = conn.shape[1]
    ke = torch.empty(conn.shape[0], nen, 2, nen, 2, dtype=torch.float64, device="cuda")
    ke[:, :, 0, :, 0] = d0 * xx + d3 * yy
    ke[:, :, 1, :, 1] = d0 * yy + d3 * xx
    ke[:, :, 0, :, 1] = d1 * xy + d3 * xy.transpose(1, 2)
    ke[:, :, 1, :, 0] = d1 * xy.transpose(1, 2) + d3 * xy
    dofs = torch.stack([2 * conn, 2 * conn + 1], 2).reshape(conn.shape[0], -1)
    return dofs, ke.reshape(conn.shape[0], 2 * nen, 2 * nen)


def _loads(p):
    """F of the Neumann conditions and the clamped dofs (all values zero)."""
    F = np.zeros(p.n_dof)
    fixed = np.zeros(p.n_dof, bool)
    for b in p.bcs:
        nodes = p.sgm[b.id].astype(np.int64) if b.where == W.ON_SEGMENT else None
        if b.kind == W.DIRICHLET:
            for j in range(2):
                if b.mask[j]:
                    fixed[2 * nodes + j] = True
        elif b.where == W.ON_POINT:
            for j in range(2):
                if b.mask[j]:
                    F[2 * int(p.vtx[b.id]) + j] += b.val[j]
        else:
            x = p.nod[nodes]
            share = np.linalg.norm(np.diff(x, axis=0), axis=1) / np.linalg.norm(x[-1] - x[0])
            for j in range(2):
                if b.mask[j]:
                    np.add.at(F, 2 * nodes[:-1] + j, 0.5 * share * b.val[j])
                    np.add.at(F, 2 * nodes[1:] + j, 0.5 * share * b.val[j])
    F[fixed] = 0.0
    return torch.from_numpy(F).cuda(), torch.from_numpy(fixed).cuda()


def _solve(p, nx, ny, E):
    """The displacements: block Cholesky along the length of the grid, one
    block per column of nodes."""
    dofs, ke = _element_stiffness(p, E)
    F, fixed = _loads(p)
    m, cols = 2 * (ny + 1), nx + 1
    free = (~fixed).to(torch.float64)
    ke = ke * free[dofs][:, :, None] * free[dofs][:, None, :]
    node = dofs // 2
    col, at = node % cols, 2 * (node // cols) + dofs % 2
    D = torch.zeros(cols * m * m, dtype=torch.float64, device="cuda")
    U = torch.zeros((cols - 1) * m * m, dtype=torch.float64, device="cuda")
    row_c, col_c = col[:, :, None].expand_as(ke), col[:, None, :].expand_as(ke)
    flat = (row_c * m + at[:, :, None]) * m + at[:, None, :]
    same, right = row_c == col_c, col_c == row_c + 1
    D.index_put_((flat[same],), ke[same], accumulate=True)
    U.index_put_((flat[right],), ke[right], accumulate=True)
    D, U = D.view(cols, m, m), U.view(cols - 1, m, m)
    i = torch.nonzero(fixed)[:, 0]
    D[(i // 2) % cols, 2 * ((i // 2) // cols) + i % 2,
      2 * ((i // 2) // cols) + i % 2] = 1.0
    # F by columns of nodes
    g = F.view(ny + 1, cols, 2).permute(1, 0, 2).reshape(cols, m, 1).clone()
    for c in range(cols):
        D[c] = torch.linalg.cholesky(D[c])
        g[c] = torch.linalg.solve_triangular(D[c], g[c], upper=False)
        if c + 1 < cols:
            U[c] = torch.linalg.solve_triangular(D[c], U[c], upper=False)
            D[c + 1] -= U[c].T @ U[c]
            g[c + 1] -= U[c].T @ g[c]
    for c in range(cols - 1, -1, -1):
        if c + 1 < cols:
            g[c] -= U[c] @ g[c + 1]
        g[c] = torch.linalg.solve_triangular(D[c].T, g[c], upper=True)
    return g.view(cols, ny + 1, 2).permute(1, 0, 2).reshape(-1), F


def _strain(p, u):
    conn, dx, dy, _ = _b_matrices(p)
    ux, uy = u[2 * conn], u[2 * conn + 1]
    s = torch.stack([torch.einsum("eig,ei->eg", dx, ux), torch.einsum("eig,ei->eg", dy, uy),
                     torch.einsum("eig,ei->eg", dy, ux) + torch.einsum("eig,ei->eg", dx, uy)], 2)
    return s


def _energy_gradient(p, rho, u):
    """dJ/drho of the compliance with E = Emin + rho^3 (E0 - Emin)."""
    dofs, ke = _element_stiffness(p, torch.ones_like(rho))
    ue = u[dofs]
    return -3.0 * rho ** 2 * (1.0 - 1e-9) * torch.einsum("ei,eij,ej->e", ue, ke, ue)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        probs, rho = _designs(case, seed)
        J, us, dJ = [], [], []
        for p, r in zip(probs, rho):
            r = torch.from_numpy(r).cuda()
            nx, ny = p.meta["nx"], p.meta["ny"]
            u, F = _solve(p, nx, ny, 1e-9 + r ** 3 * (1.0 - 1e-9))
            J.append(float(F @ u))
            us.append(u)
            dJ.append(_energy_gradient(p, r, u))
        return {"J": np.array(J), "u": torch.cat(us).cpu().numpy(),
                "dJ": torch.cat(dJ).cpu().numpy()}
    if kind == "solve" and case["budget"]:
        return None  # an iterate on the way, not a solution
    p = _problem(case, seed)
    E = torch.from_numpy(p.E).cuda()
    nx, ny = case["nx"], case["ny"]
    if kind in ("solve", "dropin"):
        return _solve(p, nx, ny, E)[0].cpu().numpy()
    if kind == "entry":
        u, _ = _solve(p, nx, ny, E)
        return {"u": u.cpu().numpy(), "strain": _strain(p, u).reshape(-1).cpu().numpy()}
    if kind == "gradient":
        rho = torch.from_numpy(np.random.Generator(np.random.PCG64(seed)).uniform(
            0.3, 0.7, size=p.n_elems)).cuda()
        u, F = _solve(p, nx, ny, 1e-9 + rho ** 3 * (1.0 - 1e-9))
        return {"J": float(F @ u), "dJ": _energy_gradient(p, rho, u).cpu().numpy()}
    if kind == "post":
        r = np.random.Generator(np.random.PCG64([seed, 9]))
        s = _strain(p, torch.from_numpy(1e-3 * r.standard_normal(p.n_dof)).cuda())
        d0, d1, d3 = (v[:, None] for v in _elasticity(E))
        t = torch.stack([d0 * s[..., 0] + d1 * s[..., 1], d1 * s[..., 0] + d0 * s[..., 1],
                         d3 * s[..., 2]], 2)
        avg = 0.5 * (t[..., 0] + t[..., 1])
        rad = torch.sqrt(0.25 * (t[..., 0] - t[..., 1]) ** 2 + t[..., 2] ** 2)
        return {"strain": s.reshape(-1), "stress": t.reshape(-1),
                "main": torch.stack([avg + rad, avg - rad], 2).reshape(-1)}
    dofs, ke = _element_stiffness(p, E)
    F, fixed = _loads(p)
    free = (~fixed).to(torch.float64)
    ke = ke * free[dofs][:, :, None] * free[dofs][:, None, :]
    if kind == "multiply":
        x = torch.from_numpy(np.random.Generator(np.random.PCG64([seed, 9])).standard_normal(
            p.n_dof)).cuda()
        y = torch.where(fixed, x, torch.zeros_like(x))
        y.index_add_(0, dofs.reshape(-1), torch.einsum("eij,ej->ei", ke, x[dofs]).reshape(-1))
        return y.cpu().numpy()
    # assemble: the entries of K in row order, those of a row by column
    n = p.n_dof
    key = (dofs[:, :, None] * n + dofs[:, None, :]).reshape(-1)
    key, at = torch.unique(key, return_inverse=True)
    K = torch.zeros(key.shape[0], dtype=torch.float64, device="cuda")
    K.index_add_(0, at, ke.reshape(-1))
    row, col = key // n, key % n
    K[(row == col) & fixed[row]] = 1.0
    return {"K": K, "F": F}
