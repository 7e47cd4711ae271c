"""The work a host program has this package do, as measurable cases.

A simulation evaluates energies (line search), gradients and Hessians of one mesh at
many displacements, projects and reduces the Hessian to a Newton system, solves it with
conjugate gradients or the sparse Cholesky, and in an optimisation loop pulls an
adjoint back to the displacement, the material and the rest shape.  Each case is one such
call (or the few calls of one step) on the synthetic meshes of ``polyfem_b200.mesh``:
the cubes of the benchmark workloads and the tests, at their sizes and at odd ones.

A case's values:
  kind       energy | value_gradient | hessian | projected | cg | direct | newton | adjoint | form_host
  element    P1 | P2 | Q1;  grid: cells per axis (6 tetrahedra or 1 hexahedron per cell)
  precision  fp64 | fp32 | split32 (the modes of the NeoHookean formulation)
  material   a formulation name of NeoHookeanAssembler.set_material
  numbering  first_touch (PolyFEM's own numbering) | random (elements and nodes shuffled,
             as an external mesher leaves them)

``exact`` restates the same quantities with torch in 64 bits from the energy density alone
(derivatives by torch's automatic differentiation, eigenvalues by torch.linalg, linear
systems by an unblocked conjugate gradient run to rounding).
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from polyfem_b200 import ConjugateGradient, DirectSolver, ElasticForm, NeoHookeanAssembler
from polyfem_b200 import mesh as M
from polyfem_b200.autograd import elastic_force

ELEMENTS = {"P1": M.P1_TET, "P2": M.P2_TET, "Q1": M.Q1_HEX}
SOLVE_TOL = 1e-12  # relative residual of the iterative solves: a linear problem solved to working accuracy


def _case(name, kind, element, grid, precision="fp64", material="NeoHookean", numbering="first_touch"):
    return {"name": name, "kind": kind, "element": element, "grid": grid, "precision": precision,
            "material": material, "numbering": numbering}


def listed():
    return [
        # one line-search evaluation on a small part: a call that is all latency
        _case("energy_p1_8", "energy", "P1", 8),
        # value and first derivative of a Newton iterate on the 663,552-tetrahedron cube
        _case("value_gradient_p1_48", "value_gradient", "P1", 48),
        # the same on jittered hexahedra in the mixed FP32 mode, an odd size
        _case("value_gradient_q1_63_fp32", "value_gradient", "Q1", 63, precision="fp32"),
        # the headline workload: the Hessian of the 384,000-element P2 cube, split precision
        _case("hessian_p2_40_split32", "hessian", "P2", 40, precision="split32"),
        # a large FP64 Hessian of distorted hexahedra
        _case("hessian_q1_64", "hessian", "Q1", 64),
        # another formulation, on a mesh with no locality left in its numbering
        _case("hessian_mooney_p2_21", "hessian", "P2", 21, material="MooneyRivlin", numbering="random"),
        # the Newton system: reduced gradient and projected, reduced Hessian
        _case("projected_p2_24", "projected", "P2", 24),
        # the iterative linear solve of that system
        _case("cg_p2_24", "cg", "P2", 24),
        # the direct linear solve of that system: factorisation and one right-hand side
        _case("direct_p2_24", "direct", "P2", 24),
        # one whole Newton step of a small part, as an interactive simulation takes it
        _case("newton_p1_13", "newton", "P1", 13),
        # forward and backward through the differentiable force (shape and material optimisation)
        _case("adjoint_p2_32", "adjoint", "P2", 32),
        # the form as a host program holds it: numpy in, value, gradient and scipy Hessian out
        _case("form_host_p1_20", "form_host", "P1", 20),
    ]


# largest grids of each kind: no drawn case costs more than the largest listed one
_MAX_GRID = {
    "energy": {"P1": 48, "P2": 40, "Q1": 64},
    "value_gradient": {"P1": 48, "P2": 40, "Q1": 64},
    "hessian": {"P1": 48, "P2": 36, "Q1": 64},
    "projected": {"P1": 40, "P2": 26, "Q1": 48},
    "cg": {"P1": 36, "P2": 22, "Q1": 40},
    "direct": {"P1": 36, "P2": 20, "Q1": 34},
    "newton": {"P1": 24, "P2": 11, "Q1": 22},
    "adjoint": {"P1": 44, "P2": 32, "Q1": 44},
    "form_host": {"P1": 22, "P2": 9, "Q1": 18},
}
_MIN_GRID = {"P1": 4, "P2": 3, "Q1": 4}


def draw(rng):
    kind = rng.choice(list(_MAX_GRID))
    element = rng.choice(list(ELEMENTS))
    lo, hi = _MIN_GRID[element], _MAX_GRID[kind][element]
    grid = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    precision, material = "fp64", "NeoHookean"
    if kind in ("energy", "value_gradient"):
        precision = rng.choice(["fp64", "fp64", "fp32"])
    if kind == "hessian":
        precision = rng.choice(["fp64", "fp64", "split32"])
    if precision == "fp64" and kind in ("energy", "value_gradient", "hessian", "projected"):
        material = rng.choice(["NeoHookean", "NeoHookean", "MooneyRivlin", "SaintVenant", "IsochoricNeoHookean"])
    numbering = rng.choice(["first_touch", "first_touch", "random"])
    return {k: v for k, v in _case("", kind, element, grid, precision, material, numbering).items() if k != "name"}


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=4)
def _topology(element, grid):
    return M.structured_hex_mesh(grid) if element == "Q1" else M.structured_tet_mesh(grid, 1 if element == "P1" else 2)


class _Inputs:
    """Mesh arrays (host), and u, adjoint (host), of one case and seed."""

    def __init__(self, case, seed):
        rng = np.random.default_rng([int(seed), 41])
        mesh = _topology(case["element"], case["grid"])
        self.element, self.h = case["element"], mesh.h
        self.conn, self.gconn = mesh.conn, mesh.gconn
        self.iso = mesh.gconn is mesh.conn
        self.n_nodes = mesh.n_nodes
        E = self.n_elements = mesh.n_elements
        # interior geometric nodes move by up to a tenth of a cell, as the jittered workloads do
        inside = np.all((mesh.X > 1e-9) & (mesh.X < 1 - 1e-9), axis=1)
        self.X = mesh.X + (0.1 * mesh.h) * rng.uniform(-1, 1, mesh.X.shape) * inside[:, None]
        self.mu = np.exp(rng.normal(np.log(3.7e4), 0.3, E))
        self.lam = self.mu * (2 * 0.35) / (1 - 2 * 0.35)
        self.params = 1e5 * rng.uniform(0.5, 1.5, (3, E)) if case["material"] == "MooneyRivlin" else None
        u = 0.02 * mesh.h * rng.standard_normal((mesh.n_nodes, 3))
        if self.element == "Q1":  # the smooth field of the hexahedral workload
            u = 0.05 * np.sin(2 * np.pi * mesh.node_pos[:, :1]) + 0.25 * u
        p = rng.standard_normal((mesh.n_nodes, 3))
        clamped = mesh.node_pos[:, 0] < 1e-9
        if case["numbering"] == "random":
            pe, pn = rng.permutation(E), rng.permutation(mesh.n_nodes)
            self.conn = pn[mesh.conn[pe]].astype(np.int32)
            back = np.argsort(pn)
            u, p, clamped = u[back], p[back], clamped[back]
            pg = pn if self.iso else rng.permutation(self.X.shape[0])
            self.gconn = self.conn if self.iso else pg[mesh.gconn[pe]].astype(np.int32)
            self.X = self.X[np.argsort(pg)]
        self.u, self.p = u.reshape(-1), p.reshape(-1)
        # the x = 0 face is clamped in the Newton systems
        self.fixed = (3 * np.flatnonzero(clamped)[:, None] + np.arange(3)).ravel()


def _cuda(x):
    return torch.as_tensor(np.ascontiguousarray(x)).cuda()


def prepare(case, seed):
    inp = _Inputs(case, seed)
    kind = case["kind"]
    asm = NeoHookeanAssembler(ELEMENTS[inp.element], inp.conn, inp.X, inp.lam, inp.mu, n_nodes=inp.n_nodes,
                              gconn=None if inp.iso else inp.gconn)
    if case["material"] != "NeoHookean":
        params = {} if inp.params is None else dict(zip(("c1", "c2", "k"), inp.params))
        asm.set_material(case["material"], **params)
    state = {"kind": kind, "precision": case["precision"], "asm": asm}
    if kind == "form_host":
        state.update(form=ElasticForm(asm), u=inp.u)
        return state
    state["u"] = _cuda(inp.u)
    if kind == "value_gradient":
        state["form"] = ElasticForm(asm, case["precision"])
    if kind == "hessian":
        asm.hessian_nnz()
    if kind == "adjoint":
        asm.hessian_nnz()
        for name in ("lam", "mu", "X"):
            state[name] = _cuda(getattr(inp, name)).requires_grad_(True)
        state["u"].requires_grad_(True)
        state["p"] = _cuda(inp.p)
    if kind in ("projected", "cg", "direct", "newton"):
        asm.set_dirichlet(inp.fixed)
    if kind in ("cg", "direct"):
        state["values"] = asm.assemble_hessian_reduced_values(state["u"], project_to_psd=True)
        state["b"] = -asm.assemble_gradient_reduced(state["u"])
    if kind in ("cg", "newton"):
        solver = state["solver"] = ConjugateGradient(asm, "reduced")
        solver.set_parameters({"tolerance": SOLVE_TOL, "max_iter": 20000})
    if kind == "direct":
        solver = state["solver"] = DirectSolver(asm, "reduced")
        solver.analyze_pattern()
    return state


# ------------------------------------------------------------------ one pass
def run(state):
    kind, asm, u = state["kind"], state["asm"], state["u"]
    if kind == "energy":
        return asm.assemble_energy(u, state["precision"])
    if kind == "value_gradient":
        form = state["form"]
        return form.value(u), form.first_derivative(u)
    if kind == "hessian":
        return asm.assemble_hessian_values(u, state["precision"])
    if kind == "projected":
        return (asm.assemble_gradient_reduced(u), asm.assemble_hessian_reduced_values(u, project_to_psd=True))
    if kind in ("cg", "direct"):
        solver = state["solver"]
        solver.factorize(state["values"])
        return solver.solve(state["b"])
    if kind == "newton":
        solver = state["solver"]
        grad = asm.assemble_gradient_reduced(u)
        solver.factorize(asm.assemble_hessian_reduced_values(u, project_to_psd=True))
        return asm.reduced_to_full(solver.solve(-grad))
    if kind == "adjoint":
        inputs = (u, state["lam"], state["mu"], state["X"])
        force = elastic_force(*inputs, asm, state["precision"])
        return (force.detach(),) + torch.autograd.grad(force, inputs, state["p"])
    # form_host
    form = state["form"]
    H = form.second_derivative(u)
    return form.value(u), form.first_derivative(u), H.data, H.indices, H.indptr


# ------------------------------------------------------------------ the work of a pass
def _sizes(case):
    """Elements, FE nodes, geometric nodes, nodes and geometric nodes per element, nonzeros."""
    g, el = case["grid"], case["element"]
    v = (g + 1) ** 3
    if el == "Q1":
        return g ** 3, v, v, 8, 8, 9 * (3 * g + 1) ** 3
    edges = 3 * g * (g + 1) ** 2 + 3 * g * g * (g + 1) + g ** 3
    if el == "P1":
        return 6 * g ** 3, v, v, 4, 4, 9 * (v + 2 * edges)
    E, N = 6 * g ** 3, (2 * g + 1) ** 3
    # node pairs that share a tetrahedron: 45 in each, counted once per pair; those of a
    # face's six nodes (15) are shared by two tetrahedra, those of an edge (3) by the edge's
    faces = 12 * g ** 3 + 6 * g * g
    pairs = edges * 3 + faces * (15 - 9) + E * (45 - 4 * (15 - 9) - 6 * 3)
    return E, N, v, 10, 4, 9 * (N + 2 * pairs)


def work(case):
    E, N, Ng, n, ng, nnz = _sizes(case)
    kind, g = case["kind"], case["grid"]
    nq = {"P1": 1, "P2": 4, "Q1": 8}[case["element"]]
    mesh_bytes = E * (n * 4 + (0 if n == ng else ng * 4) + 16) + Ng * 24 + N * 24
    kin = E * nq * (6.0 * ng * 3 + 6.0 * n * 3 + 250)  # J, grad u, their determinants and inverses
    blocks = E * nq * (n * (n + 1) / 2) * 48.0
    order = 2 if case["element"] == "P2" else 1
    iters = 2.5 * -math.log10(SOLVE_TOL) * order * g  # what the Jacobi preconditioner takes on such cubes
    if kind == "energy":
        return {"bytes": mesh_bytes + 8, "flops": kin}
    if kind == "value_gradient":
        return {"bytes": 2 * mesh_bytes + N * 24 + 8, "flops": 2 * kin + E * nq * 18.0 * n}
    if kind == "hessian":
        return {"bytes": mesh_bytes + nnz * 8, "flops": kin + blocks}
    if kind == "projected":
        return {"bytes": 2 * mesh_bytes + nnz * 8 + N * 24, "flops": 2 * kin + blocks + E * 4.0 / 3 * (3 * n) ** 3}
    if kind == "cg":
        return {"bytes": iters * (nnz * 8.0 + nnz / 9 * 4.0 + N * 24 * 10), "flops": iters * nnz * 2.0}
    if kind == "newton":
        return {"bytes": iters * (nnz * 8.0 + nnz / 9 * 4.0 + N * 24 * 10) + 2 * mesh_bytes,
                "flops": iters * nnz * 2.0 + kin + blocks}
    if kind == "direct":
        # nested dissection of a cube: the last separator is a plane of m dofs, whose
        # Cholesky is m^3 / 3 operations and about a sixth of the whole factorisation
        m = 3.0 * (order * g + 1) ** 2
        return {"bytes": nnz * 8 + N * 48, "flops": 2 * m ** 3}
    if kind == "adjoint":
        return {"bytes": 5 * mesh_bytes + 4 * N * 24 + E * 16 + Ng * 24, "flops": 6 * kin}
    return {"bytes": 3 * mesh_bytes + nnz * 12 + N * 24 + 8, "flops": 3 * kin + blocks}


# ------------------------------------------------------------------ the same in 64 bits with torch
def _reference_basis(element):
    """(FE gradients [q, n, 3], geometric gradients [q, n_g, 3], weights [q]) on the reference element."""
    p1 = np.array([[-1.0, -1, -1], [1, 0, 0], [0, 1, 0], [0, 0, 1]])
    if element == "P1":
        return p1[None], p1[None], np.array([1 / 6])
    if element == "P2":
        a, b = 0.13819660112501053, 0.5854101966249684
        pts = np.array([[a, a, b], [a, b, a], [b, a, a], [a, a, a]])
        grads = []
        for x in pts:
            L = np.array([1 - x.sum(), *x])
            vert = [(4 * L[i] - 1) * p1[i] for i in range(4)]
            edge = [4 * (L[i] * p1[j] + L[j] * p1[i]) for i, j in M.TET_EDGES]
            grads.append(np.stack(vert + edge))
        return np.stack(grads), np.repeat(p1[None], 4, 0), np.full(4, 1 / 24)
    s = 0.5 - 0.5 / math.sqrt(3)
    grads = []
    for q in range(8):
        x = np.array([s if (q >> d) & 1 == 0 else 1 - s for d in range(3)])
        c = np.array(M.HEX_CORNERS)
        f, df = np.where(c == 1, x, 1 - x), np.where(c == 1, 1.0, -1.0)
        grads.append(np.stack([df[:, 0] * f[:, 1] * f[:, 2], f[:, 0] * df[:, 1] * f[:, 2],
                               f[:, 0] * f[:, 1] * df[:, 2]], axis=1))
    return np.stack(grads), np.stack(grads), np.full(8, 1 / 8)


def _det(F):
    return (F[..., 0, :] * torch.linalg.cross(F[..., 1, :], F[..., 2, :], dim=-1)).sum(-1)


def _psi(material, F, prm):
    """Energy density at F [..., 3, 3]; prm: the element's parameters, broadcastable."""
    I3 = torch.eye(3, dtype=F.dtype, device=F.device)
    I1 = (F * F).sum((-1, -2))
    if material == "SaintVenant":
        G = 0.5 * (F.transpose(-1, -2) @ F - I3)
        return 0.5 * prm[0] * (G * I3).sum((-1, -2)) ** 2 + prm[1] * (G * G).sum((-1, -2))
    J = _det(F)
    if material == "NeoHookean":
        lj = torch.log(J)
        return 0.5 * prm[1] * (I1 - 3 - 2 * lj) + 0.5 * prm[0] * lj ** 2
    if material == "IsochoricNeoHookean":
        return 0.5 * prm[1] * (I1 * J ** (-2 / 3) - 3)
    C = F @ F.transpose(-1, -2)  # MooneyRivlin
    I2 = 0.5 * (I1 ** 2 - (C * C).sum((-1, -2)))
    return (prm[0] * (I1 * J ** (-2 / 3) - 3) + prm[1] * (I2 * J ** (-4 / 3) - 3) + 0.5 * prm[2] * torch.log(J) ** 2)


class _Exact:
    """The case's quantities from its inputs, in float64."""

    def __init__(self, case, seed):
        self.inp = inp = _Inputs(case, seed)
        self.material = case["material"]
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda x: torch.as_tensor(np.ascontiguousarray(x)).to(self.dev)
        self.conn, self.gconn = t(inp.conn).long(), t(inp.gconn).long()
        self.g, self.gg, self.w = (t(x) for x in _reference_basis(inp.element))
        self.X, self.u, self.p = t(inp.X), t(inp.u), t(inp.p)
        self.prm = t(inp.params) if inp.params is not None else torch.stack([t(inp.lam), t(inp.mu)])
        self.n, self.N = self.conn.shape[1], inp.n_nodes

    def kinematics(self, X, u, s=slice(None)):
        """Physical gradients [e, q, a, 3], weights times det J [e, q] and F [e, q, 3, 3]."""
        Jac = torch.einsum("qar,eac->eqrc", self.gg, X[self.gconn[s]])
        grads = torch.einsum("eqcr,qar->eqac", torch.linalg.inv(Jac), self.g)
        F = torch.einsum("eai,eqac->eqic", u.view(-1, 3)[self.conn[s]], grads)
        return grads, self.w * _det(Jac), F + torch.eye(3, dtype=F.dtype, device=F.device)

    def energy(self, X, u, prm):
        _, da, F = self.kinematics(X, u)
        return (_psi(self.material, F, prm[:, :, None]) * da).sum()

    def gradient(self):
        u = self.u.clone().requires_grad_(True)
        return torch.autograd.grad(self.energy(self.X, u, self.prm), u)[0]

    def chunks(self):
        E, step = self.inp.n_elements, max(1, 2_000_000 // (self.n * self.n * 9))
        return [slice(s, min(s + step, E)) for s in range(0, E, step)]

    def element_matrices(self, s, psd):
        grads, da, F = self.kinematics(self.X, self.u, s)
        prm = self.prm[:, s, None].expand(-1, *da.shape).reshape(self.prm.shape[0], -1).T
        C = torch.func.vmap(torch.func.hessian(lambda f, q: _psi(self.material, f, q)))(F.reshape(-1, 3, 3), prm)
        C = C.view(*da.shape, 3, 3, 3, 3) * da[..., None, None, None, None]
        H = torch.einsum("eqak,eqikjl,eqbl->eaibj", grads, C, grads).reshape(-1, 3 * self.n, 3 * self.n)
        if psd:
            H = 0.5 * (H + H.transpose(1, 2))
            lam, Z = torch.linalg.eigh(H)
            fixed = (Z * lam.clamp(min=0)[:, None, :]) @ Z.transpose(1, 2)
            H = torch.where((lam[:, 0] <= 0)[:, None, None], fixed, H)
        return H

    def hessian(self, psd=False):
        """CSC (values, rows, columns) with the rows of a column ascending."""
        pair = lambda s: (self.conn[s][:, None, :] * self.N + self.conn[s][:, :, None]).reshape(-1)  # column node, row node
        keys = torch.unique(torch.cat([torch.unique(pair(s)) for s in self.chunks()]))
        col, row = keys // self.N, keys % self.N
        deg = torch.bincount(col, minlength=self.N)
        first = torch.cumsum(deg, 0) - deg
        rank = torch.arange(keys.numel(), device=self.dev) - first[col]
        c3 = torch.arange(3, device=self.dev)
        # block entry (r, c) of pair k: 9 first[col] + c 3 deg[col] + 3 rank + r
        at = (9 * first[col] + 3 * rank)[:, None, None] + c3[:, None] + (3 * deg[col])[:, None, None] * c3
        vals = torch.zeros(9 * keys.numel(), dtype=torch.float64, device=self.dev)
        for s in self.chunks():
            H = self.element_matrices(s, psd).view(-1, self.n, 3, self.n, 3)
            dst = at[torch.searchsorted(keys, pair(s))].reshape(-1, self.n, self.n, 3, 3).permute(0, 1, 3, 2, 4)
            vals.index_add_(0, dst.reshape(-1), H.reshape(-1))
        rows, cols = torch.empty_like(vals, dtype=torch.int32), torch.empty_like(vals, dtype=torch.int32)
        rows[at.reshape(-1)] = (3 * row[:, None, None] + c3[:, None]).expand_as(at).reshape(-1).int()
        cols[at.reshape(-1)] = (3 * col[:, None, None] + c3).expand_as(at).reshape(-1).int()
        return vals, rows, cols

    def reduced_system(self):
        """The clamped dofs dropped: (gradient, values, rows, columns) in the free numbering."""
        free = torch.ones(3 * self.N, dtype=torch.bool, device=self.dev)
        free[torch.as_tensor(self.inp.fixed, device=self.dev)] = False
        vals, rows, cols = self.hessian(psd=True)
        keep = free[rows.long()] & free[cols.long()]
        new = torch.cumsum(free, 0) - 1
        return self.gradient()[free], vals[keep], new[rows[keep].long()], new[cols[keep].long()], free

    def solve(self):
        """x with H x = -gradient over the free dofs, by conjugate gradients run to rounding."""
        grad, vals, rows, cols, free = self.reduced_system()
        n = grad.numel()
        outer = torch.zeros(n + 1, dtype=torch.int64, device=self.dev)
        outer[1:] = torch.cumsum(torch.bincount(cols, minlength=n), 0)
        A = torch.sparse_csr_tensor(outer, rows, vals, size=(n, n))  # symmetric: columns serve as rows
        diag = torch.ones(n, dtype=torch.float64, device=self.dev)
        on = rows == cols
        diag[rows[on]] = vals[on]
        x, r = torch.zeros_like(grad), -grad
        z = r / diag
        d, rz, stop = z.clone(), torch.dot(r, z), 1e-15 * float(grad.norm())
        for it in range(6000):
            q = A @ d
            alpha = rz / torch.dot(d, q)
            x += alpha * d
            r -= alpha * q
            z = r / diag
            rz, old = torch.dot(r, z), rz
            d = z + (rz / old) * d
            if it % 20 == 0 and float(r.norm()) <= stop:
                break
        return x, free


def exact(case, seed):
    kind = case["kind"]
    if kind in ("cg", "direct", "newton") and _sizes(case)[1] > 130_000:
        return None
    ex = _Exact(case, seed)
    if kind == "energy":
        return ex.energy(ex.X, ex.u, ex.prm)
    if kind == "value_gradient":
        return ex.energy(ex.X, ex.u, ex.prm), ex.gradient()
    if kind == "hessian":
        return ex.hessian()[0]
    if kind == "projected":
        return ex.reduced_system()[:2]
    if kind in ("cg", "direct"):
        return ex.solve()[0]
    if kind == "newton":
        x, free = ex.solve()
        full = torch.zeros(3 * ex.N, dtype=torch.float64, device=ex.dev)
        full[free] = x
        return full
    if kind == "adjoint":
        u, X, prm = (t.clone().requires_grad_(True) for t in (ex.u, ex.X, ex.prm))
        force = torch.autograd.grad(ex.energy(X, u, prm), u, create_graph=True)[0]
        gu, gprm, gX = torch.autograd.grad(force, (u, prm, X), ex.p)
        return force.detach(), gu, gprm[0], gprm[1], gX
    vals, rows, _ = ex.hessian()
    return float(ex.energy(ex.X, ex.u, ex.prm)), ex.gradient().cpu().numpy(), vals.cpu().numpy(), None, None
