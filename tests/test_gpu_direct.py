"""Sparse direct solve on the device (pfg_direct_*, polyfem_b200.DirectSolver): the
factorisation polysolve's direct choices compute for the Newton system, run on the
Hessian the assembler left on the GPU.  Checked against scipy's SuperLU solve of
the same matrix and by the residual; the factor and solution are bitwise
deterministic."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spla

from polyfem_b200 import DirectSolver, NeoHookeanAssembler, PfgError
from polyfem_b200 import mesh as M
from polyfem_b200._lib import PFG_ERR_NUMERIC, PFG_ERR_STATE

from _cases import make_case, rel_err

pytestmark = pytest.mark.gpu

CASES = [(M.P1_TET, 3), (M.P2_TET, 2), (M.Q1_HEX, 3), (M.P1_TET, 8), (M.P2_TET, 5), (M.Q1_HEX, 7)]


def reduced_system(et, g, seed=3):
    """Dirichlet-reduced (x = 0 face fixed), PSD-projected Hessian of a compressed
    state: symmetric positive definite."""
    mesh, lam, mu, u, _ = make_case(et, g, seed=seed, jitter=0.1 if et != M.P1_TET else 0.0)
    rng = np.random.default_rng(seed + 1)
    u = (-0.2 * mesh.node_pos + 0.02 * mesh.h * rng.standard_normal(mesh.node_pos.shape)).ravel()
    asm = NeoHookeanAssembler.from_mesh(mesh, lam, mu)
    face = np.flatnonzero(mesh.node_pos[:, 0] <= 1e-12)
    asm.set_dirichlet((3 * face[:, None] + np.arange(3)).ravel())
    H = asm.assemble_hessian_reduced(u, "fp64", project_to_psd=True)  # values stay in the context
    g_red = asm.assemble_gradient_reduced(u, "fp64")
    return mesh, asm, u, H, g_red


@pytest.mark.parametrize("et,g", CASES, ids=["P1-3", "P2-2", "Q1-3", "P1-8", "P2-5", "Q1-7"])
def test_reduced_solve_matches_superlu(require_gpu, et, g):
    mesh, asm, u, H, grad = reduced_system(et, g)
    b = -grad
    ds = DirectSolver(asm, "reduced")
    ds.analyze_pattern(H, H.shape[0])
    info = ds.get_info()
    assert info["n"] == H.shape[0] and info["fronts"] >= 1
    assert info["nnz_L"] >= (H.nnz + H.shape[0]) // 2  # L holds A's lower triangle
    ds.factorize()
    x = ds.solve(b)
    res = np.linalg.norm(b - H @ x) / np.linalg.norm(b)
    assert res <= 1e-12, res
    xd = spla.spsolve(H.tocsc(), b)
    assert rel_err(x, xd) <= 1e-10
    asm.close()


def test_medium_system_residual(require_gpu):
    """P2 12^3 (about 45k free dofs, fronts up to ~3,900): the residual of the
    device solve, checked with a host sparse product."""
    mesh, asm, u, H, grad = reduced_system(M.P2_TET, 12)
    ds = DirectSolver(asm, "reduced")
    ds.analyze_pattern()
    ds.factorize()
    b = -grad
    x = ds.solve(b)
    assert np.linalg.norm(b - H @ x) / np.linalg.norm(b) <= 1e-11
    asm.close()


def test_deterministic_device_and_host_mode(require_gpu):
    import torch
    mesh, asm, u, H, grad = reduced_system(M.P2_TET, 3)
    ds = DirectSolver(asm, "reduced")
    ds.analyze_pattern()
    ds.factorize()
    xh = ds.solve(-grad)
    bd = torch.tensor(-grad, dtype=torch.float64, device="cuda")
    x1 = ds.solve(bd).cpu().numpy()
    ds.factorize()  # a second factorisation of the same values
    x2 = ds.solve(bd).cpu().numpy()
    assert np.array_equal(x1, x2)
    assert np.array_equal(x1, xh)
    # in place: x aliases b
    bd2 = bd.clone()
    ds.solve(bd2, bd2)
    assert np.array_equal(bd2.cpu().numpy(), x1)
    asm.close()


def test_caller_values_and_not_positive_definite(require_gpu):
    """Caller values (device memory) replace the context's: H + s I on the full
    (singular) system solves; -H on the reduced system is refused with
    PFG_ERR_NUMERIC, after which the solver needs a successful factorisation."""
    import torch
    mesh, lam, mu, u, _ = make_case(M.P1_TET, 3, seed=5)
    asm = NeoHookeanAssembler.from_mesh(mesh, lam, mu)
    H = asm.assemble_hessian(u, "fp64", project_to_psd=True).tocsc()
    H.sort_indices()
    s = 1e-3 * abs(H.diagonal()).max()
    A = (H + s * sp.identity(H.shape[0], format="csc")).tocsc()
    A.sort_indices()
    assert np.array_equal(A.indptr, H.indptr) and np.array_equal(A.indices, H.indices)
    ds = DirectSolver(asm, "full")
    ds.analyze_pattern()
    vals = torch.tensor(A.data, dtype=torch.float64, device="cuda")
    ds.factorize(vals)
    b = np.random.default_rng(1).standard_normal(H.shape[0])
    x = ds.solve(b)
    assert rel_err(x, spla.spsolve(A, b)) <= 1e-10
    with pytest.raises(PfgError) as ei:
        ds.factorize(-vals)
    assert ei.value.status == PFG_ERR_NUMERIC
    with pytest.raises(PfgError) as ei:
        ds.solve(b)
    assert ei.value.status == PFG_ERR_STATE
    ds.factorize(vals)
    assert np.array_equal(ds.solve(b), x)
    asm.close()


def test_state_errors(require_gpu):
    mesh, asm, u, H, grad = reduced_system(M.P1_TET, 3)
    ds = DirectSolver(asm, "reduced")
    with pytest.raises(PfgError) as ei:
        ds.factorize()
    assert ei.value.status == PFG_ERR_STATE
    ds.analyze_pattern()
    ds.factorize()
    x = ds.solve(-grad)
    # a new Dirichlet set changes the reduced pattern: the analysis is discarded
    face = np.flatnonzero(mesh.node_pos[:, 0] <= 1e-12)
    asm.set_dirichlet((3 * face[:, None] + np.arange(3)).ravel())
    with pytest.raises(PfgError) as ei:
        ds.solve(-grad)
    assert ei.value.status == PFG_ERR_STATE
    H2 = asm.assemble_hessian_reduced(u, "fp64", project_to_psd=True)
    ds.analyze_pattern()
    ds.factorize()
    assert np.array_equal(ds.solve(-grad), x)
    with pytest.raises(ValueError):
        ds.solve(np.zeros(H2.shape[0] + 1))
    # released: the factor is gone until the next analysis
    ds.free()
    with pytest.raises(PfgError) as ei:
        ds.solve(-grad)
    assert ei.value.status == PFG_ERR_STATE
    ds.analyze_pattern()
    ds.factorize()
    assert np.array_equal(ds.solve(-grad), x)
    asm.close()


def test_newton_step_direct_equals_cg(require_gpu):
    """One Newton step of NLProblem with the direct solve: the step agrees with the
    tight CG solve of the same system (to the CG residual times the condition)."""
    from polyfem_b200 import ConjugateGradient
    mesh, asm, u, H, grad = reduced_system(M.Q1_HEX, 4)
    ds = DirectSolver(asm, "reduced")
    ds.analyze_pattern()
    ds.factorize()
    xd = ds.solve(-grad)
    cg = ConjugateGradient(asm, "reduced")
    cg.set_parameters({"tolerance": 1e-13, "max_iter": 20000})
    xc = cg.solve(-grad)
    assert rel_err(xd, xc) <= 1e-7
    asm.close()


@pytest.mark.parametrize("et,g", [(M.P1_TET, 6), (M.P2_TET, 4), (M.Q1_HEX, 6)], ids=["P1", "P2", "Q1"])
def test_position_ordering_on_shuffled_and_flat_meshes(require_gpu, et, g):
    """The analysis cuts across node positions: shuffled numbering, and a mesh so flat
    that one axis has next to no extent, solve to the same residual; on the shuffled
    cube the cuts need no more operations than those of the bare pattern."""
    from polyfem_b200 import direct_symbolic
    from _cases import permuted
    mesh, lam, mu, u, _ = make_case(et, g, seed=9)
    for flat in (1.0, 1e-2):
        m2, u2, _, pe = permuted(mesh, u, seed=4)
        m2.X = m2.X * np.array([1.0, 1.0, flat])
        u2 = u2.reshape(-1, 3) * np.array([1.0, 1.0, flat])
        asm = NeoHookeanAssembler.from_mesh(m2, lam[pe], mu[pe])
        face = np.flatnonzero(m2.node_pos[:, 0] <= 1e-12)
        asm.set_dirichlet((3 * face[:, None] + np.arange(3)).ravel())
        H = asm.assemble_hessian_reduced(u2.ravel(), "fp64", project_to_psd=True)
        ds = DirectSolver(asm, "reduced")
        ds.analyze_pattern()
        if flat == 1.0:
            H.sort_indices()
            assert ds.get_info()["flops"] <= direct_symbolic(H.indptr, H.indices)["flops"]
        ds.factorize()
        b = np.random.default_rng(1).standard_normal(H.shape[0])
        x = ds.solve(b)
        scale = abs(H).sum(axis=1).max() * np.abs(x).max()  # normwise backward error
        assert np.abs(b - H @ x).max() <= 1e-13 * scale
        asm.close()


@pytest.mark.parametrize("et,g,n", [(M.P1_TET, 2, n) for n in (1, 7, 8, 9, 31, 32, 33, 63, 64, 65, 81)]
                         + [(M.Q1_HEX, 8, n) for n in (1900, 2100, 2187)] + [(M.P2_TET, 4, n) for n in (2049, 2187)])
def test_front_sizes_around_the_panel_edges(require_gpu, et, g, n):
    """Free dofs chosen at random give fronts whose column counts fall on and beside the
    edges of the 8-column, 64-column and 128-column steps (the 81-dof meshes are one
    front).  Normwise backward error of the solve at rounding level."""
    mesh, lam, mu, u, _ = make_case(et, g, seed=6)
    asm = NeoHookeanAssembler.from_mesh(mesh, lam, mu)
    rng = np.random.default_rng(n)
    asm.set_dirichlet(np.sort(rng.permutation(mesh.n_dofs)[: mesh.n_dofs - n]))
    asm.assemble_hessian_reduced(u, "fp64", project_to_psd=True)
    outer, inner = asm.reduced_pattern()
    # any symmetric positive definite values in the pattern: a random diagonally dominant matrix
    A = sp.csc_matrix((rng.standard_normal(inner.size), inner, outer), shape=(n, n))
    A = ((A + A.T) * 0.5).tocsc()
    A.sort_indices()
    A.setdiag(np.asarray(abs(A).sum(axis=0)).ravel() + rng.uniform(0.5, 2.0, n))
    import torch
    ds = DirectSolver(asm, "reduced")
    ds.analyze_pattern()
    assert np.array_equal(A.indices, inner)
    ds.factorize(torch.tensor(A.data, device="cuda"))
    b = rng.standard_normal(n)
    x = ds.solve(b)
    scale = abs(A).sum(axis=1).max() * np.abs(x).max()
    assert np.abs(b - A @ x).max() <= 1e-13 * scale
    asm.close()


@pytest.mark.parametrize("width", [0.1, 0.25])
@pytest.mark.parametrize("et,g", [(M.Q1_HEX, 1), (M.P2_TET, 1), (M.Q1_HEX, 2), (M.Q1_HEX, 6), (M.P2_TET, 4)], ids=str)
def test_ill_conditioned_systems(require_gpu, et, g, width):
    """Element matrices that are Gaussian Gram matrices (nearly singular, condition 1e11): the
    residual of the solve stays at the bound of Cholesky and substitution.  The computed x
    solves (A + dA) x = b with |dA| <= gamma(3n + 1) |L||L^T| (Higham, Accuracy and Stability,
    theorem 10.4), and (|L||L^T|)_ij <= sqrt(a_ii a_jj); two roundings more a pivot where a
    reciprocal takes the division's place: 5 n u.  A product with an explicit inverse of the
    diagonal blocks misses it by the root of the blocks' condition."""
    import torch
    mesh, lam, mu, _, _ = make_case(et, g, seed=2)
    asm = NeoHookeanAssembler.from_mesh(mesh, lam, mu)
    outer, inner = asm.hessian_pattern()
    n, k = asm.n_dofs, 3 * mesh.conn.shape[1]
    t = np.linspace(0.0, 1.0, k)
    gram = np.exp(-(((t[:, None] - t) / width) ** 2)) + 1e-11 * np.eye(k)
    dofs = (3 * mesh.conn[:, :, None] + np.arange(3)).reshape(mesh.n_elements, k)
    A = sp.coo_matrix((np.tile(gram.ravel(), mesh.n_elements), (np.repeat(dofs, k, 1).ravel(), np.tile(dofs, (1, k)).ravel())),
                      shape=(n, n)).tocsc()
    A.sort_indices()
    assert np.array_equal(A.indptr, outer) and np.array_equal(A.indices, inner)
    ds = DirectSolver(asm, "full")
    ds.analyze_pattern()
    ds.factorize(torch.tensor(A.data, device="cuda"))
    root = np.sqrt(A.diagonal())
    R = A.tocsr()
    for b in (A @ np.ones(n), np.random.default_rng(3).standard_normal(n)):
        x = ds.solve(b)
        Ax = np.add.reduceat(R.data.astype(np.longdouble) * x[R.indices], R.indptr[:-1])
        bound = 5 * n * 2.0 ** -53 * root * (root @ np.abs(x))
        assert np.all(np.abs(b - Ax) <= bound), float(np.max(np.abs(b - Ax) / bound))
    asm.close()


def turned(angle, axis):
    a = np.asarray(axis, dtype=float) / np.linalg.norm(axis)
    K = np.array([[0, -a[2], a[1]], [a[2], 0, -a[0]], [-a[1], a[0], 0]])
    return lambda X: X @ (np.eye(3) + np.sin(angle) * K + (1 - np.cos(angle)) * K @ K).T


def spiral(X):
    r, t = 3 + 0.5 * X[:, 0] + 0.3 * X[:, 1], 4 * X[:, 0]
    return np.stack([r * np.cos(t), r * np.sin(t), X[:, 2]], axis=1)


SHAPES = {"turned": turned(0.5, (1, 2, 3)), "diagonal": turned(np.arccos(3 ** -0.5), (0, -1, 1)),
          "z45": turned(np.pi / 4, (0, 0, 1)), "spiral": spiral}


@pytest.mark.parametrize("shape", list(SHAPES))
@pytest.mark.parametrize("et,g,slender", [(M.P1_TET, 12, 1), (M.P2_TET, 8, 1), (M.Q1_HEX, 12, 1), (M.Q1_HEX, 16, 6)], ids=str)
def test_ordering_of_bodies_off_the_axes(require_gpu, et, g, slender, shape):
    """The work of the factorisation does not depend on how the body lies in space: turned and
    bent cubes and beams stay within a quarter of the operations of the bare pattern's analysis,
    which has no positions (cuts across x, y and z alone need two to three times as many)."""
    from polyfem_b200 import direct_symbolic
    mesh, lam, mu, _, _ = make_case(et, g, seed=9)
    if slender > 1:  # a beam: the first cells of y and z
        c = mesh.X[mesh.gconn].mean(axis=1)
        keep = np.all(c[:, 1:] < 1.0 / slender + 1e-9, axis=1)
        used, conn = np.unique(mesh.conn[keep], return_inverse=True)
        mesh.conn = mesh.gconn = conn.reshape(-1, mesh.conn.shape[1]).astype(np.int32)
        mesh.X = mesh.node_pos = mesh.X[used]
        mesh.n_nodes = used.size
        lam, mu = lam[keep], mu[keep]
    mesh.X = SHAPES[shape](mesh.X)
    asm = NeoHookeanAssembler.from_mesh(mesh, lam, mu)
    outer, inner = asm.hessian_pattern()
    ds = DirectSolver(asm, "full")
    ds.analyze_pattern()
    assert ds.get_info()["flops"] <= 1.25 * direct_symbolic(outer, inner)["flops"]
    asm.close()
