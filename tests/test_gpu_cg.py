"""Device conjugate gradient (pfg_cg_solve, polyfem_b200.ConjugateGradient): the
linear solve NewtonMethod makes after every assembly, run on the Hessian the
assembler left on the GPU.  Checked against the oracle's restatement of Eigen's
ConjugateGradient with the diagonal preconditioner on the same matrix, and
against a direct solve."""
import ctypes

import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spla

from oracle.binding import conjugate_gradient
from polyfem_b200 import ConjugateGradient, NeoHookeanAssembler, PfgError
from polyfem_b200 import mesh as M
from polyfem_b200._lib import PFG_MEM_HOST, lib

from _cases import make_case, rel_err

pytestmark = pytest.mark.gpu

CASES = [(M.P1_TET, 3), (M.P2_TET, 2), (M.Q1_HEX, 3)]


def reduced_system(et, g, seed=3, compress=True):
    """Dirichlet-reduced (x = 0 face fixed), PSD-projected Hessian: symmetric positive definite."""
    mesh, lam, mu, u, _ = make_case(et, g, seed=seed, jitter=0.1 if et != M.P1_TET else 0.0)
    if compress:
        rng = np.random.default_rng(seed + 1)
        u = (-0.2 * mesh.node_pos + 0.02 * mesh.h * rng.standard_normal(mesh.node_pos.shape)).ravel()
    asm = NeoHookeanAssembler.from_mesh(mesh, lam, mu)
    face = np.flatnonzero(mesh.node_pos[:, 0] <= 1e-12)
    asm.set_dirichlet((3 * face[:, None] + np.arange(3)).ravel())
    H = asm.assemble_hessian_reduced(u, "fp64", project_to_psd=True)  # host mode: values stay in the context
    g_red = asm.assemble_gradient_reduced(u, "fp64")
    return mesh, asm, u, H, g_red


@pytest.mark.parametrize("et,g", CASES, ids=["P1", "P2", "Q1"])
def test_reduced_solve_matches_oracle_and_direct(require_gpu, et, g):
    mesh, asm, u, H, grad = reduced_system(et, g)
    b = -grad
    cg = ConjugateGradient(asm, "reduced")
    cg.set_parameters({"tolerance": 1e-11, "max_iter": 5000})
    cg.analyze_pattern(H, H.shape[0])
    cg.factorize()
    x = cg.solve(b)
    info = cg.get_info()
    xo, it_o, res_o = conjugate_gradient(H.indptr, H.indices, H.data, b, 1e-11, 5000)
    # same iteration up to the rounding of the dot products (tree vs sequential order)
    assert abs(info["solver_iter"] - it_o) <= max(2, it_o // 50), (info, it_o)
    assert info["solver_error"] < 1e-11 and res_o < 1e-11
    res = np.linalg.norm(b - H @ x) / np.linalg.norm(b)
    assert res <= 2e-11 and abs(res - info["solver_error"]) <= 1e-11
    xd = spla.spsolve(H.tocsc(), b)
    assert rel_err(x, xd) <= 1e-8
    assert rel_err(x, xo) <= 1e-8
    asm.close()


def test_device_mode_deterministic_and_equal_to_host_mode(require_gpu):
    import torch
    mesh, asm, u, H, grad = reduced_system(M.P2_TET, 2)
    cg = ConjugateGradient(asm, "reduced")
    cg.set_parameters({"tolerance": 1e-10, "max_iter": 2000})
    xh = cg.solve(-grad)
    bd = torch.tensor(-grad, dtype=torch.float64, device="cuda")
    x1 = cg.solve(bd).cpu().numpy()
    x2 = cg.solve(bd).cpu().numpy()
    assert np.array_equal(x1, x2)
    assert np.array_equal(x1, xh)
    asm.close()


def test_caller_values_on_the_full_system(require_gpu):
    """The full Hessian is singular (rigid motions); a caller-supplied values array
    H + s I (device memory) takes the context's place."""
    import torch
    mesh, lam, mu, u, _ = make_case(M.P1_TET, 3, seed=5)
    asm = NeoHookeanAssembler.from_mesh(mesh, lam, mu)
    vals = asm.assemble_hessian_values(u, "fp64", project_to_psd=True)
    outer, inner = asm.hessian_pattern()
    n = asm.n_dofs
    cols = np.repeat(np.arange(n), np.diff(outer))
    shift = 1e-3 * np.abs(vals).max()
    vals_s = vals.copy()
    vals_s[inner == cols] += shift
    A = sp.csc_matrix((vals_s, inner, outer), shape=(n, n))
    b = np.random.default_rng(2).standard_normal(n)
    cg = ConjugateGradient(asm, "full")
    cg.set_parameters({"tolerance": 1e-12, "max_iter": 5000})
    cg.factorize(torch.tensor(vals_s, device="cuda"))
    x = cg.solve(b)
    assert np.linalg.norm(b - A @ x) / np.linalg.norm(b) <= 2e-12
    xo, it_o, _ = conjugate_gradient(outer, inner, vals_s, b, 1e-12, 5000)
    assert abs(cg.get_info()["solver_iter"] - it_o) <= max(2, it_o // 50)
    assert rel_err(x, xo) <= 1e-9
    asm.close()


def test_guess_zero_rhs_and_iteration_cap(require_gpu):
    mesh, asm, u, H, grad = reduced_system(M.P1_TET, 3)
    b = -grad
    cg = ConjugateGradient(asm, "reduced")
    cg.set_parameters({"tolerance": 1e-10, "max_iter": 3000})
    x = cg.solve(b)
    # starting from the solution: converged before the first iteration
    x2 = x.copy()
    cg.solve(b, x2, guess=True)
    assert cg.get_info()["solver_iter"] == 0 and np.array_equal(x2, x)
    # b = 0: x = 0 without iterating, whatever the guess
    xz = np.ones_like(b)
    cg.solve(np.zeros_like(b), xz, guess=True)
    assert cg.get_info() == {"solver_iter": 0, "solver_error": 0.0} and not xz.any()
    # the iteration cap is reached and reported through the residual, not as an error
    cg.set_parameters({"max_iter": 3})
    cg.solve(b)
    info = cg.get_info()
    assert info["solver_iter"] == 3 and info["solver_error"] > 1e-10
    _, it_o, res_o = conjugate_gradient(H.indptr, H.indices, H.data, b, 1e-10, 3)
    assert it_o == 3 and abs(info["solver_error"] - res_o) <= 1e-9 * res_o
    asm.close()


def test_newton_step_is_a_descent_direction(require_gpu):
    """dx = -H^-1 g with the projected reduced Hessian: g.dx < 0 and the energy drops
    along dx (the step NewtonMethod takes)."""
    mesh, asm, u, H, grad = reduced_system(M.P2_TET, 2)
    cg = ConjugateGradient(asm, "reduced")
    cg.set_parameters({"tolerance": 1e-10, "max_iter": 3000})
    dx = cg.solve(-grad)
    assert grad @ dx < 0
    du = asm.reduced_to_full(dx, np.zeros(asm.n_dofs))
    e0 = asm.assemble_energy(u)
    e1 = asm.assemble_energy(u + 1e-3 * du)
    assert e1 < e0
    asm.close()


def test_argument_and_state_errors(require_gpu):
    mesh, lam, mu, u, _ = make_case(M.P1_TET, 2, seed=1)
    asm = NeoHookeanAssembler.from_mesh(mesh, lam, mu)
    L = lib()
    b = np.zeros(asm.n_dofs)
    x = np.zeros(asm.n_dofs)
    bp, xp = ctypes.c_void_p(b.ctypes.data), ctypes.c_void_p(x.ctypes.data)
    it, res = ctypes.c_int(), ctypes.c_double()
    args = (bp, PFG_MEM_HOST, 1e-10, 100, 0, xp, ctypes.byref(it), ctypes.byref(res))
    assert L.pfg_cg_solve(asm.handle, 7, None, *args) == 1               # PFG_ERR_INVALID: no such system
    assert L.pfg_cg_solve(asm.handle, 1, None, *args) == 5               # PFG_ERR_STATE: no Dirichlet set
    assert L.pfg_cg_solve(asm.handle, 0, None, bp, PFG_MEM_HOST, -1.0, 100, 0, xp, None, None) == 1
    with pytest.raises(PfgError):
        ConjugateGradient(asm, "reduced").solve(np.zeros(0))
    asm.close()


def star_mesh(n, seed=0):
    """P1 tetrahedra from one centre node to the triangles of a sphere's hull: the centre
    neighbours every node."""
    from scipy.spatial import ConvexHull
    rng = np.random.default_rng(seed)
    pts = rng.standard_normal((n, 3))
    pts /= np.linalg.norm(pts, axis=1)[:, None]
    tri = ConvexHull(pts).simplices
    X = np.concatenate([pts, np.zeros((1, 3))])
    tets = np.concatenate([tri, np.full((tri.shape[0], 1), n)], axis=1)
    e = X[tets[:, 1:]] - X[tets[:, :1]]
    flip = np.linalg.det(e) < 0
    tets[flip, 0], tets[flip, 1] = tets[flip, 1].copy(), tets[flip, 0].copy()
    return tets.astype(np.int32), X


@pytest.mark.parametrize("case", ["star-20", "star-60", "star-rest-150", "P1-mixed", "P2-mixed", "Q1-mixed", "P2-long"])
def test_group_sizes_and_partly_fixed_nodes(require_gpu, case):
    """Column groups of every kind the iteration distinguishes: neighbours beyond one warp
    (star-60, P2 vertices), beyond a shared-memory stage (star-rest-150), nodes with one or two
    free dofs (random Dirichlet dofs), and a matrix that streams in several chunks a warp
    (P2-long).  The residual against a host product, and the oracle's iteration count."""
    if case.startswith("star"):
        conn, X = star_mesh(int(case.split("-")[-1]))
        asm = NeoHookeanAssembler(M.P1_TET, conn, X, 1e5, 5e4)
        u, n_dofs = 0.01 * np.random.default_rng(1).standard_normal(3 * X.shape[0]), 3 * X.shape[0]
        if "rest" in case:  # its thin tetrahedra would invert under u
            u = np.zeros(n_dofs)
    else:
        et = {"P1": M.P1_TET, "P2": M.P2_TET, "Q1": M.Q1_HEX}[case[:2]]
        mesh, lam, mu, u, _ = make_case(et, 13 if case == "P2-long" else 4, seed=8)
        asm = NeoHookeanAssembler.from_mesh(mesh, lam, mu)
        n_dofs = mesh.n_dofs
    rng = np.random.default_rng(3)
    asm.set_dirichlet(np.sort(rng.permutation(n_dofs)[: max(12, n_dofs // 9)]))
    H = asm.assemble_hessian_reduced(u, "fp64", project_to_psd=True)
    b = rng.standard_normal(H.shape[0])
    cg = ConjugateGradient(asm, "reduced")
    cg.set_parameters({"tolerance": 1e-10, "max_iter": 20000})
    x = cg.solve(b)
    assert np.linalg.norm(b - H @ x) <= 2e-10 * np.linalg.norm(b)
    _, it_o, _ = conjugate_gradient(H.indptr, H.indices, H.data, b, 1e-10, 20000)
    assert abs(cg.get_info()["solver_iter"] - it_o) <= max(2, it_o // 20)
    assert np.array_equal(cg.solve(b), x)
    asm.close()


@pytest.mark.parametrize("et,g", [(M.P1_TET, 1), (M.P1_TET, 4), (M.P2_TET, 13)], ids=["one chunk", "resident", "streaming"])
@pytest.mark.parametrize("n_fixed", [9, 10])
def test_values_at_any_alignment(require_gpu, et, g, n_fixed):
    """Values that begin on 8 bytes, with even and odd counts (the bulk copies move 16-byte
    units): the same bits as from an aligned array."""
    import torch
    mesh, lam, mu, u, _ = make_case(et, g, seed=5)
    asm = NeoHookeanAssembler.from_mesh(mesh, lam, mu)
    asm.set_dirichlet(np.arange(n_fixed))
    v = asm.assemble_hessian_reduced_values(torch.tensor(u, device="cuda"), project_to_psd=True)
    b = torch.tensor(np.random.default_rng(2).standard_normal(asm.n_free), device="cuda")
    cg = ConjugateGradient(asm, "reduced")
    cg.set_parameters({"tolerance": 1e-10, "max_iter": 300})
    cg.factorize(v)
    x = cg.solve(b)
    assert torch.isfinite(x).all() and bool(x.abs().max() > 0)
    shifted = torch.full((v.numel() + 1,), float("nan"), dtype=torch.float64, device="cuda")
    shifted[1:] = v
    cg.factorize(shifted[1:])
    assert torch.equal(cg.solve(b), x)
    asm.close()


@pytest.mark.parametrize("et,g", [(M.P1_TET, 8), (M.P2_TET, 13)], ids=["resident", "streaming"])
@pytest.mark.parametrize("mem", ["host", "device"])
def test_a_wait_that_gave_up_is_reported_and_leaves_nothing_behind(require_gpu, et, g, mem):
    """A solve whose grid waits for a CTA that never comes ends with an error, and so does one
    in which a CTA other than the first gave up, whatever state the first one left; the solves
    after it return the bits of the one before."""
    import torch

    from polyfem_b200._lib import PFG_ERR_CUDA
    mesh, lam, mu, u, _ = make_case(et, g, seed=5)
    asm = NeoHookeanAssembler.from_mesh(mesh, lam, mu)
    asm.set_dirichlet(np.arange(9))
    asm.assemble_hessian_reduced(u, "fp64", project_to_psd=True)
    b = np.random.default_rng(2).standard_normal(asm.n_free)
    if mem == "device":
        b = torch.tensor(b, device="cuda")
    cg = ConjugateGradient(asm, "reduced")
    cg.set_parameters({"tolerance": 1e-10, "max_iter": 120})
    bits = lambda x: x.cpu().numpy() if mem == "device" else x
    x = bits(cg.solve(b))
    for how in (1, 2):
        assert lib().pfg_selftest_cg_give_up(asm.handle, how) == 0
        with pytest.raises(PfgError) as e:
            cg.solve(b)
        assert e.value.status == PFG_ERR_CUDA
        for _ in range(2):
            assert np.array_equal(bits(cg.solve(b)), x)
    asm.close()


@pytest.mark.parametrize("most", [1, 2, 7])
@pytest.mark.parametrize("et,g", [(M.P1_TET, 3), (M.P1_TET, 9), (M.Q1_HEX, 13)], ids=["small", "P1-9", "Q1-13"])
def test_streams_with_part_of_the_device(require_gpu, et, g, most):
    """Where the stream takes fewer CTAs than the plan has (a context limited to part of the
    SMs), the solve goes on with as many as it takes: the oracle's iteration count and the same
    residual, also with runs of many chunks and more than 256 groups a CTA; on another stream
    the whole device again."""
    import torch
    mesh, lam, mu, u, _ = make_case(et, g, seed=8)
    asm = NeoHookeanAssembler.from_mesh(mesh, lam, mu)
    asm.set_dirichlet(np.arange(12))
    H = asm.assemble_hessian_reduced(u, "fp64", project_to_psd=True)
    b = np.random.default_rng(3).standard_normal(H.shape[0])
    cg = ConjugateGradient(asm, "reduced")
    cg.set_parameters({"tolerance": 1e-10, "max_iter": 5000})
    x = cg.solve(b)
    _, it_o, _ = conjugate_gradient(H.indptr, H.indices, H.data, b, 1e-10, 5000)
    assert lib().pfg_selftest_cg_most(asm.handle, most) == 0
    for _ in range(2):
        y = cg.solve(b)
        assert np.linalg.norm(b - H @ y) <= 2e-10 * np.linalg.norm(b)
        assert abs(cg.get_info()["solver_iter"] - it_o) <= max(2, it_o // 20)
    with torch.cuda.stream(torch.cuda.Stream()):
        z = cg.solve(torch.tensor(b, device="cuda")).cpu().numpy()
    assert np.linalg.norm(b - H @ z) <= 2e-10 * np.linalg.norm(b)
    assert lib().pfg_selftest_cg_most(asm.handle, 0) == 0
    assert np.array_equal(cg.solve(b), x)
    asm.close()


def test_many_groups_per_cta(require_gpu):
    """More than 256 column groups a CTA, whose H p (and, with resident runs, direction) stay in
    global memory: P1 34^3 on the whole device (streaming), and 2,000 single tetrahedra on 20
    CTAs (resident), against a host product and the oracle's iteration count."""
    mesh, lam, mu, u, _ = make_case(M.P1_TET, 34, seed=8)
    asm = NeoHookeanAssembler.from_mesh(mesh, lam, mu)
    face = np.flatnonzero(mesh.node_pos[:, 0] <= 1e-12)
    asm.set_dirichlet((3 * face[:, None] + np.arange(3)).ravel())
    H = asm.assemble_hessian_reduced(u, "fp64", project_to_psd=True)
    _check_solve(ConjugateGradient(asm, "reduced"), H, None)
    asm.close()

    import torch
    rng = np.random.default_rng(4)
    corner = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [0, 0, 1.0]])
    X = (corner[None] + 3 * np.arange(2000)[:, None, None] + 0.1 * rng.uniform(-1, 1, (2000, 4, 3))).reshape(-1, 3)
    asm = NeoHookeanAssembler(M.P1_TET, np.arange(8000, dtype=np.int32).reshape(2000, 4), X, 1e5, 5e4)
    H = asm.assemble_hessian(np.zeros(24000))
    H.sort_indices()
    H.setdiag(H.diagonal() + 10.0 ** rng.uniform(3, 5, 24000))  # free bodies: a shift for a definite matrix
    assert lib().pfg_selftest_cg_most(asm.handle, 20) == 0
    _check_solve(ConjugateGradient(asm, "full"), H, torch.tensor(H.data, device="cuda"))
    asm.close()


def _check_solve(cg, H, values):
    cg.factorize(values)
    cg.set_parameters({"tolerance": 1e-10, "max_iter": 5000})
    b = np.random.default_rng(3).standard_normal(H.shape[0])
    x = cg.solve(b)
    assert np.linalg.norm(b - H @ x) <= 2e-10 * np.linalg.norm(b)
    _, it_o, _ = conjugate_gradient(H.indptr, H.indices, H.data, b, 1e-10, 5000)
    assert abs(cg.get_info()["solver_iter"] - it_o) <= max(2, it_o // 20)
    assert np.array_equal(cg.solve(b), x)


def test_two_threads_on_two_streams(require_gpu):
    """Two contexts solve at the same time from two threads, each on its own stream, with launches
    that each want the whole device: both return the bits of a solve alone."""
    import threading

    import torch
    solvers = []
    for et, g in ((M.P1_TET, 20), (M.Q1_HEX, 16)):
        mesh, lam, mu, u, _ = make_case(et, g, seed=5)
        asm = NeoHookeanAssembler.from_mesh(mesh, lam, mu)
        asm.set_dirichlet(np.arange(9))
        v = asm.assemble_hessian_reduced_values(torch.tensor(u, device="cuda"), project_to_psd=True)
        b = torch.tensor(np.random.default_rng(2).standard_normal(asm.n_free), device="cuda")
        cg = ConjugateGradient(asm, "reduced")
        cg.set_parameters({"tolerance": 0.0, "max_iter": 300})
        cg.factorize(v)
        solvers.append((asm, cg, b, cg.solve(b).clone()))
    torch.cuda.synchronize()
    wrong = []

    def work(k):
        _, cg, b, x = solvers[k]
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(8):
                    y = cg.solve(b)
                    torch.cuda.current_stream().synchronize()
                    if not torch.equal(y, x):
                        wrong.append(k)
        except Exception as e:
            wrong.append(repr(e))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    for asm, _, _, _ in solvers:
        asm.close()
