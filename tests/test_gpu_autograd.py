"""ElasticForce (torch.autograd.Function): forward = assembled gradient, backward =
the adjoint kernels, checked against the CPU oracle and central finite differences."""
import numpy as np
import pytest

from polyfem_b200 import NeoHookeanAssembler
from polyfem_b200 import mesh as M

from _cases import make_case, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("et", [M.P1_TET, M.P2_TET, M.Q1_HEX], ids=["P1", "P2", "Q1"])
def test_backward_equals_oracle_adjoint_terms(require_gpu, et):
    import torch

    from oracle.binding import Oracle
    from polyfem_b200.autograd import elastic_force

    mesh, lam, mu, u, p = make_case(et, 2, seed=21, jitter=0.1)
    asm = NeoHookeanAssembler.from_mesh(mesh, lam, mu)
    orc = Oracle(mesh, lam, mu)
    t = lambda a, g=True: torch.tensor(a, dtype=torch.float64, device="cuda", requires_grad=g)
    ut, lt, mt, Xt = t(u), t(lam), t(mu), t(mesh.X)
    pt = t(p, False)
    f = elastic_force(ut, lt, mt, Xt, asm)
    assert rel_err(f.detach().cpu().numpy(), orc.gradient(u)) <= 1e-12
    (f * pt).sum().backward()
    E = mesh.n_elements
    term = orc.material_vjp(u, p)
    assert rel_err(lt.grad.cpu().numpy(), -term[:E]) <= 1e-12
    assert rel_err(mt.grad.cpu().numpy(), -term[E:]) <= 1e-12
    assert rel_err(Xt.grad.cpu().numpy().ravel(), orc.shape_vjp(u, p)) <= 1e-12
    outer, inner, vals = orc.hessian(u)
    import scipy.sparse as sp
    Hp = sp.csc_matrix((vals, inner, outer), shape=(mesh.n_dofs, mesh.n_dofs)) @ p
    assert rel_err(ut.grad.cpu().numpy(), Hp) <= 1e-12
    asm.close()


def test_backward_matches_central_differences(require_gpu):
    import torch

    from polyfem_b200.autograd import elastic_force

    mesh, lam, mu, u, p = make_case(M.P2_TET, 2, seed=23, jitter=0.1)
    asm = NeoHookeanAssembler.from_mesh(mesh, lam, mu)
    dev = "cuda"
    base = [torch.tensor(a, dtype=torch.float64, device=dev) for a in (u, lam, mu, mesh.X)]
    pt = torch.tensor(p, dtype=torch.float64, device=dev)
    leaves = [b.clone().requires_grad_(True) for b in base]
    (elastic_force(*leaves, asm) * pt).sum().backward()

    def phi(args):
        with torch.no_grad():
            return float((elastic_force(*args, asm) * pt).sum())

    rng = np.random.default_rng(4)
    steps = [1e-6 * mesh.h, 1e-6 * float(np.median(lam)), 1e-6 * float(np.median(mu)), 1e-6 * mesh.h]
    for k in range(4):
        g = leaves[k].grad.cpu().numpy().ravel()
        for idx in rng.choice(g.size, 4, replace=False):
            plus = [b.clone() for b in base]
            minus = [b.clone() for b in base]
            plus[k].view(-1)[idx] += steps[k]
            minus[k].view(-1)[idx] -= steps[k]
            fd = (phi(plus) - phi(minus)) / (2 * steps[k])
            scale = max(abs(fd), 1e-3 * np.abs(g).max())
            assert abs(g[idx] - fd) <= 1e-5 * scale, (k, idx, g[idx], fd)
    asm.close()


@pytest.mark.parametrize("et", [M.P1_TET, M.P2_TET, M.Q1_HEX], ids=["P1", "P2", "Q1"])
@pytest.mark.parametrize("g", [1, 3, 4])
def test_hessian_vector_equals_assembled_product(require_gpu, et, g):
    """H(u) p without the matrix against the assembled FP64 Hessian times p on shuffled
    meshes (element counts off the block size), in host and device memory; NaN exactly on
    the rows of inverted elements; refused for another formulation."""
    import torch

    from polyfem_b200 import PfgError
    from _cases import permuted
    mesh, lam, mu, u, p = make_case(et, g, seed=31, jitter=0.1 if g > 1 else 0.0)
    m2, u2, _, pe = permuted(mesh, u, seed=2)
    asm = NeoHookeanAssembler.from_mesh(m2, lam[pe], mu[pe])
    H = asm.assemble_hessian(u2)
    q = asm.hessian_vector(u2, p)
    assert rel_err(q, H @ p) <= 1e-13
    dev = lambda a: torch.tensor(a, device="cuda")
    assert np.array_equal(asm.hessian_vector(dev(u2), dev(p)).cpu().numpy(), q)
    flipped = u2.copy()
    flipped.reshape(-1, 3)[m2.conn[0, 0]] += 3.0  # inverts elements around one node
    bad = np.isnan(asm.hessian_vector(flipped, p))
    Hn = asm.assemble_hessian(flipped).tocsr()
    assert np.array_equal(bad, np.isnan(Hn @ p)) and bad.any()
    asm.set_material("SaintVenant")
    with pytest.raises(PfgError):
        asm.hessian_vector(u2, p)
    asm.close()


@pytest.mark.parametrize("et", [M.P1_TET, M.P2_TET, M.Q1_HEX], ids=["P1", "P2", "Q1"])
def test_backward_leaves_its_hessian_in_the_context(require_gpu, et):
    """After a backward the context's matrix is H at the u, lambda, mu and X of that backward,
    whatever was set, evaluated or overwritten in place since; a later assembly replaces it, an
    assembly into the caller's array does not; and a captured backward leaves the matrix of
    each replay."""
    import ctypes

    import torch

    from polyfem_b200 import PfgError, _lib
    from polyfem_b200.autograd import elastic_force

    mesh, lam, mu, u, p = make_case(et, 3, seed=5, jitter=0.1)
    t = lambda a: torch.tensor(a, dtype=torch.float64, device="cuda")
    X = np.ascontiguousarray(mesh.X).reshape(-1)

    def assembled(u_, lam_, mu_, X_):
        ref = NeoHookeanAssembler.from_mesh(mesh, lam_, mu_)
        ref.set_rest_positions(t(X_))
        v = ref.assemble_hessian_values(t(u_))
        ref.close()
        return v

    def backward(asm, u_, lam_, mu_, X_):
        leaves = [t(a).requires_grad_(True) for a in (u_, lam_, mu_, X_)]
        (elastic_force(*leaves, asm) * t(p)).sum().backward()
        return leaves

    asm = NeoHookeanAssembler.from_mesh(mesh, lam, mu)
    leaves = backward(asm, u, lam, mu, X)
    with torch.no_grad():
        for a in leaves:
            a.data.mul_(1.5)  # an optimiser's step
        elastic_force(*leaves, asm)  # the next forward, other parameters
    v = assembled(u, lam, mu, X)
    asm.assemble_hessian_values(t(0.5 * u))  # into the caller's array
    asm.set_material("SaintVenant")
    asm.assemble_gradient(t(u))
    q = asm.hessian_apply(t(p))
    assert torch.equal(q, asm.hessian_apply(t(p), v))
    asm.set_material("NeoHookean")
    ptr = ctypes.c_void_p()
    _lib.check(_lib.lib().pfg_hessian_device_csc(asm.handle, None, None, ctypes.byref(ptr)), asm.handle, "csc")
    assert ptr.value
    # another backward, then an assembly that replaces its matrix
    backward(asm, 0.7 * u, 2 * lam, mu, X)
    assert torch.equal(asm.hessian_apply(t(p)), asm.hessian_apply(t(p), assembled(0.7 * u, 2 * lam, mu, X)))
    backward(asm, u, lam, mu, X)
    asm.assemble_hessian_into_context(t(0.3 * u))
    assert torch.equal(asm.hessian_apply(t(p)), asm.hessian_apply(t(p), assembled(0.3 * u, lam, mu, X)))
    asm.close()

    # the first read is the solver's
    asm = NeoHookeanAssembler.from_mesh(mesh, lam, mu)
    backward(asm, 0 * u, lam, mu, X)
    from polyfem_b200 import ConjugateGradient
    cg = ConjugateGradient(asm, "full")
    cg.set_parameters({"max_iter": 7, "tolerance": 0.0})
    b = t(p)
    x = cg.solve(b)
    cg.factorize(assembled(0 * u, lam, mu, X))
    assert torch.equal(cg.solve(b), x)
    asm.close()

    # captured
    asm = NeoHookeanAssembler.from_mesh(mesh, lam, mu)
    leaves = backward(asm, u, lam, mu, X)
    graph = torch.cuda.CUDAGraph()
    qq, pp = asm.hessian_vector(t(u), t(p)), t(p)
    with torch.cuda.graph(graph):
        qq.add_(0.0)
        with pytest.raises(PfgError):  # its first read cannot be part of a graph
            asm.hessian_apply(pp)
    asm.hessian_apply(t(p))  # buffers of the first call
    uu, pp = t(u), t(p)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        asm.hessian_later(uu)
    for f in (1.0, 0.4):
        uu.copy_(t(f * u))
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(asm.hessian_apply(pp), asm.hessian_apply(pp, assembled(f * u, lam, mu, X)))
    asm.close()
