"""Sum-factorised FP64 Mooney-Rivlin kernels at the edges of their size rules.

The finite-difference Jacobian splits an element over 1, 3 or 9 CTAs by the number of elements and
adds the columns all at once through element matrices (up to 4,096 elements) or colour by colour;
every branch is compared with the oracle's element matrices on sampled elements, and the assembled
values with the sum of the dense element matrices.  The FP64 tangent takes eight elements a CTA and the
contraction two CTAs an SM; it is compared with automatic differentiation of the element residual
written in plain torch, at element counts around those edges.  Tolerances: FP64 on both sides, summed in
different orders, 1e-12 x max|K| as in test_mr_gpu; residual and adjoint entries the same relative to
their largest, and dc, a sum over all elements, relative to the sum of the magnitudes it adds; the difference quotient amplifies the
rounding of two FP64 residuals by 1 / delta (1e-9 x max|K|, as in test_mr_fd_jacobian_gpu); sums of at
most 8 FP64 element entries in another order agree to 8 eps max|K|.
"""
import numpy as np
import pytest
import torch

import oracle
from iron_gb300.elasticity import MooneyRivlinAssembly

pytestmark = pytest.mark.gpu

C1, C2 = 2.0, 6.0
EPS = np.finfo(np.float64).eps


def _state(A, seed, amp=0.02):
    rng = np.random.default_rng(seed)
    x = A.xg.cpu().numpy()
    z = x * np.array([1.05, 0.98, 0.97])[:, None] + rng.normal(0, amp / max(A.mesh.nelem), x.shape)
    return np.r_[z.ravel(), -1.0 + rng.normal(0, 0.2, A.n_lin)]


def _element(A, dep, e):
    nq = A.n_q2
    en, el = A.mesh.elem_nodes[e], A.elin[e].cpu().numpy()
    return A.xg.cpu().numpy()[:, en], dep[: 3 * nq].reshape(3, nq)[:, en], dep[3 * nq:][el]


@pytest.mark.parametrize("ne", [(1, 1, 1), (8, 8, 7), (11, 10, 12), (17, 15, 17)])
def test_fd_jacobian_size_rules(gfe_cuda, ne):
    A = MooneyRivlinAssembly.from_regular_mesh(ne)
    dep = _state(A, 3)
    d = torch.from_numpy(dep).cuda()
    K = A.jacobian_fd(d, [C1, C2], dense=True)
    delta = (1.0 + np.linalg.norm(dep)) * 1e-6
    for e in sorted({0, A.n_elements // 3, A.n_elements - 1}):
        Ko = oracle.mr_element_jacobian_fd(*_element(A, dep, e), C1, C2, delta)
        assert np.abs(K[e].cpu().numpy() - Ko).max() <= 1e-9 * np.abs(Ko).max(), e
    v = A.jacobian_fd(d, [C1, C2])
    ref = torch.zeros_like(v).index_add_(0, A.slots.reshape(-1).long(), K.reshape(-1))
    assert float((v - ref).abs().max()) <= 8 * EPS * float(K.abs().max())


def _point_tables():
    """Basis gradients [27, 3, 27], pressure functions [27, 8] and weights [27], xi1 fastest."""
    x, w = np.polynomial.legendre.leggauss(3)
    x, w = (x + 1) / 2, w / 2
    V = np.stack([2 * (x - 0.5) * (x - 1), 4 * x * (1 - x), 2 * x * (x - 0.5)], axis=1)
    D = np.stack([4 * x - 3, 4 - 8 * x, 4 * x - 1], axis=1)
    L = np.stack([1 - x, x], axis=1)
    kron = lambda a, b, c: np.einsum("gi,hj,kl->khglji", a, b, c).reshape(27, -1)  # noqa: E731
    G = np.stack([kron(D, V, V), kron(V, D, V), kron(V, V, D)], axis=1)
    return torch.from_numpy(G), torch.from_numpy(kron(L, L, L)), torch.from_numpy(np.einsum("g,h,k->khg", w, w, w).ravel())


def _torch_residual(u, xe, c=(C1, C2)):
    G, psi, w = _point_tables()
    Z = torch.einsum("cn,gkn->gck", u[:81].reshape(3, 27), G)
    X = torch.einsum("cn,gkn->gck", xe, G)
    Jz, Jx = torch.linalg.det(Z).abs(), torch.linalg.det(X).abs()
    N = X / X.norm(dim=1, keepdim=True)
    F = Z @ torch.linalg.inv(N.transpose(1, 2) @ X)
    J = Jz / Jx
    Fb = F * J[:, None, None] ** (-1.0 / 3.0)
    C = Fb.transpose(1, 2) @ Fb
    eye = torch.eye(3, dtype=torch.float64)
    I1 = C.diagonal(dim1=1, dim2=2).sum(1)
    S = -2 * c[1] * C + 2 * (c[0] + I1 * c[1])[:, None, None] * eye
    sg = Fb @ S @ Fb.transpose(1, 2) / J[:, None, None]
    p = psi @ u[81:]
    sg = sg + (p - sg.diagonal(dim1=1, dim2=2).sum(1) / 3)[:, None, None] * eye
    P = (w * Jz)[:, None, None] * (torch.linalg.inv(Z) @ sg)
    return torch.cat([torch.einsum("gkm,gkn->mn", P, G).reshape(-1), (w * (Jz - Jx)) @ psi])


@pytest.mark.parametrize("ne", [(1, 1, 1), (7, 1, 1), (2, 2, 2), (3, 3, 1), (7, 8, 6)])
def test_tangent_fp64_element_counts(gfe_cuda, ne):
    A = MooneyRivlinAssembly.from_regular_mesh(ne, extent=(1.0, 1.3, 0.8))
    dep = _state(A, 5)
    d = torch.from_numpy(dep).cuda()
    K = A.element_tangents(d, [C1, C2], precision="fp64")
    for e in sorted({0, A.n_elements // 2, A.n_elements - 1}):
        xe, ze, pe = _element(A, dep, e)
        u = torch.from_numpy(np.r_[ze.ravel(), pe])
        Kt = torch.autograd.functional.jacobian(lambda v: _torch_residual(v, torch.from_numpy(xe)), u)
        assert float((K[e].cpu() - Kt).abs().max()) <= 1e-12 * float(Kt.abs().max()), e
    v = A.tangent(d, [C1, C2], precision="fp64")
    ref = torch.zeros_like(v).index_add_(0, A.slots.reshape(-1).long(), K.reshape(-1))
    assert float((v - ref).abs().max()) <= 8 * EPS * float(K.abs().max())


@pytest.mark.parametrize("ne,batch", [((1, 1, 1), 1), ((7, 1, 1), 3), ((3, 3, 1), 2), ((5, 4, 3), 17), ((13, 12, 11), 230)])
def test_residual_and_adjoint_sizes(gfe_cuda, ne, batch):
    """Element counts around a CTA's eight, batches around its share of sets; the last size exceeds the
    scratch of the all-at-once form and adds colour by colour."""
    A = MooneyRivlinAssembly.from_regular_mesh(ne, extent=(1.0, 0.7, 1.2), build_jacobian=False)
    rng = np.random.default_rng(11)
    dep = np.stack([_state(A, 20 + b % 3) for b in range(batch)])
    c = np.tile([[C1, C2]], (batch, 1))
    v = rng.normal(0, 1, dep.shape)
    d, cd, vd = (torch.from_numpy(t).cuda() for t in (dep, c, v))
    R = A.residual(d, cd).cpu().numpy()
    du, dc = (t.cpu().numpy() for t in A.residual_vjp(d, cd, vd))
    nq, eq2, elin = A.n_q2, A.mesh.elem_nodes, A.elin.cpu().numpy()
    for b in sorted({0, batch - 1}):
        Ro = oracle.mr_assemble_residual(eq2, elin, nq, A.n_lin, A.xg.cpu().numpy(), dep[b], [C1, C2])
        assert np.abs(R[b] - Ro).max() <= 1e-12 * np.abs(Ro).max()
        Vo, dco, mag = np.zeros(A.ndof), np.zeros(2), np.zeros(2)
        for e in range(A.n_elements if A.n_elements < 100 else 0):
            xe, ze, pe = _element(A, dep[b], e)
            dofs = np.r_[eq2[e], eq2[e] + nq, eq2[e] + 2 * nq, elin[e] + 3 * nq]
            u = torch.from_numpy(np.r_[ze.ravel(), pe]).requires_grad_()
            cc = torch.tensor([C1, C2], dtype=torch.float64, requires_grad=True)
            r = _torch_residual(u, torch.from_numpy(xe), cc)
            gu, gc = torch.autograd.grad(r, (u, cc), torch.from_numpy(v[b][dofs]))
            Vo[dofs] += gu.numpy()
            dco += gc.numpy()
            mag += np.abs(gc.numpy())
        if A.n_elements < 100:
            assert np.abs(du[b] - Vo).max() <= 1e-12 * np.abs(Vo).max()
            assert (np.abs(dc[b] - dco) <= 1e-12 * mag).all()
    # one parameter set alone gives the same bits as in the batch
    k = batch - 1
    assert np.array_equal(A.residual(d[k], cd[k]).cpu().numpy(), R[k])
    du1, dc1 = A.residual_vjp(d[k:k + 1], cd[k:k + 1], vd[k:k + 1])
    assert np.array_equal(du1[0].cpu().numpy(), du[k]) and np.array_equal(dc1[0].cpu().numpy(), dc[k])
