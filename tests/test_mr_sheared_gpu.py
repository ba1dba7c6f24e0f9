"""FP64 Mooney-Rivlin kernels on reference meshes that are not boxes: sheared by 1, 3 and 10 in two
planes, and jittered and curved.

The residual, its adjoint, the consistent tangent and the finite-difference Jacobian are compared with the
same formulas in Iron's order of operations (F = Z (N^T X)^-1) in extended precision (numpy longdouble;
derivatives by complex steps, exact to its rounding).  The reference gradients of a sheared element are
ill-conditioned, so FP64 itself loses digits there; how many is measured by the same reference code in FP64.
One Gauss point can carry most of the error, so one evaluation in FP64 is a poor measure of it (two of them
differ by up to 2.5); the largest of three is taken, with the element's xi directions in each cyclic order,
which leaves the exact result as it is.  Errors of the same conditioning stay within a small factor of each
other (at a single point at most 2 in the median over shears of 1 to 100): a factor of 4 is allowed, and
64 eps (a chain of about as many operations) where FP64 loses nothing.
"""
import numpy as np
import pytest
import torch

from iron_gb300.elasticity import MooneyRivlinAssembly

pytestmark = pytest.mark.gpu

C = np.array([2.0, 6.0])
EPS = np.finfo(np.float64).eps
LD, CLD = np.longdouble, np.clongdouble


def _tables(T):
    t = np.sqrt(T(6) / T(10)) / 2
    x, w = np.array([T(1) / 2 - t, T(1) / 2, T(1) / 2 + t]), np.array([T(5), T(8), T(5)]) / 18
    V = np.stack([2 * (x - T(1) / 2) * (x - 1), 4 * x * (1 - x), 2 * x * (x - T(1) / 2)], axis=1)
    D = np.stack([4 * x - 3, 4 - 8 * x, 4 * x - 1], axis=1)
    L = np.stack([1 - x, x], axis=1)
    kron = lambda a, b, c: np.einsum("gi,hj,kl->khglji", a, b, c).reshape(27, -1)  # noqa: E731
    return (np.stack([kron(D, V, V), kron(V, D, V), kron(V, V, D)], axis=1), kron(L, L, L),
            np.einsum("g,h,k->khg", w, w, w).ravel())


def _cof(M):
    """Cofactors and determinant of M[..., c, k]."""
    a, b, c = M[..., 0, :], M[..., 1, :], M[..., 2, :]
    cross = lambda u, v: np.stack([u[..., 1] * v[..., 2] - u[..., 2] * v[..., 1],  # noqa: E731
                                   u[..., 2] * v[..., 0] - u[..., 0] * v[..., 2],
                                   u[..., 0] * v[..., 1] - u[..., 1] * v[..., 0]], axis=-1)
    co = np.stack([cross(b, c), cross(c, a), cross(a, b)], axis=-2)
    return co, (a * co[..., 0, :]).sum(-1)


def _inv(M):
    co, det = _cof(M)
    return co.swapaxes(-1, -2) / det[..., None, None]


def _residual(u, xe, c, T):
    """Element residual [..., 89] from u[..., 89]; T: the real type, u may be of its complex type."""
    G, psi, w = _tables(T)
    mm = lambda a, b: (a[..., :, :, None] * b[..., None, :, :]).sum(-2)  # noqa: E731
    Z = (u[..., :81].reshape(*u.shape[:-1], 1, 3, 1, 27) * G[:, None]).sum(-1)
    X = (xe.astype(T)[None, :, None, :] * G[:, None]).sum(-1)
    Zi, Jz, Jx = _inv(Z), _cof(Z)[1], _cof(X)[1]  # det Z > 0 in these states
    N = X / np.sqrt((X * X).sum(-2, keepdims=True))
    F = mm(Z, _inv(mm(N.swapaxes(-1, -2), X)))
    J = Jz / Jx
    Fb = F * (J ** (-T(1) / T(3)))[..., None, None]
    Cg = mm(Fb.swapaxes(-1, -2), Fb)
    eye = np.eye(3, dtype=T)
    tr = lambda A: A[..., 0, 0] + A[..., 1, 1] + A[..., 2, 2]  # noqa: E731
    S = -2 * c[1] * Cg + (2 * (c[0] + tr(Cg) * c[1]))[..., None, None] * eye
    sg = mm(mm(Fb, S), Fb.swapaxes(-1, -2)) / J[..., None, None]
    p = (u[..., None, 81:] * psi).sum(-1)
    sg = sg + (p - tr(sg) / 3)[..., None, None] * eye
    P = (w * Jz)[..., None, None] * mm(Zi, sg)  # [..., g, k, m]
    R = (P.swapaxes(-1, -2)[..., None, :] * np.moveaxis(G, 1, 2)[:, None]).sum((-1, -4))  # [..., m, n]
    return np.concatenate([R.reshape(*u.shape[:-1], 81), ((w * (Jz - Jx))[..., None] * psi).sum(-2)], axis=-1)


def _jacobian(u, xe, T):
    """dR/du [89, 89] and dR/dc [89, 2] by complex steps."""
    CT, h = (CLD, T(1e-30)) if T is LD else (np.complex128, T(1e-30))
    c = C.astype(T)
    K = np.stack([_residual(u.astype(T) + (1j * h * np.eye(89, dtype=T)[j]).astype(CT), xe, c, T).imag / h
                  for j in range(89)], axis=1)
    dc = np.stack([_residual(u.astype(CT), xe, c.astype(CT) + (1j * h * np.eye(2, dtype=T)[q]).astype(CT), T).imag / h
                   for q in range(2)], axis=1)
    return K, dc


def _fd(u, xe, delta, T):
    c = C.astype(T)
    up = u[None] + delta * np.eye(89)  # rounded to FP64, as the step is taken
    R0 = _residual(u.astype(T), xe, c, T)
    return np.stack([(_residual(up[j].astype(T), xe, c, T) - R0) / T(delta) for j in range(89)], axis=1)


def _problem(shape):
    A = MooneyRivlinAssembly.from_regular_mesh((2, 1, 1), extent=(1.0, 0.7, 0.6))
    rng = np.random.default_rng(7)
    x = A.xg.cpu().numpy()
    jit = rng.uniform(-0.02, 0.02, (2,) + x.shape)
    S = np.eye(3)
    if shape == "curved":
        x = x + 0.08 * np.sin(2.0 * np.roll(x, 1, axis=0) + 0.3)
    else:
        S[0, 1] = S[1, 2] = float(shape)
    xg = S @ (x + jit[0])
    F = np.array([[1.05, 0.1, 0.0], [0.0, 0.98, 0.05], [0.02, 0.0, 0.97]])
    dep = np.r_[(F @ S @ (x + jit[0] + jit[1])).ravel(), -1.0 + rng.normal(0, 0.2, A.n_lin)]
    A.xg.copy_(torch.from_numpy(xg))
    en, el = A.mesh.elem_nodes, A.elin.cpu().numpy()
    elems = []
    for e in range(A.n_elements):
        u = np.r_[dep[: 3 * A.n_q2].reshape(3, -1)[:, en[e]].ravel(), dep[3 * A.n_q2:][el[e]]]
        dofs = np.r_[en[e], en[e] + A.n_q2, en[e] + 2 * A.n_q2, 3 * A.n_q2 + el[e]]
        elems.append((u, xg[:, en[e]], dofs))
    return A, dep, elems


# element parameters with the xi directions in each cyclic order
_CYCLES = [np.concatenate([27 * c + np.arange(27).reshape(3, 3, 3).transpose(p).ravel() for c in range(3)] +
                          [81 + np.arange(8).reshape(2, 2, 2).transpose(p).ravel()])
           for p in ((0, 1, 2), (1, 2, 0), (2, 0, 1))]


def _element_values(u, xe, v, delta, T, cycle):
    """Residual, Jacobian, FD Jacobian, v^T dR/du and v^T dR/dc of one element, evaluated in T."""
    up, xp, inv = u[cycle], xe[:, cycle[:27]], np.argsort(cycle)
    K, dc = _jacobian(up, xp, T)
    K, dc = K[inv][:, inv], dc[inv]
    return (_residual(up.astype(T), xp, C.astype(T), T)[inv], K, _fd(up, xp, delta, T)[inv][:, inv],
            v.astype(T) @ K, v.astype(T) @ dc)


def _close(got, exact, own, what):
    n = np.sqrt((exact.astype(np.float64) ** 2).sum())
    err = lambda a: float(np.sqrt((((a.astype(LD) - exact) ** 2).sum()).astype(np.float64))) / n  # noqa: E731
    g, o = err(got), max(err(a) for a in own)
    assert g <= 4 * o + 64 * EPS, f"{what}: {g:.2e}, the reference's own FP64 error {o:.2e}"


@pytest.mark.parametrize("shape", [1, 3, 10, "curved"])
def test_fp64_kernels_on_sheared_and_curved_meshes(gfe_cuda, shape):
    A, dep, elems = _problem(shape)
    d = torch.from_numpy(dep).cuda()
    v = np.random.default_rng(8).normal(0, 1, A.ndof)
    K = A.element_tangents(d, C, precision="fp64").cpu().numpy()
    Kf = A.jacobian_fd(d, C, dense=True).cpu().numpy()
    delta = (1.0 + np.linalg.norm(dep)) * 1e-6
    runs = [(LD, _CYCLES[0])] + [(np.float64, c) for c in _CYCLES]
    R, du, dc = [[np.zeros(n, T) for T, _ in runs] for n in (A.ndof, A.ndof, 2)]
    for e, (u, xe, dofs) in enumerate(elems):
        vals = [_element_values(u, xe, v[dofs], delta, T, c) for T, c in runs]
        for i, val in enumerate(vals):
            R[i][dofs] += val[0]
            du[i][dofs] += val[3]
            dc[i] += val[4]
        _close(K[e], vals[0][1], [x[1] for x in vals[1:]], "tangent")
        _close(Kf[e], vals[0][2], [x[2] for x in vals[1:]], "finite-difference Jacobian")
    _close(A.residual(d, C).cpu().numpy(), R[0], R[1:], "residual")
    gu, gc = A.residual_vjp(d[None], torch.from_numpy(C[None]).cuda(), torch.from_numpy(v[None]).cuda())
    _close(gu[0].cpu().numpy(), du[0], du[1:], "adjoint")
    _close(gc[0].cpu().numpy(), dc[0], dc[1:], "cotangent of the constants")
