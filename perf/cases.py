"""Performance cases of the finite-element engine: what a user's program has it do, through the
public entry points of iron_gb300.

Kinds of case (key "kind"):

  laplace   trilinear Laplace / diffusion assembly on a generated mesh (LaplaceAssembly.assemble):
            nx x ny x nz jittered hexahedra, one conductivity an element
  solve     the same assembly, then the Jacobi-CG solve with fixed faces (LaplaceAssembly.solve)
  bases     the basis-generic assembly: triquadratic ("q2") and tricubic ("q3") Lagrange and tricubic
            Hermite elements with arc-length scale factors ("hermite")
  tangent   Mooney-Rivlin consistent tangent assembled into CSR (MooneyRivlinAssembly.tangent)
  fd        Iron's finite-difference Jacobian (MooneyRivlinAssembly.jacobian_fd)
  adjoint   batched Mooney-Rivlin residual and its gradients through autograd (mr_residual)
  newton    a load step of the uniaxial stretch of a Mooney-Rivlin box (NewtonSolver.solve)

`prepare` builds what a program keeps (mesh, structure, slot map); `run` is one pass; `exact` gives the
same outputs in plain 64-bit torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from iron_gb300.elasticity import MooneyRivlinAssembly, mr_residual
from iron_gb300.laplace import LaplaceAssembly
from iron_gb300.mesh import HermiteMesh, RegularMesh, linear_component
from iron_gb300.newton import NewtonSolver, uniaxial_roller_conditions

F64 = torch.float64


def listed():
    return [
        # the smallest mesh of the serving stream and the smoke test: launches and host latency
        {"name": "laplace_4_fp64", "kind": "laplace", "nx": 4, "ny": 4, "nz": 4, "precision": "fp64"},
        # an ordinary mesh with odd, unequal sides, FP32 element arithmetic for a mixed-precision solve
        {"name": "laplace_ragged_mixed", "kind": "laplace", "nx": 45, "ny": 33, "nz": 51, "precision": "mixed"},
        # the plain FP64 element loop on a large mesh whose sides no tile divides
        {"name": "laplace_fp64", "kind": "laplace", "nx": 90, "ny": 77, "nz": 101, "precision": "fp64"},
        # the benchmark's headline mesh in its default precision
        {"name": "laplace_128_df", "kind": "laplace", "nx": 128, "ny": 128, "nz": 128, "precision": "mixed_df"},
        # a whole static linear problem: assembly and mixed-precision CG at the largest side served
        {"name": "laplace_solve_64", "kind": "solve", "nx": 64, "ny": 64, "nz": 64, "precision": "mixed_df"},
        # triquadratic elements, float-float
        {"name": "lagrange_q2_df", "kind": "bases", "basis": "q2", "nx": 36, "ny": 31, "nz": 33,
         "precision": "mixed_df"},
        # cubic Hermite elements with arc-length scale factors (64 parameters an element), FP64
        {"name": "hermite_fp64", "kind": "bases", "basis": "hermite", "nx": 13, "ny": 11, "nz": 12,
         "precision": "fp64"},
        # the Newton solver's Jacobian in mixed precision at the benchmark's size
        {"name": "mr_tangent_32_tf32x3", "kind": "tangent", "nx": 32, "ny": 32, "nz": 32, "precision": "tf32x3"},
        # the plain FP64 Jacobian, unequal sides
        {"name": "mr_tangent_fp64", "kind": "tangent", "nx": 15, "ny": 18, "nz": 13, "precision": "fp64"},
        # Iron's default Jacobian for finite elasticity
        {"name": "mr_fd", "kind": "fd", "nx": 9, "ny": 8, "nz": 7},
        # parameter estimation: residual and gradients for 64 parameter sets (forward and backward)
        {"name": "mr_adjoint_16x64", "kind": "adjoint", "nx": 16, "ny": 16, "nz": 16, "batch": 64},
        # one Mooney-Rivlin request of a serving stream: a load step to convergence
        {"name": "mr_newton_8", "kind": "newton", "nx": 8, "ny": 8, "nz": 8, "precision": "mixed"},
    ]


def _side(rng, lo, hi):
    """A side in [lo, hi], uniform in the logarithm."""
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _sides(rng, lo, hi):
    return {"nx": _side(rng, lo, hi), "ny": _side(rng, lo, hi), "nz": _side(rng, lo, hi)}


def draw(rng):
    kind = rng.choice(["laplace", "laplace", "solve", "bases", "bases", "tangent", "tangent", "fd", "adjoint", "newton"])
    if kind == "laplace":
        return {"kind": kind, **_sides(rng, 4, 128), "precision": rng.choice(["fp64", "mixed_df", "mixed"])}
    if kind == "solve":
        return {"kind": kind, **_sides(rng, 4, 64), "precision": rng.choice(["fp64", "mixed_df"])}
    if kind == "bases":
        basis = rng.choice(["q2", "q3", "hermite"])
        top = {"q2": 36, "q3": 14, "hermite": 13}[basis]
        return {"kind": kind, "basis": basis, **_sides(rng, 2, top),
                "precision": rng.choice(["fp64", "mixed_df", "mixed", "tf32x3"])}
    if kind == "tangent":
        precision = rng.choice(["fp64", "mixed", "tf32x3"])
        return {"kind": kind, **_sides(rng, 2, 18 if precision == "fp64" else 32), "precision": precision}
    if kind == "fd":
        return {"kind": kind, **_sides(rng, 2, 9)}
    if kind == "adjoint":
        return {"kind": kind, **_sides(rng, 2, 16), "batch": _side(rng, 1, 64)}
    return {"kind": kind, **_sides(rng, 2, 8), "precision": rng.choice(["fp64", "mixed"])}


# ---- inputs -------------------------------------------------------------------------------------

def _nelem(case):
    return case["nx"], case["ny"], case["nz"]


def _laplace_mesh(case, seed):
    """Jittered mesh and a conductivity log-uniform in [0.1, 10]."""
    basis = case.get("basis", "q1")
    if basis == "hermite":
        m = HermiteMesh(_nelem(case), scaling="arc_length")
    else:
        m = RegularMesh(_nelem(case), order=int(basis[1]))
    m.jitter_interior(seed)
    kappa = np.exp(np.random.default_rng(seed + 1).uniform(math.log(0.1), math.log(10.0), m.n_elements))
    return m, kappa


def _fixed_faces(m, seed):
    """Potential fixed on the two xi1 faces: 0 and a seeded value."""
    fixed = np.zeros(m.n_nodes, np.uint8)
    x0 = np.zeros(m.n_nodes)
    fixed[m.face_nodes(0, 0)] = 1
    fixed[m.face_nodes(0, 1)] = 1
    x0[m.face_nodes(0, 1)] = np.random.default_rng(seed + 2).uniform(0.5, 2.0)
    return fixed, x0


def _lateral_pressure(lam, c10, c01):
    """Pressure of the homogeneous stretch diag(lam, lam^-1/2, lam^-1/2) with free lateral faces."""
    lat = 1.0 / math.sqrt(lam)
    C = np.diag([lam * lam, 1.0 / lam, 1.0 / lam])
    S = 2.0 * (c10 + np.trace(C) * c01) * np.eye(3) - 2.0 * c01 * C
    F = np.diag([lam, lat, lat])
    sb = F @ S @ F.T
    return np.trace(sb) / 3.0 - sb[1, 1]


def _mr_grid(case):
    """(element nodes, pressure elements, coordinates, pressure nodes) of the Q2/Q1 box."""
    m = RegularMesh(_nelem(case), order=2)
    elin, lin2g = linear_component(m.elem_nodes, 2)
    return m.elem_nodes, elin, m.coords, len(lin2g)


def _mr_state(case, seed, x, n_lin, batch):
    """Stretched states with a nodal perturbation N(0, (0.01 h)^2), and material parameters."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    rng = np.random.default_rng(seed)
    if case["kind"] == "adjoint":
        c = np.exp(rng.uniform(math.log(0.5), math.log(10.0), (batch, 2)))
        lam = np.ones(batch)
    else:
        c = np.array([[2.0, 6.0]]) * rng.uniform(0.8, 1.25, (batch, 2))
        lam = rng.uniform(1.05, 1.15, batch)
    h = 1.0 / max(_nelem(case))
    xd = torch.as_tensor(x, dtype=F64, device="cuda")
    stretch = torch.as_tensor(np.stack([lam, lam ** -0.5, lam ** -0.5], axis=1), dtype=F64, device="cuda")
    z = xd[None] * stretch[:, :, None] + 0.01 * h * torch.randn((batch, *xd.shape), generator=g, dtype=F64, device="cuda")
    p = torch.as_tensor([_lateral_pressure(lam[b], *c[b]) for b in range(batch)], dtype=F64, device="cuda")
    dep = torch.cat([z.reshape(batch, -1), p[:, None].expand(batch, n_lin)], dim=1).contiguous()
    v = torch.randn(dep.shape, generator=g, dtype=F64, device="cuda")
    return dep, torch.as_tensor(c, dtype=F64, device="cuda"), v


def _newton_data(seed):
    rng = np.random.default_rng(seed)
    return rng.uniform(1.03, 1.10), rng.uniform(1.0, 3.0), rng.uniform(4.0, 8.0)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("laplace", "solve", "bases"):
        m, kappa = _laplace_mesh(case, seed)
        if case.get("basis") == "hermite":
            A = LaplaceAssembly.from_hermite_mesh(m, kappa=kappa)
        else:
            A = LaplaceAssembly.from_regular_mesh(m, kappa=kappa)
        state = {"case": case, "A": A}
        if kind == "solve":
            fixed, x0 = _fixed_faces(m, seed)
            state["fixed"], state["x0"] = torch.from_numpy(fixed).cuda(), torch.from_numpy(x0).cuda()
        return state
    A = MooneyRivlinAssembly.from_regular_mesh(_nelem(case), build_jacobian=kind != "adjoint")
    state = {"case": case, "A": A}
    if kind == "newton":
        lam, c10, c01 = _newton_data(seed)
        fixed, full = uniaxial_roller_conditions(A, lam)
        solver = NewtonSolver(A, [c10, c01], precision=case["precision"], absolute_tolerance=1e-12,
                              relative_tolerance=1e-12, solution_tolerance=0.0, linear_relative_tolerance=1e-6)
        state.update(solver=solver, fixed=fixed, full=full)
        return state
    dep, c, v = _mr_state(case, seed, A.xg.cpu().numpy(), A.n_lin, case.get("batch", 1))
    if kind == "adjoint":
        state.update(dep=dep.requires_grad_(), c=c.requires_grad_(), v=v)
    else:
        state.update(dep=dep[0].clone(), c=c[0].clone())
    return state


# ---- one pass -----------------------------------------------------------------------------------

def run(state):
    case, A = state["case"], state["A"]
    kind = case["kind"]
    if kind in ("laplace", "bases"):
        out = {"values": A.assemble(case["precision"]), "rhs": A.rhs}
        if case["precision"] != "fp64":
            out["values32"] = A.values32
        return out
    if kind == "solve":
        values = A.assemble(case["precision"])
        x = state["x0"].clone()
        A.solve(state["fixed"], x, precision=case["precision"])
        return {"values": values, "x": x}
    if kind == "tangent":
        return {"values": A.tangent(state["dep"], state["c"], precision=case["precision"])}
    if kind == "fd":
        return {"values": A.jacobian_fd(state["dep"], state["c"])}
    if kind == "adjoint":
        R = mr_residual(A, state["dep"], state["c"])
        g_dep, g_c = torch.autograd.grad(R, (state["dep"], state["c"]), grad_outputs=state["v"])
        return {"residual": R.detach(), "grad_dep": g_dep, "grad_c": g_c}
    dep = A.initial_state(0.0)
    state["solver"].solve(dep, state["fixed"], state["full"])
    return {"dep": dep}


# ---- what a pass cannot do without --------------------------------------------------------------

def _box_nnz(nelem, order):
    """Entries of the nodal matrix of a box of Lagrange elements of one order (product over axes of
    the 1D counts: a vertex couples to both neighbouring elements, an inner node to its own)."""
    nnz = 1
    for n in nelem:
        nnz *= 2 * (order + 1) + (n - 1) * (2 * order + 1) + n * (order - 1) * (order + 1)
    return nnz


def _mr_counts(case):
    n = _nelem(case)
    E = math.prod(n)
    nq, nl = math.prod(2 * s + 1 for s in n), math.prod(s + 1 for s in n)
    # displacement-pressure coupling per axis: a vertex of the grid sees up to 3 pressure nodes, an
    # inner node 2
    up = math.prod(2 * 2 + (s - 1) * 3 + s * 2 for s in n)
    nnz = 9 * _box_nnz(n, 2) + 2 * 3 * up + _box_nnz(n, 1)
    return E, nq, nl, nnz


def work(case):
    kind, n = case["kind"], _nelem(case)
    E = math.prod(n)
    if kind in ("laplace", "solve", "bases"):
        basis = case.get("basis", "q1")
        if basis == "hermite":
            nns, ng, ndof, nnz = 64, 64, 8 * math.prod(s + 1 for s in n), 64 * _box_nnz(n, 1)
        else:
            o = int(basis[1])
            nns = ng = (o + 1) ** 3
            ndof, nnz = math.prod(o * s + 1 for s in n), _box_nnz(n, o)
        byts = E * (4 * nns + 8) + ndof * (24 + 8) + nnz * (8 if case["precision"] == "fp64" else 12)
        if basis == "hermite":
            byts += 8 * E * nns
        if kind == "solve":
            byts += ndof * (1 + 8 + 8)
        # sum factorisation over the three directions, one symmetric half: an element's fewest sums
        p = round(nns ** (1 / 3))
        flops = E * (3 * 6 * p ** 4 * 2 + ng * 60 + (6 * p ** 5 + 9 * p ** 6 + 4 * p ** 7) * 2 // 2)
        return {"bytes": byts, "flops": flops}
    E, nq, nl, nnz = _mr_counts(case)
    ndof = 3 * nq + nl
    mesh = E * (27 * 4 + 8 * 4) + nq * 24
    if kind == "newton":
        return {"bytes": mesh + ndof * (8 + 1 + 8), "flops": E * 27 * 500}
    if kind == "adjoint":
        B = case["batch"]
        return {"bytes": mesh + B * (ndof * 8 * 4 + 32), "flops": E * B * (15 * 648 * 2 + 27 * 1200)}
    if kind == "fd":
        return {"bytes": mesh + ndof * 8 + nnz * 8, "flops": E * 89 * (3 * 648 * 2 + 27 * 150)}
    # tangent: point tensors, then the sum-factorised u-u block (symmetric half) and u-p
    return {"bytes": mesh + ndof * 8 + nnz * 8,
            "flops": E * (6 * 648 * 2 + 27 * 1500 + 5 * 17500 * 2 + 27 * 81 * 8 * 2)}


# ---- the same outputs in plain 64-bit torch -----------------------------------------------------

def _rule(n):
    """Gauss-Legendre points and weights on [0, 1]."""
    x, w = np.polynomial.legendre.leggauss(n)
    return (x + 1.0) / 2.0, w / 2.0


def _one_d(kind, t):
    """Values and slopes at t of the 1D functions of one direction: Lagrange order or "h" (cubic
    Hermite: node 0 value and slope, node 1 value and slope)."""
    if kind == "h":
        P = [np.array([2.0, -3.0, 0.0, 1.0]), np.array([1.0, -2.0, 1.0, 0.0]),
             np.array([-2.0, 3.0, 0.0, 0.0]), np.array([1.0, -1.0, 0.0, 0.0])]
    else:
        at = np.arange(kind + 1) / kind
        P = []
        for a in range(kind + 1):
            others = np.delete(at, a)
            P.append(np.poly(others) / np.prod(at[a] - others))
    return np.array([np.polyval(q, t) for q in P]), np.array([np.polyval(np.polyder(q), t) for q in P])


def _tables(kind, ng):
    """Gradients [points, 3, functions], values [points, functions] and weights [points] of the
    tensor-product basis, functions in Iron's order, points xi1 fastest."""
    x, w = _rule(ng)
    V, D = zip(*[_one_d(kind, t) for t in x])
    V, D = np.array(V), np.array(D)  # [point, function]
    if kind == "h":  # nodes xi1 fastest, then the derivative bits of each node
        fn = [tuple(2 * ((node >> d) & 1) + ((k >> d) & 1) for d in range(3)) for node in range(8) for k in range(8)]
    else:
        r = range(kind + 1)
        fn = [(a, b, c) for c in r for b in r for a in r]
    grad, val, wt = [], [], []
    for g3 in range(ng):
        for g2 in range(ng):
            for g1 in range(ng):
                g = (g1, g2, g3)
                wt.append(w[g1] * w[g2] * w[g3])
                val.append([V[g1][f[0]] * V[g2][f[1]] * V[g3][f[2]] for f in fn])
                grad.append([[math.prod((D if d == k else V)[g[d]][f[d]] for d in range(3)) for f in fn]
                             for k in range(3)])
    dev = {"dtype": F64, "device": "cuda"}
    return torch.tensor(grad, **dev), torch.tensor(val, **dev), torch.tensor(wt, **dev)


def _positions(dofs, n):
    """Position of every element entry in the row-by-row, column-sorted matrix, and the number of
    entries and the rows and columns of them."""
    keys = (dofs[:, :, None] * n + dofs[:, None, :]).reshape(-1)
    uniq, inv = torch.unique(keys, return_inverse=True)
    return inv.reshape(dofs.shape[0], -1), uniq.numel(), uniq


def _cross_rows(J):
    """Cofactors of J[..., 3, 3] (rows: cross products of its columns) and its determinant."""
    a, b, c = J[..., 0], J[..., 1], J[..., 2]
    cof = torch.stack([torch.linalg.cross(b, c), torch.linalg.cross(c, a), torch.linalg.cross(a, b)], dim=-2)
    return cof, (a * cof[..., 0, :]).sum(-1)


def _exact_laplace(case, seed):
    m, kappa = _laplace_mesh(case, seed)
    basis = case.get("basis", "q1")
    if basis == "hermite":
        en, x, scale = m.elem_params, m.params, torch.from_numpy(np.ascontiguousarray(m.scale)).cuda()
        grad, _, w = _tables("h", 4)
    else:
        en, x, scale = m.elem_nodes, m.coords, None
        grad, _, w = _tables(int(basis[1]), int(basis[1]) + 1)
    en = torch.from_numpy(en).cuda().long()
    x, kap = torch.from_numpy(x).cuda(), torch.from_numpy(kappa).cuda()
    n = x.shape[1]
    pos, nnz, uniq = _positions(en, n)
    values = torch.zeros(nnz, dtype=F64, device="cuda")
    step = max(1, (1 << 25) // (grad.shape[0] * en.shape[1]))
    for e0 in range(0, en.shape[0], step):
        nodes = en[e0:e0 + step]
        xe = x[:, nodes].permute(1, 0, 2)
        if scale is not None:
            xe = xe * scale[e0:e0 + step, None, :]
        J = torch.einsum("ecn,gan->egca", xe, grad)
        cof, det = _cross_rows(J)
        # rows of cof are det * grad(xi_a): K = sum_g w kappa / det (cof^T dphi_m) . (cof^T dphi_n)
        B = torch.einsum("egac,gan->egcn", cof, grad)
        s = w[None] * kap[e0:e0 + step, None] / det
        Bs = (B * s[:, :, None, None]).flatten(1, 2)
        K = torch.matmul(B.flatten(1, 2).transpose(1, 2), Bs)
        if scale is not None:
            sf = scale[e0:e0 + step]
            K = K * sf[:, :, None] * sf[:, None, :]
        values.index_add_(0, pos[e0:e0 + step].reshape(-1), K.reshape(-1))
    if case["kind"] != "solve":
        out = {"values": values, "rhs": torch.zeros(n, dtype=F64, device="cuda")}
        if case["precision"] != "fp64":
            out["values32"] = values.float()
        return out
    fixed, x0 = _fixed_faces(m, seed)
    rows, cols = uniq // n, uniq % n
    rp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rp[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
    K = torch.sparse_csr_tensor(rp, cols, values, (n, n))
    free = torch.from_numpy(fixed == 0).cuda()
    u = torch.from_numpy(x0).cuda()
    diag = torch.ones(n, dtype=F64, device="cuda")
    diag[rows[rows == cols]] = values[rows == cols]
    for _ in range(3):  # conjugate gradients, restarted from the true residual
        r = -(K @ u) * free
        z = r / diag
        p, rz, r0 = z.clone(), r @ z, float(r.norm())
        d = torch.zeros_like(u)
        for k in range(4000):
            q = (K @ p) * free
            a = rz / (p @ q)
            d += a * p
            r -= a * q
            if k % 20 == 19 and float(r.norm()) <= 1e-12 * r0:
                break
            z = r / diag
            rz, old = r @ z, rz
            p = z + (rz / old) * p
        u = u + d
    return {"values": values, "x": u}


def _mr_point(Z, p, X, w, c10, c01):
    """P[..., xi, mh] = w J_z Z^-1 sigma and the pressure-row density w (J_z - J_x) at points with
    deformed and reference gradients Z, X [..., component, xi]: the isochoric Mooney-Rivlin Cauchy
    stress, its deviator plus p, in the frame of the normalised reference tangents."""
    _, Jx = _cross_rows(X)
    cof, dz = _cross_rows(Z)
    Jx, Jz = Jx.abs(), dz.abs()
    N = X / X.norm(dim=-2, keepdim=True)
    A = torch.linalg.inv(N.transpose(-1, -2) @ X)
    J = Jz / Jx
    Fb = (Z @ A) * (J ** (-1.0 / 3.0))[..., None, None]
    C = Fb.transpose(-1, -2) @ Fb
    I = torch.eye(3, dtype=F64, device=Z.device)
    I1 = C.diagonal(dim1=-2, dim2=-1).sum(-1)
    S = -2.0 * c01[..., None, None] * C + (2.0 * (c10 + I1 * c01))[..., None, None] * I
    sg = Fb @ S @ Fb.transpose(-1, -2) / J[..., None, None]
    tr = sg.diagonal(dim1=-2, dim2=-1).sum(-1) / 3.0
    sg = sg + (p - tr)[..., None, None] * I
    P = (w * Jz / dz)[..., None, None] * (cof @ sg)
    return P, w * (Jz - Jx)


class _MR:
    """Element data of a Mooney-Rivlin box for the exact values."""

    def __init__(self, case):
        eq2, elin, x, self.nl = _mr_grid(case)
        self.eq2, self.elin = torch.from_numpy(eq2).cuda().long(), torch.from_numpy(elin).cuda().long()
        self.x = torch.from_numpy(x).cuda()
        self.nq = x.shape[1]
        self.grad, _, self.w = _tables(2, 3)
        xg, _ = _rule(3)
        hat = np.array([[1.0 - t, t] for t in xg])
        psi = [[hat[a][i] * hat[b][j] * hat[c][k] for k in (0, 1) for j in (0, 1) for i in (0, 1)]
               for c in range(3) for b in range(3) for a in range(3)]
        self.psi = torch.tensor(psi, dtype=F64, device="cuda")
        self.ndof = 3 * self.nq + self.nl
        e = self.eq2
        self.dofs = torch.cat([e, e + self.nq, e + 2 * self.nq, self.elin + 3 * self.nq], dim=1)
        self.X = torch.einsum("cen,gan->egca", self.x[:, self.eq2], self.grad)

    def points(self, ue):
        """Gradients and pressures at the points from element parameters ue [..., E, 89]."""
        z = ue[..., :81].unflatten(-1, (3, 27))
        return torch.einsum("...ecn,gan->...egca", z, self.grad), ue[..., 81:] @ self.psi.T

    def element_residual(self, ue, c10, c01):
        Z, p = self.points(ue)
        P, q = _mr_point(Z, p, self.X, self.w, c10, c01)
        return torch.cat([torch.einsum("...egam,gan->...emn", P, self.grad).flatten(-2), q @ self.psi], dim=-1)

    def assemble(self, Ke):
        pos, nnz, _ = _positions(self.dofs, self.ndof)
        return torch.zeros(nnz, dtype=F64, device="cuda").index_add_(0, pos.reshape(-1), Ke.reshape(-1))


def exact(case, seed):
    kind = case["kind"]
    if kind in ("laplace", "solve", "bases"):
        return _exact_laplace(case, seed)
    if kind == "newton":  # the homogeneous stretch solves the problem
        lam, c10, c01 = _newton_data(seed)
        x = _mr_grid(case)
        z = x[2] * np.array([lam, lam ** -0.5, lam ** -0.5])[:, None]
        return {"dep": torch.from_numpy(np.r_[z.ravel(), np.full(x[3], _lateral_pressure(lam, c10, c01))]).cuda()}
    M = _MR(case)
    batch = case.get("batch", 1)
    dep, c, v = _mr_state(case, seed, M.x.cpu().numpy(), M.nl, batch)
    if kind == "adjoint":
        R, gd, gc = [], [], []
        for b in range(batch):
            d, cb = dep[b].clone().requires_grad_(), c[b].clone().requires_grad_()
            re = M.element_residual(d[M.dofs], cb[0].expand(1, 1), cb[1].expand(1, 1))
            r = torch.zeros(M.ndof, dtype=F64, device="cuda").index_add(0, M.dofs.reshape(-1), re.reshape(-1))
            a, q = torch.autograd.grad(r, (d, cb), grad_outputs=v[b])
            R.append(r.detach())
            gd.append(a)
            gc.append(q)
        return {"residual": torch.stack(R), "grad_dep": torch.stack(gd), "grad_c": torch.stack(gc)}
    ue = dep[0][M.dofs]
    c10, c01 = c[0, 0].expand(1, 1), c[0, 1].expand(1, 1)
    E = ue.shape[0]
    Ke = torch.zeros((E, 89, 89), dtype=F64, device="cuda")
    if kind == "fd":
        delta = (1.0 + dep[0].norm()) * 1e-6
        r0 = M.element_residual(ue, c10, c01)
        for j in range(89):
            up = ue.clone()
            up[:, j] += delta
            Ke[:, :, j] = (M.element_residual(up, c10, c01) - r0) / delta
        Ke[:, 81:, 81:] = 0.0
        return {"values": M.assemble(Ke)}
    # derivatives of the point quantities in the nine gradient entries and the pressure, then the
    # contraction with the basis gradients
    Zall, pall = M.points(ue)
    G = M.grad
    step = 2048
    for e0 in range(0, E, step):
        Z, p, X = Zall[e0:e0 + step], pall[e0:e0 + step], M.X[e0:e0 + step]
        def point(Zt, pt, X=X):
            return _mr_point(Zt, pt, X, M.w, c10, c01)
        K = Ke[e0:e0 + step]
        for nh in range(3):
            for zeta in range(3):
                dZ = torch.zeros_like(Z)
                dZ[..., nh, zeta] = 1.0
                _, (dP, dq) = torch.func.jvp(point, (Z, p), (dZ, torch.zeros_like(p)))
                left = torch.einsum("egam,gai->emig", dP, G).flatten(1, 2)  # [e, (mh, ms), g]
                K[:, :81, 27 * nh:27 * nh + 27] += left @ G[:, zeta]
                K[:, 81:, 27 * nh:27 * nh + 27] += (dq[:, None, :] * M.psi.T[None]) @ G[:, zeta]
        _, (dP, _) = torch.func.jvp(point, (Z, p), (torch.zeros_like(Z), torch.ones_like(p)))
        K[:, :81, 81:] = torch.einsum("egam,gai->emig", dP, G).flatten(1, 2) @ M.psi
    return {"values": M.assemble(Ke)}
