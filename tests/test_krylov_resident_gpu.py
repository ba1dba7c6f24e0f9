"""CG and MINRES in resident kernels: one CTA (125 rows), rows around a CTA's 992 and the grid's 152 x 992,
more than one kernel's 200 iterations, both precisions, node groups of a warp and of half a warp (more than
31 groups a CTA), iteration limits that end inside a kernel, breakdown.  The solution is checked by its
FP64 residual formed in torch, against the tolerance the solver was given (its own FP64 residual meets it;
1 % is far above the rounding of forming it again).
"""
import numpy as np
import pytest
import torch

from iron_gb300._lib import GfeError
from iron_gb300.elasticity import MooneyRivlinAssembly
from iron_gb300.laplace import LaplaceAssembly
from iron_gb300.mesh import RegularMesh
from iron_gb300.newton import minres_solve, saddle_preconditioner

pytestmark = pytest.mark.gpu


def _matvec(row_ptr, col_idx, values, x):
    n = row_ptr.numel() - 1
    return torch.sparse_csr_tensor((row_ptr - 1).long(), (col_idx - 1).long(), values, (n, n)) @ x


def _laplace(ne, seed=0):
    m = RegularMesh(ne)
    m.jitter_interior(seed)
    kap = np.random.default_rng(seed + 1).uniform(0.1, 10.0, m.n_elements)
    A = LaplaceAssembly.from_regular_mesh(m, kappa=kap)
    fixed = np.zeros(m.n_nodes, np.uint8)
    x0 = np.zeros(m.n_nodes)
    fixed[m.face_nodes(0, 0)] = 1
    fixed[m.face_nodes(0, 1)] = 1
    x0[m.face_nodes(0, 1)] = 1.0
    return A, torch.from_numpy(fixed).cuda(), torch.from_numpy(x0).cuda()


@pytest.mark.parametrize("ne", [(1, 1, 1), (4, 4, 4), (9, 9, 9), (10, 9, 8), (31, 30, 32), (53, 52, 53), (60, 61, 59)])
@pytest.mark.parametrize("precision", ["fp64", "mixed_df"])
@pytest.mark.parametrize("with_f", [False, True])
def test_cg(gfe_cuda, ne, precision, with_f):
    A, fixed, x0 = _laplace(ne)
    v = A.assemble(precision, fp32_copy=True)
    free = (fixed == 0).double()
    f = torch.randn(A.n_nodes, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(1)) if with_f else None
    x = x0.clone()
    info = A.solve(fixed, x, f=f, rtol=1e-10, precision=precision)
    b = torch.zeros_like(x) if f is None else f
    r0 = (b - _matvec(A.row_ptr, A.col_idx, v, x0)) * free
    r = (b - _matvec(A.row_ptr, A.col_idx, v, x)) * free
    assert float(r.norm()) <= 1.01e-10 * float(r0.norm())
    assert torch.equal(x * (1 - free), x0)
    y = x0.clone()
    again = A.solve(fixed, y, f=f, rtol=1e-10, precision=precision)
    assert torch.equal(x, y) and again.iterations == info.iterations  # independent of scheduling


@pytest.mark.parametrize("precision", ["fp64", "mixed_df"])
def test_cg_iteration_limit_and_breakdown(gfe_cuda, precision):
    A, fixed, x0 = _laplace((12, 11, 13))
    A.assemble(precision, fp32_copy=True)
    with pytest.raises(GfeError, match="after 7 iterations"):
        A.solve(fixed, x0.clone(), rtol=1e-12, max_iters=7, precision=precision)
    A.values.neg_()
    A.values32.neg_()
    with pytest.raises(GfeError, match="breakdown"):
        A.solve(fixed, x0.clone(), rtol=1e-12, precision=precision)


@pytest.mark.parametrize("ne", [(1, 1, 1), (2, 2, 2), (5, 4, 3), (8, 8, 7)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nodal", [True, False])
def test_minres(gfe_cuda, ne, precision, nodal):
    A = MooneyRivlinAssembly.from_regular_mesh(ne)
    rng = np.random.default_rng(2)
    x = A.xg.cpu().numpy()
    z = x * np.array([1.05, 0.98, 0.97])[:, None] + rng.normal(0, 0.005 / max(ne), x.shape)
    dep = torch.from_numpy(np.r_[z.ravel(), np.zeros(A.n_lin)]).cuda()
    v = A.tangent(dep, [2.0, 6.0])
    fixed = np.zeros(A.ndof, np.uint8)
    for c in range(3):
        fixed[c * A.n_q2:(c + 1) * A.n_q2][x[0] == 0.0] = 1
    fixed = torch.from_numpy(fixed).cuda()
    free = (fixed == 0).double()
    f = torch.from_numpy(rng.normal(0, 1e-3, A.ndof)).cuda()
    minv = saddle_preconditioner(A.row_ptr, A.col_idx, v, 3 * A.n_q2, fixed)
    u = torch.zeros_like(f)
    info = minres_solve(A.row_ptr, A.col_idx, v, f, fixed, u, minv=minv, values32=v.float(), rtol=1e-6,
                        precision=precision, n_node=A.n_q2 if nodal else 0)
    assert info.nodal == (nodal and precision == "mixed")
    r, r0 = (f - _matvec(A.row_ptr, A.col_idx, v, u)) * free, f * free
    assert float((minv * r * r).sum().sqrt()) <= 1.01e-6 * float((minv * r0 * r0).sum().sqrt())
    w = torch.zeros_like(f)
    again = minres_solve(A.row_ptr, A.col_idx, v, f, fixed, w, minv=minv, values32=v.float(), rtol=1e-6,
                         precision=precision, n_node=A.n_q2 if nodal else 0)
    assert torch.equal(u, w) and again.iterations == info.iterations
    with pytest.raises(GfeError, match="after 3 iterations"):
        minres_solve(A.row_ptr, A.col_idx, v, f, fixed, u, minv=minv, values32=v.float(), rtol=1e-6, max_iters=3,
                     precision=precision, n_node=A.n_q2 if nodal else 0)
