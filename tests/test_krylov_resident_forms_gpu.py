"""Instances of the resident CG and MINRES kernels that the small meshes do not reach: 32-bit column offsets with one,
two and three slices of rows a warp (node numbers permuted, so that columns lie further than 32,767 from their row),
three slices with 16-bit ones on the 27-point stencil, and MINRES on matrices of which shared memory holds a part.  The
solution is checked by its FP64 residual formed in torch (1 % above the solver's tolerance is far more than
the rounding of forming it again) and against a second run, to the bit."""
import ctypes as C

import numpy as np
import pytest
import torch

from iron_gb300 import _lib
from iron_gb300.elasticity import MooneyRivlinAssembly
from iron_gb300.laplace import LaplaceAssembly
from iron_gb300.mesh import RegularMesh
from iron_gb300.newton import minres_solve, saddle_preconditioner

pytestmark = pytest.mark.gpu


def _matvec(row_ptr, col_idx, values, x):
    n = row_ptr.numel() - 1
    return torch.sparse_csr_tensor((row_ptr - 1).long(), (col_idx - 1).long(), values, (n, n)) @ x


def _permuted_stencil(m):
    """7-point operator of m nodes a side, node numbers permuted."""
    n = m ** 3
    i = np.random.default_rng(4).permutation(n).reshape(m, m, m)
    a = np.concatenate([i[1:].ravel(), i[:, 1:].ravel(), i[:, :, 1:].ravel()])
    b = np.concatenate([i[:-1].ravel(), i[:, :-1].ravel(), i[:, :, :-1].ravel()])
    r, c, v = np.r_[a, b, np.arange(n)], np.r_[b, a, np.arange(n)], np.r_[-np.ones(2 * len(a)), np.full(n, 6.05)]
    o = np.lexsort((c, r))
    ptr = np.r_[0, np.cumsum(np.bincount(r, minlength=n))]
    to = lambda x, t: torch.from_numpy(np.ascontiguousarray(x.astype(t))).cuda()  # noqa: E731
    return to(ptr + 1, np.int32), to(c[o] + 1, np.int32), to(v[o], np.float64)


def _cg(rp, ci, v, mixed, rtol):
    n = rp.numel() - 1
    f = torch.randn(n, dtype=torch.float64, generator=torch.Generator().manual_seed(3)).cuda()
    v32 = v.float() if mixed else None
    it, rel = C.c_int32(0), C.c_double(0.0)
    x = [torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(2)]
    for y in x:
        _lib.call("gfe_cg_solve", n, _lib.ptr(rp), _lib.ptr(ci), _lib.ptr(v), _lib.ptr(v32), _lib.ptr(f), None,
                  _lib.ptr(y), rtol, 20000, 1 if mixed else 0, C.byref(it), C.byref(rel), _lib.stream_handle(None))
    assert float((f - _matvec(rp, ci, v, x[0])).norm()) <= 1.01 * rtol * float(f.norm())
    assert torch.equal(x[0], x[1])


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("slices", [1, 2, 3])
def test_cg_far_columns(gfe_cuda, slices, mixed):
    rows = 32 * 31 * torch.cuda.get_device_properties(0).multi_processor_count
    sys = _permuted_stencil(int((rows * (slices - 0.3)) ** (1 / 3)))
    row = torch.repeat_interleave(torch.arange(sys[0].numel() - 1, device="cuda"), (sys[0][1:] - sys[0][:-1]).long())
    assert int((sys[1].long() - 1 - row).abs().max()) > 32767
    _cg(*sys, mixed, 1e-10)


@pytest.mark.parametrize("precision,ne", [("fp64", (66, 66, 68)), ("mixed_df", (67, 70, 65))])
def test_cg_three_slices_of_the_27_point_stencil(gfe_cuda, precision, ne):
    """As many rows as the byte limit admits, on 152 SMs about 310,000 (FP64) and 320,000."""
    m = RegularMesh(ne)
    m.jitter_interior(0)
    A = LaplaceAssembly.from_regular_mesh(m)
    v = A.assemble(precision, fp32_copy=True)
    fixed = np.zeros(m.n_nodes, np.uint8)
    fixed[m.face_nodes(0, 0)] = fixed[m.face_nodes(0, 1)] = 1
    x0 = np.zeros(m.n_nodes)
    x0[m.face_nodes(0, 1)] = 1.0
    fixed, x0 = torch.from_numpy(fixed).cuda(), torch.from_numpy(x0).cuda()
    free = (fixed == 0).double()
    x, y = x0.clone(), x0.clone()
    A.solve(fixed, x, rtol=1e-10, precision=precision)
    A.solve(fixed, y, rtol=1e-10, precision=precision)
    r0, r = (_matvec(A.row_ptr, A.col_idx, v, t) * free for t in (x0, x))
    assert float(r.norm()) <= 1.01e-10 * float(r0.norm())
    assert torch.equal(x, y)


@pytest.mark.parametrize("precision,nodal", [("mixed", True), ("mixed", False), ("fp64", False)])
def test_minres_beyond_shared_memory(gfe_cuda, precision, nodal):
    A = MooneyRivlinAssembly.from_regular_mesh((11, 11, 11))
    per = 4 if precision == "mixed" else 8
    assert A.nnz * (per + 4) <= 100 << 20 and A.nnz * (per + (4 / 3 if nodal else 4)) > 152 * (212 << 10)
    rng = np.random.default_rng(2)
    x = A.xg.cpu().numpy()
    z = x * np.array([1.05, 0.98, 0.97])[:, None] + rng.normal(0, 0.005 / 11, x.shape)
    v = A.tangent(torch.from_numpy(np.r_[z.ravel(), np.zeros(A.n_lin)]).cuda(), [2.0, 6.0])
    fixed = np.zeros(A.ndof, np.uint8)
    for c in range(3):
        fixed[c * A.n_q2:(c + 1) * A.n_q2][x[0] == 0.0] = 1
    fixed = torch.from_numpy(fixed).cuda()
    free = (fixed == 0).double()
    f = torch.from_numpy(rng.normal(0, 1e-3, A.ndof)).cuda()
    minv = saddle_preconditioner(A.row_ptr, A.col_idx, v, 3 * A.n_q2, fixed)
    u, w = torch.zeros_like(f), torch.zeros_like(f)
    infos = [minres_solve(A.row_ptr, A.col_idx, v, f, fixed, t, minv=minv, values32=v.float(), rtol=1e-5,
                          precision=precision, n_node=A.n_q2 if nodal else 0) for t in (u, w)]
    assert infos[0].nodal == nodal
    r, r0 = (f - _matvec(A.row_ptr, A.col_idx, v, u)) * free, f * free
    assert float((minv * r * r).sum().sqrt()) <= 1.01e-5 * float((minv * r0 * r0).sum().sqrt())
    assert torch.equal(u, w) and infos[0].iterations == infos[1].iterations
