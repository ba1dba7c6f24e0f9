"""Sum-factorised basis-generic assembly (quadratic and cubic hexahedra, FP64 and float-float) against the
oracle: every mixture of cubic Lagrange and cubic Hermite directions (element parameter order and scale
factors), element counts around the kernel's forms (all elements at once through scratch, or colour by
colour beyond 256 MB of element matrices), with the slot map and with the row search.  Tolerance 1e-12
relative to max|K|, as for the same precisions in test_laplace_tp_gpu.
"""
import itertools

import numpy as np
import pytest
import torch

import oracle
from iron_gb300.laplace import LaplaceAssembly
from iron_gb300.mesh import RegularMesh

pytestmark = pytest.mark.gpu


def _separate_elements(order, E, seed):
    """E disjoint curved elements of one basis: parameters of a perturbed identity map."""
    rng = np.random.default_rng(seed)
    nn = [2 if o == 4 else o + 1 for o in order]
    herm = [d for d in range(3) if order[d] == 4]
    rows = []
    for a3, a2, a1 in itertools.product(range(nn[2]), range(nn[1]), range(nn[0])):
        for k in range(2 ** len(herm)):
            on = [d for i, d in enumerate(herm) if (k >> i) & 1]
            at = (a1, a2, a3)
            rows.append([at[c] / (nn[c] - 1) if not on else float(on == [c]) for c in range(3)])
    base = np.array(rows).T  # [3][nns]
    nns = base.shape[1]
    x = base[:, None, :] + rng.uniform(-0.02, 0.02, (3, E, nns))
    return np.arange(E * nns, dtype=np.int32).reshape(E, nns), x.reshape(3, -1), rng.uniform(0.8, 1.25, (E, nns)), rng


@pytest.mark.parametrize("order", [(2, 2, 2), (3, 3, 3), (4, 4, 4), (4, 3, 3), (3, 4, 3), (3, 3, 4), (3, 4, 4), (4, 3, 4)])
@pytest.mark.parametrize("precision", ["fp64", "mixed_df"])
@pytest.mark.parametrize("E,slot_map,scaled", [(1, True, False), (5, False, True)])
def test_bases_match_oracle(gfe_cuda, order, precision, E, slot_map, scaled):
    ep, x, sf, rng = _separate_elements(order, E, 3)
    kap = rng.uniform(0.5, 2.0, E)
    ng = [o + 1 if o < 4 else 4 for o in order]
    scale = sf if scaled else None
    if scaled:  # scaled parameters interpolate the same geometry
        x = x / sf.reshape(1, -1)
    A = LaplaceAssembly(ep, x, kappa=kap, order=order, n_gauss=ng, scale=scale, slot_map=slot_map)
    v = A.assemble(precision).cpu().numpy()
    rp, ci = oracle.csr_structure(ep, x.shape[1])
    ov = oracle.laplace_assemble_scaled(3, list(order), ng, ep, x, scale, kap, rp, ci, 1)
    assert np.abs(v - ov).max() <= 1e-12 * np.abs(ov).max()


@pytest.mark.parametrize("precision", ["fp64", "mixed_df"])
@pytest.mark.parametrize("order,ne", [(2, (46, 45, 44)), (3, (26, 25, 25))])
def test_colour_by_colour_beyond_scratch(gfe_cuda, order, ne, precision):
    m = RegularMesh(ne, order=order)
    m.jitter_interior(1)
    kap = np.random.default_rng(2).uniform(0.5, 2.0, m.n_elements)
    A = LaplaceAssembly.from_regular_mesh(m, kappa=kap)
    nns = (order + 1) ** 3
    assert 8 * m.n_elements * nns * (nns + 1) // 2 > 256 << 20
    v = A.assemble(precision).cpu().numpy()
    rp, ci = A.row_ptr.cpu().numpy(), A.col_idx.cpu().numpy()
    ov = oracle.laplace_assemble_scaled(3, [order] * 3, [order + 1] * 3, m.elem_nodes, m.coords, None, kap, rp, ci, 16)
    assert np.abs(v - ov).max() <= 1e-12 * np.abs(ov).max()
    assert torch.equal(A.values, A.assemble(precision))


@pytest.mark.parametrize("ne", [(1, 1, 1), (4, 4, 4), (33, 1, 7), (16, 2, 1), (22, 21, 21), (22, 22, 21), (40, 17, 31)])
@pytest.mark.parametrize("with_kappa", [True, False])
def test_fp64_regular_mesh_forms(gfe_cuda, ne, with_kappa):
    """FP64 on the regular mesh: eight lanes an element up to 64 elements an SM (22 x 21 x 21 lies below,
    22 x 22 x 21 above on 152 SMs), a thread an element beyond, then the row gather, against the colour
    kernel and the tiled kernel (sums of at most 8 element entries of FP64 arithmetic in other orders:
    1e-13 relative to max|K|) and, on small meshes, the oracle."""
    m = RegularMesh(ne, extent=(1.0, 0.7, 1.3))
    m.jitter_interior(4)
    kap = np.random.default_rng(5).uniform(0.1, 10.0, m.n_elements) if with_kappa else None
    A = LaplaceAssembly.from_regular_mesh(m, kappa=kap)
    A.rhs.fill_(1.0)
    v = A.assemble("fp64", fp32_copy=True).clone()
    assert float(A.rhs.abs().max()) == 0.0 and torch.equal(A.values32, v.float())
    for path in ("general", "regular"):
        w = A.assemble("fp64", path=path)
        assert float((v - w).abs().max()) <= 1e-13 * float(w.abs().max()), path
    if m.n_elements < 1000:
        rp, ci = oracle.csr_structure(m.elem_nodes, m.n_nodes)
        ov, _ = oracle.laplace_assemble(3, [1, 1, 1], [2, 2, 2], m.elem_nodes, m.coords, kap, rp, ci)
        assert np.abs(v.cpu().numpy() - ov).max() <= 1e-13 * np.abs(ov).max()


@pytest.mark.parametrize("scale", [1.0, 3e-4, 7e5])
def test_float_float_element_chain(gfe_cuda, scale):
    """Float-float assembly with sums that are renormalised only before products, on a sheared, distorted mesh off the
    origin and over several sizes, against FP64.  Bound: coordinates split to 2^-48 of their magnitude, 8 elements
    and offsets of about one mesh length a side give differences to 2^-48 * 16, cubed ratios and cancelling sums a
    factor of about 100 on top: 1e-11 of max|K|."""
    A = LaplaceAssembly.from_regular_mesh(RegularMesh((7, 8, 5)))
    g = torch.Generator().manual_seed(5)
    x = A.coords.cpu()
    x = x + 0.3 * x.roll(1, 0) + 0.02 * torch.rand(x.shape, generator=g, dtype=torch.float64) + 0.7
    A.coords.copy_(x * scale)
    ref = A.assemble("fp64").clone()
    got = A.assemble("mixed_df")
    assert (got - ref).abs().max().item() <= 1e-11 * ref.abs().max().item()


@pytest.mark.parametrize("ne", [(1, 1, 1), (2, 1, 1), (7, 5, 3), (33, 9, 17), (24, 31, 19)])
def test_fp32_gather_equals_tiled_rows(gfe_cuda, ne):
    """FP32 on the regular mesh: the whole assembly through element matrices, with a workspace, with scratch and in
    layer slabs (the tiled kernel, which sums a row's eight contributions in the same order), gives the same bits."""
    from iron_gb300 import _lib
    A = LaplaceAssembly.from_regular_mesh(RegularMesh(ne))
    g = torch.Generator().manual_seed(11)
    x = A.coords.cpu() + 0.1 / max(ne) * torch.rand(A.coords.shape, generator=g, dtype=torch.float64)
    A.coords.copy_(x)
    got = A.assemble("mixed").clone()
    nx, ny, nz = ne
    ws = torch.empty(int(_lib.load().gfe_laplace_regular_workspace_bytes(nx, ny, nz, 1)), dtype=torch.uint8, device="cuda")
    for mode in ("scratch", "slabs"):
        A.values.fill_(-7.0)
        args = (nx, ny, nz, _lib.ptr(A.coords), _lib.ptr(A.kappa), _lib.ptr(A.row_ptr), _lib.ptr(A.values), None, None, 1)
        if mode == "scratch":
            _lib.call("gfe_laplace_assemble_regular_ws", *args, None, _lib.stream_handle(None))
        else:
            for l0 in range(0, nz + 1, 8):
                _lib.call("gfe_laplace_assemble_regular_layers", *args, _lib.ptr(ws), l0, min(l0 + 8, nz + 1),
                          int(l0 == 0), _lib.stream_handle(None))
        torch.cuda.synchronize()
        assert torch.equal(A.values, got), mode
