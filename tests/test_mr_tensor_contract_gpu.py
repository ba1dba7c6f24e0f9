"""Tensor-core contraction of the Mooney-Rivlin element Jacobians where its persistent CTAs take no, one, two or many
elements (two CTAs an SM; 304 on 152 SMs), on every element, against the CUDA-core contraction of the same FP32
Gauss-point blocks.

Tolerance, relative to max|K|: that of the small-mesh parity tests of the same precisions (81-term FP32 sums of split
products: 2e-5; one TF32 pass, 2^-11 an operand: 4e-3)."""
import numpy as np
import pytest
import torch

from iron_gb300.elasticity import MooneyRivlinAssembly
from test_mr_gpu import C1, C2, _state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fn", ["element_jacobians", "element_tangents"])
@pytest.mark.parametrize("ne", [(1, 1, 1), (3, 1, 1), (19, 16, 1), (61, 5, 1), (9, 9, 12)])
def test_contraction_on_every_element(gfe_cuda, ne, fn):
    A = MooneyRivlinAssembly.from_regular_mesh(ne, build_jacobian=False)
    dep = torch.from_numpy(_state(A, 7)).cuda()
    ref = getattr(A, fn)(dep, [C1, C2], precision="mixed").clone()
    scale = ref.abs().max().item()
    for precision, tol in (("tf32x3", 2e-5), ("tf32", 4e-3)):
        got = getattr(A, fn)(dep, [C1, C2], precision=precision)
        assert (got - ref).abs().max().item() <= tol * scale, precision
        # another launch gives the same bits: no element is read before it is complete
        assert torch.equal(getattr(A, fn)(dep, [C1, C2], precision=precision), got), precision


def test_row_gather_of_any_node_valence(gfe_cuda):
    """Rows whose node has 1, 2, 4 and 8 elements, on rows that start at even and odd entries: the CSR values are the
    FP32 sums of the element matrices in element order, bit for bit."""
    A = MooneyRivlinAssembly.from_regular_mesh((3, 2, 2))
    dep = torch.from_numpy(_state(A, 9)).cuda()
    slots = A.slots.cpu().numpy().reshape(A.n_elements, 89, 89)
    K = A.element_tangents(dep, [C1, C2], precision="tf32x3").cpu().numpy().reshape(A.n_elements, 89, 89)
    want = np.zeros(A.nnz, np.float32)
    for e in range(A.n_elements):
        s, k = slots[e], K[e].astype(np.float32)
        keep = s >= 0
        keep[81:, 81:] = False
        want[s[keep]] += k[keep]
    rp = A.row_ptr.cpu().numpy()
    assert {0, 1} == set(((rp[:-1] - 1) % 2).tolist())
    assert np.array_equal(A.tangent(dep, [C1, C2], precision="tf32x3").cpu().numpy(), want.astype(np.float64))
