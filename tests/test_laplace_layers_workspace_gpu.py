"""Layer calls of the regular-mesh assembly write no more of the workspace than they say: nothing in FP64 and the
converted coordinates (12 bytes a node) in FP32, also when one call covers the whole mesh.  The bytes behind are as
many as the element matrices that a whole-mesh assembly may write there, so a call that did would not leave the
allocation."""
import pytest
import torch

from iron_gb300 import _lib
from iron_gb300.laplace import LaplaceAssembly
from iron_gb300.mesh import RegularMesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("ne", [(1, 1, 1), (7, 5, 3), (24, 31, 33)])
def test_layer_calls_leave_the_bytes_behind_the_coordinates(gfe_cuda, ne, precision):
    nx, ny, nz = ne
    prec = {"fp64": 0, "mixed": 1}[precision]
    A = LaplaceAssembly.from_regular_mesh(RegularMesh(ne))
    g = torch.Generator().manual_seed(3)
    A.coords.copy_(A.coords.cpu() + 0.1 / max(ne) * torch.rand(A.coords.shape, generator=g, dtype=torch.float64))
    ref = A.assemble(precision, path="general").clone()
    used = 0 if prec == 0 else (12 * A.n_nodes + 255) // 256 * 256  # rounded up, as the coordinates' place is
    ws = torch.full((used + 36 * 8 * A.n_elements + 256,), 0xA5, dtype=torch.uint8, device="cuda")
    A.values.fill_(-7.0)
    _lib.call("gfe_laplace_assemble_regular_layers", nx, ny, nz, _lib.ptr(A.coords), _lib.ptr(A.kappa),
              _lib.ptr(A.row_ptr), _lib.ptr(A.values), None, None, prec, _lib.ptr(ws), 0, nz + 1, 1,
              _lib.stream_handle(None))
    torch.cuda.synchronize()
    assert bool((ws[used:] == 0xA5).all())
    # sums of eight element entries in another order; FP32 element matrices may differ by their rounding
    tol = 1e-12 if prec == 0 else 1e-5
    assert (A.values - ref).abs().max().item() <= tol * ref.abs().max().item()
