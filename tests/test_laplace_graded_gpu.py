"""Float-float assembly on the regular mesh where a coordinate is much larger than the edges that meet in it: meshes
graded by up to 1e-9 towards the origin or towards another point, and far from the origin.

Bound against FP64: the edges are formed without loss, the elements are right-angled (nothing cancels), and an entry
then takes a chain of about 64 float-float operations of 2^-48 each.  Layer calls read a copy of the coordinates and
give the same bits.  Coordinates that no float holds are reported like any other degenerate element.
"""
import math

import numpy as np
import pytest
import torch

from iron_gb300 import _lib
from iron_gb300._lib import GfeError
from iron_gb300.laplace import LaplaceAssembly
from iron_gb300.mesh import RegularMesh

pytestmark = pytest.mark.gpu


def _graded(t, span):
    """[0, 1] onto itself, the first of the steps about `span` of the last."""
    return np.expm1(t * math.log(1.0 / span)) / math.expm1(math.log(1.0 / span))


@pytest.mark.parametrize("ne", [(5, 4, 3), (32, 9, 17)])
@pytest.mark.parametrize("kind", ["origin", "one", "negative", "far"])
@pytest.mark.parametrize("span", [1e-3, 1e-6, 1e-9])
def test_graded_mesh(gfe_cuda, ne, kind, span):
    A = LaplaceAssembly.from_regular_mesh(RegularMesh(ne))
    x = A.coords.cpu().numpy().copy()
    for c in (0, 2):
        x[c] = _graded(x[c], span) if c == 0 else _graded(x[c], 1e-2)
    x = {"origin": x, "one": 1.0 - x, "negative": -x, "far": x + np.array([[1.0], [-1e3], [1e5]])}[kind]
    if kind in ("one", "negative"):
        x = x[:, ::-1]  # the numbering reversed: a positive Jacobian in every direction
    A.coords.copy_(torch.from_numpy(np.ascontiguousarray(x)))
    ref = A.assemble("fp64", path="general").clone()
    got = A.assemble("mixed_df").clone()
    assert (got - ref).abs().max().item() <= 64 * 2.0 ** -48 * ref.abs().max().item()
    nx, ny, nz = ne
    nbytes = int(_lib.load().gfe_laplace_regular_workspace_bytes(nx, ny, nz, 2))
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    A.values.fill_(-7.0)
    coords = A.coords.clone()
    for l0 in range(0, nz + 1, 8):
        _lib.call("gfe_laplace_assemble_regular_layers", nx, ny, nz, _lib.ptr(coords), _lib.ptr(A.kappa),
                  _lib.ptr(A.row_ptr), _lib.ptr(A.values), None, None, 2, _lib.ptr(ws), l0, min(l0 + 8, nz + 1),
                  int(l0 == 0), _lib.stream_handle(None))
        coords.fill_(0.0)  # later calls read the workspace's copy
    torch.cuda.synchronize()
    assert torch.equal(A.values, got)


@pytest.mark.parametrize("value", [math.inf, -math.inf, math.nan, 1e39, -1e300])
def test_coordinates_beyond_a_float(gfe_cuda, value):
    A = LaplaceAssembly.from_regular_mesh(RegularMesh((4, 3, 3)))
    A.coords[1, 17] = value
    with pytest.raises(GfeError, match="non-positive Jacobian"):
        A.assemble("mixed_df")
    assert _lib.device_errors() == 0


@pytest.mark.parametrize("value", [0.0, -0.0, 5e-324, 1e-30])
def test_coordinates_next_to_zero(gfe_cuda, value):
    """The zero coordinates of the origin's faces as tiny numbers of either sign."""
    A = LaplaceAssembly.from_regular_mesh(RegularMesh((4, 3, 3)))
    ref = A.assemble("mixed_df").clone()
    A.coords[A.coords == 0.0] = value
    assert torch.equal(A.assemble("mixed_df"), ref)
