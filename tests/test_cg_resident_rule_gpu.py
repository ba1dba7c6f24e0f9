"""Which CG systems run in the resident kernels: at most three slices of 32 rows a warp (31 warps an SM) and, in FP64,
where no other form uses it, a sliced-ELL copy of at most 150 MB with its padding.  The profiler counts one launch per
resident kernel of up to 200 iterations and one per product of the launched form (chunks of 50), so the count says which
form ran and that no other one was tried first; the solution is checked by its residual formed in torch (1 % above the tolerance is
far more than the rounding of forming it again)."""
import ctypes as C
import math

import numpy as np
import pytest
import torch

from iron_gb300 import _lib

pytestmark = pytest.mark.gpu


def _csr(rows, cols, vals, n):
    """1-based int32 CSR of A + A^T + a dominant diagonal from the strict upper entries of A."""
    r, c, v = np.r_[rows, cols], np.r_[cols, rows], np.r_[vals, vals]
    d = np.bincount(r, weights=np.abs(v), minlength=n) + 0.05
    r, c, v = np.r_[r, np.arange(n)], np.r_[c, np.arange(n)], np.r_[v, d]
    o = np.lexsort((c, r))
    ptr = np.r_[0, np.cumsum(np.bincount(r, minlength=n))]
    to = lambda a, t: torch.from_numpy(np.ascontiguousarray(a.astype(t))).cuda()  # noqa: E731
    return to(ptr + 1, np.int32), to(c[o] + 1, np.int32), to(v[o], np.float64)


def _stencil(m):
    """7-point Laplacian of m nodes a side."""
    i = np.arange(m ** 3).reshape(m, m, m)
    rows = np.concatenate([i[1:].ravel(), i[:, 1:].ravel(), i[:, :, 1:].ravel()])
    cols = np.concatenate([i[:-1].ravel(), i[:, :-1].ravel(), i[:, :, :-1].ravel()])
    return _csr(rows, cols, -np.ones(len(rows)), m ** 3)


def _hubs(n, degree):
    """One row of about `degree` entries in every slice of 32, the others short."""
    rng = np.random.default_rng(1)
    hub = np.repeat(np.arange(0, n, 32), degree)
    other = rng.integers(0, n, len(hub))
    ok = other % 32 != 0
    pair = np.unique(np.stack([hub[ok], other[ok]]), axis=1)
    return _csr(pair[0], pair[1], -rng.uniform(0.1, 1.0, pair.shape[1]), n)


def _solve(sys, mixed, rtol=1e-10):
    rp, ci, v = sys
    n = rp.numel() - 1
    g = torch.Generator().manual_seed(3)
    f = torch.randn(n, dtype=torch.float64, generator=g).cuda()
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    v32 = v.float() if mixed else None
    it, rel = C.c_int32(0), C.c_double(0.0)
    _lib.profile_enable(True)
    _lib.profile_read(_lib.STAGE_SPMV, reset=True)
    try:
        _lib.call("gfe_cg_solve", n, _lib.ptr(rp), _lib.ptr(ci), _lib.ptr(v), _lib.ptr(v32), _lib.ptr(f), None,
                  _lib.ptr(x), rtol, 20000, 1 if mixed else 0, C.byref(it), C.byref(rel), _lib.stream_handle(None))
        launches = _lib.profile_read(_lib.STAGE_SPMV, reset=True)[1]
    finally:
        _lib.profile_enable(False)
    A = torch.sparse_csr_tensor((rp - 1).long(), (ci - 1).long(), v, (n, n))
    assert float((f - A @ x).norm()) <= 1.01 * rtol * float(f.norm())
    return it.value, launches


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("case", ["three slices", "too many rows", "padding fits", "too much padding"])
def test_form_by_size_and_padding(gfe_cuda, case, mixed):
    rows = 3 * 32 * 31 * torch.cuda.get_device_properties(0).multi_processor_count
    side = {"three slices": int(rows ** (1 / 3)) - 1, "too many rows": int(rows ** (1 / 3)) + 2}
    sys = _stencil(side[case]) if case in side else _hubs(60000, 60 if case == "padding fits" else 420)
    n, nnz = sys[0].numel() - 1, sys[1].numel()
    assert nnz / n <= 32 and 12 * nnz <= 100 << 20
    it, launches = _solve(sys, mixed)
    if case in ("three slices", "padding fits") or (case == "too much padding" and mixed):
        # at least one kernel for each 200 iterations and each restart of the refinement, and no product launched
        assert math.ceil(it / 200) <= launches <= math.ceil(it / 200) + 40 and launches < it
    else:
        assert launches % 50 == 0 and launches >= it  # whole chunks of products, nothing else
