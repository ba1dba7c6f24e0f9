"""Sum-factorised FP64 Mooney-Rivlin kernels at the edges of their size rules.

The finite-difference Jacobian splits an element over 1, 3 or 9 CTAs by the number of elements and
adds the columns all at once through element matrices (up to 4,096 elements) or colour by colour;
every branch is compared with the oracle's element matrices on sampled elements, and the assembled
values with the sum of the dense element matrices.  Tolerances: the difference quotient amplifies the
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
