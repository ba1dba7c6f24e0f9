"""The workspaces that LaplaceAssembly keeps for the regular-mesh kernels: whose they are, how long they live, and
what happens without room for them.

A stream is held up by a spinning kernel of about 20 ms, so that work queued behind it is still to come while the
host goes on.  The same mesh assembled alone is the reference, to the bit: the kernels sum in a fixed order.
"""
import copy

import numpy as np
import pytest
import torch

from iron_gb300 import laplace
from iron_gb300.laplace import LaplaceAssembly
from iron_gb300.mesh import RegularMesh

pytestmark = pytest.mark.gpu


def _assembly(ne=(24, 21, 26), seed=0):
    m = RegularMesh(ne)
    m.jitter_interior(seed)
    return LaplaceAssembly.from_regular_mesh(m, kappa=np.random.default_rng(seed).uniform(0.1, 10.0, m.n_elements))


def _hold(stream):
    with torch.cuda.stream(stream):
        torch.cuda._sleep(40_000_000)


@pytest.mark.parametrize("precision", ["fp64", "mixed", "mixed_df"])
def test_workspace_lives_as_long_as_its_use(gfe_cuda, precision):
    """Called on another stream than torch's current one and dropped at once: memory taken on the current stream
    afterwards is not the workspace that the queued kernels still write."""
    ref = _assembly().assemble(precision).clone()
    A = _assembly()
    values, kept = A.values, {k: v for k, v in A.__dict__.items() if k != "_ws_cache"}
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    _hold(s)
    A.assemble(precision, stream=s, check=False)
    (buf,) = [getattr(w, "buf", w) for w in A._ws_cache.values()]
    nbytes, place = buf.numel(), buf.data_ptr()
    kept.update(A.__dict__)
    kept.pop("_ws_cache")
    del A, buf
    junk = [torch.empty(nbytes, dtype=torch.uint8, device="cuda") for _ in range(4)]  # nothing is written to them
    assert all(j.data_ptr() != place for j in junk)
    torch.cuda.synchronize()
    assert torch.equal(values, ref)


@pytest.mark.parametrize("precision", ["fp64", "mixed", "mixed_df"])
def test_copies_do_not_share_a_workspace(gfe_cuda, precision):
    A = _assembly()
    A.assemble(precision)
    B, D = copy.copy(A), copy.deepcopy(A)
    for other in (B, D):
        other.values = torch.empty_like(A.values)
        other.assemble(precision)
    place = {x._ws_cache[k].buf.data_ptr() for x in (A, B, D) for k in x._ws_cache}
    assert len(place) == 3
    assert torch.equal(B.values, A.values) and torch.equal(D.values, A.values)


@pytest.mark.parametrize("precision", ["fp64", "mixed", "mixed_df"])
def test_one_assembly_on_two_streams(gfe_cuda, precision):
    """Values and conductivities exchanged between calls on two streams: a call waits until the workspace is free."""
    A = _assembly()
    sets = []
    for i in range(2):
        kappa = A.kappa * (1.0 + i)
        R = copy.copy(A)
        R.kappa, R.values = kappa, torch.empty_like(A.values)
        sets.append((kappa, torch.empty_like(A.values), R.assemble(precision).clone(), torch.cuda.Stream()))
    for r in range(10):
        for kappa, values, _, s in sets:
            values.zero_()
            s.wait_stream(torch.cuda.current_stream())
        for kappa, values, _, s in sets[:: 1 if r % 2 else -1]:
            A.kappa, A.values = kappa, values
            _hold(s)
            for _ in range(3):
                A.assemble(precision, stream=s, check=False, fp32_copy=False)
        torch.cuda.synchronize()
        for _, values, ref, _ in sets:
            assert torch.equal(values, ref)
    assert len(A._ws_cache) == 1  # one workspace, whatever the streams


def test_no_room_for_element_matrices(gfe_cuda, monkeypatch):
    """With little free memory FP64 takes the colour kernel and FP32 the tiled one; both for good, and with the
    results of those kernels."""
    ne = (80, 64, 64)  # 94 MB of FP64 element matrices
    A, B = _assembly(ne), _assembly(ne)
    want32 = B.assemble("mixed").clone()
    want64 = B.assemble("fp64", path="general").clone()
    asked = []

    def little(device=None):
        asked.append(device)
        return 200 << 20, 1 << 40

    with monkeypatch.context() as m:
        m.setattr(torch.cuda, "mem_get_info", little)
        m.setattr(laplace, "_ASK_FOR_ROOM", 64 << 20)
        first = A.assemble("fp64").clone()
        again = A.assemble("fp64").clone()
        assert len(asked) == 1
    later = A.assemble("fp64").clone()
    assert torch.equal(first, want64) and torch.equal(again, first) and torch.equal(later, first)
    # no room at all
    empty = torch.empty

    nbytes = (12 * A.n_nodes + 255) // 256 * 256 + 36 * 4 * A.n_elements

    def refuse(*args, **kw):
        if args and args[0] == nbytes:
            raise torch.OutOfMemoryError("refused by the test")
        return empty(*args, **kw)

    with monkeypatch.context() as m:
        m.setattr(torch, "empty", refuse)
        got32 = A.assemble("mixed").clone()
    assert torch.equal(got32, want32) and A._ws_cache[1].buf is None
    assert torch.equal(A.assemble("mixed"), want32)


def test_graph_captured_on_another_stream(gfe_cuda):
    """Warm-up on one stream, capture on another, then eager calls between replays."""
    A = _assembly()
    ref = A.assemble("fp64").clone()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        A.assemble("fp64", check=False)
    for _ in range(2):
        A.values.zero_()
        g.replay()
        assert torch.equal(A.values, ref)
        A.values.zero_()
        assert torch.equal(A.assemble("fp64", stream=torch.cuda.current_stream()), ref)
    # captured without a call before it: nothing is allocated, the colour kernel runs
    B = _assembly()
    h = torch.cuda.CUDAGraph()
    with torch.cuda.graph(h):
        B.assemble("fp64", check=False)
    want = _assembly().assemble("fp64", path="general")
    h.replay()
    torch.cuda.synchronize()
    assert torch.equal(B.values, want)
