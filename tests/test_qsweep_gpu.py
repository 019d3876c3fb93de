"""GPU parity of the query-step sweep at its own edges: many blocks, kernels enqueued."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

import evgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blocks", [65_535, 65_536, 70_000])
def test_many_blocks(bw, torch_cuda, oracle_mod, blocks):
    S, C, E, Q = 20_000, 16, 60_000, 360_000
    rng = np.random.default_rng(blocks)
    parent = evgen.make_tree(S, "fork", rng)
    ev, qs = evgen.make_events(S, C, E, rng), evgen.make_queries(S, C, Q, rng)
    p, e, q = evgen.to_device(torch_cuda, parent, ev, qs)
    got = bw.replay(p, C, e, q, blocks=blocks).cpu().numpy()
    np.testing.assert_array_equal(got, oracle_mod.ev_sweep(parent, C, ev, qs))


def test_kernels_enqueued(bw, torch_cuda):
    """info() counts the kernels of a launch: those of a captured one."""
    torch = torch_cuda
    S, C, E, Q = 3000, 500, 40_000, 240_000
    rng = np.random.default_rng(1)
    p, e, q = evgen.to_device(torch, evgen.make_tree(S, "fork", rng), evgen.make_events(S, C, E, rng),
                              evgen.make_queries(S, C, Q, rng))
    out = torch.empty(Q, dtype=torch.int64, device="cuda")
    plan = bw.Replay(p, C, E, Q)
    plan.launch(p, e, q, out)
    torch.cuda.synchronize()
    g, s = torch.cuda.CUDAGraph(keep_graph=True), torch.cuda.Stream()
    with torch.cuda.graph(g, stream=s):
        plan.launch(p, e, q, out, stream=s)
    rt = ctypes.CDLL("libcudart.so." + torch.version.cuda.split(".")[0])
    n, kind = ctypes.c_size_t(0), ctypes.c_int(0)
    graph = ctypes.c_void_p(g.raw_cuda_graph())
    assert rt.cudaGraphGetNodes(graph, None, ctypes.byref(n)) == 0
    nodes = (ctypes.c_void_p * n.value)()
    assert rt.cudaGraphGetNodes(graph, nodes, ctypes.byref(n)) == 0
    kernels = 0
    for x in nodes:
        assert rt.cudaGraphNodeGetType(ctypes.c_void_p(x), ctypes.byref(kind)) == 0
        kernels += kind.value == 0   # cudaGraphNodeTypeKernel
    assert plan.info()[0] == kernels
