"""GPU parity of the query-step sweep at its own edges: many blocks, kernels enqueued, states
asked or edited much more than the others."""
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


@pytest.mark.parametrize("big", [False, True])   # int32 and int64 windows, several of each
@pytest.mark.parametrize("blocks", [0, 1, 7])
def test_hot_states(bw, torch_cuda, oracle_mod, blocks, big):
    """Steps around 256 queries (a thread pair's first), 1,024 (a carry group's share), and
    around 512 events, among ordinary ones."""
    S, C, E, Q = 700, 90_000, 90_000, 60_000
    rng = np.random.default_rng(blocks)
    parent = evgen.make_tree(S, "fork", rng)
    ev, qs = evgen.make_events(S, C, E, rng, big=big), evgen.make_queries(S, C, Q, rng)
    counts = [255, 256, 257, 511, 512, 513, 1023, 1024, 1025, 1280, 1281, 4097, 9000]
    hot = rng.choice(S, len(counts), replace=False)
    for arr, n in ((qs, Q), (ev, E)):
        state = rng.choice(np.setdiff1d(np.arange(S), hot), n)
        state[: sum(counts)] = np.repeat(hot, counts)
        arr["state"] = np.sort(state)
    p, e, q = evgen.to_device(torch_cuda, parent, ev, qs)
    got = bw.replay(p, C, e, q, blocks=blocks).cpu().numpy()
    np.testing.assert_array_equal(got, oracle_mod.ev_sweep(parent, C, ev, qs))


@pytest.mark.parametrize("hot", [0, 1500, 2599, None])
def test_all_queries_heavy(bw, torch_cuda, oracle_mod, hot):
    """More heavy groups than a carry CTA's list holds (every state asked some 300 queries, one
    block), and every query on one state."""
    S, C, E, Q = 2600, 3000, 20_000, 780_000
    rng = np.random.default_rng(3)
    parent = evgen.make_tree(S, "fork", rng)
    ev, qs = evgen.make_events(S, C, E, rng), evgen.make_queries(S, C, Q, rng)
    if hot is not None:
        qs["state"] = hot
    p, e, q = evgen.to_device(torch_cuda, parent, ev, qs)
    want = oracle_mod.ev_sweep(parent, C, ev, qs)
    for blocks in (0, 1, 2):
        np.testing.assert_array_equal(bw.replay(p, C, e, q, blocks=blocks).cpu().numpy(), want)
