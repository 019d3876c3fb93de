"""GPU parity of the chain path's carry (k_chain_carry) and of its block and geometry rules.

Where queries are many, the blocks are cut by events and queries together: clumped events,
all events or all queries on one state (blocks without events), queries before the first and
after the last event, more queries on one state than a tile stages.
The carry splits the blocks' prefix rows into 32 ranges and holds up to eight rows of a
range in registers: the block counts lie around both limits, the key domains around the
32 columns that a CTA takes.  The workloads of the second test get three 384-thread CTAs an
SM (dense queries; int64 window), two with fewer blocks, so that the rows stay within 32 MiB,
and two of 256 threads; the last is the first size whose carry
is launched the ordinary way.
Whole numbers: every answer is compared exactly, with the general path."""
from __future__ import annotations

import numpy as np
import pytest

import evgen

pytestmark = pytest.mark.gpu


def replay(bw, torch, p, C, e, q, **kw):
    r = bw.Replay(p, C, e.shape[0], q.shape[0], **kw)
    ans = torch.empty(q.shape[0], dtype=torch.int64, device=p.device)
    r.launch(p, e, q, ans)
    assert r.status() == 0
    return r, ans.cpu().numpy()


@pytest.mark.parametrize("C", [1, 32, 33, 4096])
@pytest.mark.parametrize("blocks", [2, 31, 33, 256, 257, 700])
def test_carry_over_block_counts(bw, torch_cuda, blocks, C):
    rng = np.random.default_rng(blocks * 5000 + C)
    S, E, Q = 3000, 30_001, 3001
    parent = evgen.make_tree(S, "chain", rng)
    ev, qs = evgen.make_events(S, C, E, rng, big=True), evgen.make_queries(S, C, Q, rng)
    p, e, q = evgen.to_device(torch_cuda, parent, ev, qs)
    r, got = replay(bw, torch_cuda, p, C, e, q, chain=True, path="chain", blocks=blocks)
    assert r.chain_path(e)
    _, want = replay(bw, torch_cuda, p, C, e, q, chain=True, path="general")
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("C,E,Q,wide", [(8000, 3_800_001, 90_001, False), (3001, 3_800_001, 400_000, True),
                                        (8001, 2_600_003, 20_000, True), (16_384, 2_600_003, 20_000, False),
                                        (900, 4_194_304, 20_000, False)])
def test_geometry_rules(bw, torch_cuda, C, E, Q, wide):
    rng = np.random.default_rng(C)
    S = 50_000
    parent = evgen.make_tree(S, "chain", rng)
    ev, qs = evgen.make_events(S, C, E, rng, zipf=1.1, big=wide), evgen.make_queries(S, C, Q, rng)
    p, e, q = evgen.to_device(torch_cuda, parent, ev, qs)
    r, got = replay(bw, torch_cuda, p, C, e, q, chain=True, path="chain", wide=wide)
    assert r.chain_path(e)
    if C == 8001:
        assert r.workspace.numel() <= 32 << 20
    _, want = replay(bw, torch_cuda, p, C, e, q, chain=True, path="general")
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("blocks", [0, 1, 7, 400])
@pytest.mark.parametrize("shape", ["clumps", "events on one state", "queries on one state", "queries at the ends"])
def test_blocks_cut_by_events_and_queries(bw, torch_cuda, shape, blocks, wide):
    rng = np.random.default_rng(len(shape) + blocks)
    S, C, E, Q = 5000, 3001, 40_001, 9000
    parent = evgen.make_tree(S, "chain", rng)
    ev, qs = evgen.make_events(S, C, E, rng, big=wide), evgen.make_queries(S, C, Q, rng)
    if shape == "clumps":
        ev["state"] = np.sort(np.where(rng.random(E) < 0.9, rng.integers(0, 30, E) * 160, rng.integers(0, S, E)))
    elif shape == "events on one state":
        ev["state"] = 2500
    elif shape == "queries on one state":
        qs["state"] = 2500
    else:
        ev["state"] = np.sort(rng.integers(1000, 1200, E))
        qs["state"] = np.sort(np.where(rng.random(Q) < 0.5, rng.integers(0, 1000, Q), rng.integers(1200, S, Q)))
    p, e, q = evgen.to_device(torch_cuda, parent, ev, qs)
    r, got = replay(bw, torch_cuda, p, C, e, q, chain=True, path="chain", blocks=blocks, wide=wide)
    assert r.chain_path(e)
    _, want = replay(bw, torch_cuda, p, C, e, q, chain=True, path="general")
    np.testing.assert_array_equal(got, want)
