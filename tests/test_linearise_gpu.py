"""GPU parity of the tour building at the sizes where its kernels change.

The inclusive scans sum the totals of earlier tiles in the kernel that applies them up to
2,048 tiles of 4,096 elements (twice the states), above in a kernel of their own; tours
below 2^24 states are built by chained launches.  Whole numbers, compared exactly with the chain path or the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import evgen

pytestmark = pytest.mark.gpu


def run(bw, torch, p, C, e, q, **kw):
    r = bw.Replay(p, C, e.shape[0], q.shape[0], **kw)
    out = torch.empty(q.shape[0], dtype=torch.int64, device=p.device)
    r.launch(p, e, q, out)
    assert r.status() == 0
    return out.cpu().numpy()


@pytest.mark.parametrize("S", [4 << 20, (4 << 20) + 1, (1 << 24) - 1, 1 << 24])
def test_scan_of_many_tiles(bw, torch_cuda, S):
    rng = np.random.default_rng(S)
    C, E, Q = 300, 50_000, 5000
    parent = evgen.make_tree(S, "chain", rng)
    ev, qs = evgen.make_events(S, C, E, rng, big=True), evgen.make_queries(S, C, Q, rng)
    p, e, q = evgen.to_device(torch_cuda, parent, ev, qs)
    want = run(bw, torch_cuda, p, C, e, q, chain=True, path="chain")
    np.testing.assert_array_equal(run(bw, torch_cuda, p, C, e, q), want)


@pytest.mark.parametrize("kind", ["fork", "chain", "star", "bushy"])
@pytest.mark.parametrize("S,C,E,Q", [(1, 1, 40, 64), (50, 1, 500, 3100), (300, 70_000, 9000, 18_500), (200, 300, 0, 12_500),
                                     (64, 20_000, 50_000, 1537), (3000, 4097, 600_000, 54_001),
                                     (20_000, 4097, 50_000, 360_001), (19_999, 500, 40_000, 360_001)])
def test_query_step_sweep(bw, torch_cuda, oracle_mod, S, C, E, Q, kind):
    """Single trees whose states are asked 18 queries and more take the query-step sweep (the
    last case, just below 20,000 states, the Euler-tile sweep)."""
    rng = np.random.default_rng(S + C)
    parent = evgen.make_tree(S, kind, rng)
    ev, qs = evgen.make_events(S, C, E, rng, zipf=1.2, big=S == 300), evgen.make_queries(S, C, Q, rng)
    want = oracle_mod.ev_sweep(parent, C, ev, qs)
    p, e, q = evgen.to_device(torch_cuda, parent, ev, qs)
    for blocks in (0, 1, 7):
        np.testing.assert_array_equal(run(bw, torch_cuda, p, C, e, q, blocks=blocks), want)
