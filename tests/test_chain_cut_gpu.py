"""GPU parity of the chain path where the cut of its blocks changes: single blocks for few
events, queries after the last event, all queries on one state."""
from __future__ import annotations

import numpy as np
import pytest

import evgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,C,E,Q,hot,share", [
    (1000, 100, 4102, 0, 0, 0), (1000, 100, 4101, 1, 0, 0), (1000, 32_000, 6095, 1, 0, 0), (1000, 32_000, 6096, 1, 0, 0),
    (1000, 32_000, 6000, 7, 0, 0), (3, 10, 2, 40, 0, 0), (1, 1700, 20_000, 9000, 0, 1.0),
    (1000, 1700, 50_000, 16, -1, 1.0), (1000, 1700, 50_000, 4001, -1, 1.0), (1000, 1700, 50_000, 4001, -1, 0.062),
    (1000, 1700, 50_000, 4001, -1, 0.063), (1000, 1700, 50_000, 4001, 0, 1.0), (1000, 1700, 50_000, 4001, 600, 0.9),
])
@pytest.mark.parametrize("blocks", [0, 1, 17, 2000])
@pytest.mark.parametrize("wide", [False, True])
def test_cut(bw, torch_cuda, oracle_mod, S, C, E, Q, hot, share, blocks, wide):
    rng = np.random.default_rng(S + E + Q)
    parent = evgen.make_tree(S, "chain", rng)
    ev, qs = evgen.make_events(S, C, E, rng), evgen.make_queries(S, C, Q, rng)
    qs["state"][: int(Q * share)] = hot % S
    qs["state"].sort()
    p, e, q = evgen.to_device(torch_cuda, parent, ev, qs)
    got = bw.replay(p, C, e, q, chain=True, path="chain", blocks=blocks, wide=wide).cpu().numpy()
    np.testing.assert_array_equal(got, oracle_mod.ev_sweep(parent, C, ev, qs))


def test_few_events_take_one_block(bw, torch_cuda):
    """1,493 events and one query over 10,423 keys: one block (two cost a carry pass and a fix-up
    more than they save), several where the queries are many."""
    rng = np.random.default_rng(0)
    parent = evgen.make_tree(4, "chain", rng)
    for Q, one in ((1, True), (1493, False)):
        p, e, q = evgen.to_device(torch_cuda, parent, evgen.make_events(4, 10_423, 1493, rng),
                                  evgen.make_queries(4, 10_423, Q, rng))
        plan = bw.Replay(p, 10_423, 1493, Q, chain=True, path="chain")
        plan.launch(p, e, q, torch_cuda.empty(Q, dtype=torch_cuda.int64, device="cuda"))
        assert plan.status() == 0
        assert (plan.info()[1] == 1) == one
