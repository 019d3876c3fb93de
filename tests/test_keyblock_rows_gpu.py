"""GPU parity of the key-block replay where the work lies unevenly: points and columns
(queried states) along the tour, which the row pass cuts by both, and probes over the key
blocks, where several CTAs share a block."""
from __future__ import annotations

import numpy as np
import pytest

import evgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tree", ["fork", "chain", "star"])
@pytest.mark.parametrize("S,E,Q,events", [
    (5000, 12, 9000, "any"),          # columns without points between them
    (5000, 60_000, 9000, "first"),    # every event on the root: all points before all columns
    (5000, 60_000, 9000, "last"),
    (5000, 60_000, 9000, "one"),
    (5000, 60_000, 40, "any"),        # few columns
    (5000, 60_000, 9000, "ends"),
    (40, 60_000, 9000, "any"),
])
def test_uneven_tours(bw, torch_cuda, oracle_mod, tree, S, E, Q, events):
    C = 400_000
    rng = np.random.default_rng(S + E + Q)
    parent = evgen.make_tree(S, tree, rng)
    ev, qs = evgen.make_events(S, C, E, rng, big=True), evgen.make_queries(S, C, Q, rng)
    if events == "ends":
        ev["state"] = np.sort(np.where(rng.random(E) < 0.5, 0, S - 1))
    elif events != "any":
        ev["state"] = {"first": 0, "last": S - 1, "one": S // 3}[events]
    p, e, q = evgen.to_device(torch_cuda, parent, ev, qs)
    plan = bw.Replay(p, C, E, Q)
    got = torch_cuda.empty(Q, dtype=torch_cuda.int64, device="cuda")
    plan.launch(p, e, q, got)
    assert plan.status() == 0
    assert plan.info()[1] == E // 512 + 1, "not the key-block path"
    np.testing.assert_array_equal(got.cpu().numpy(), oracle_mod.ev_sweep(parent, C, ev, qs))


@pytest.mark.parametrize("big", [False, True])
@pytest.mark.parametrize("queries,Q", [("prefix", 16_895), ("prefix", 16_896), ("prefix", 16_897), ("prefix", 33_792),
                                       ("prefix", 33_793), ("point", 120_000), ("whole", 120_000), ("half", 250_000)])
def test_shared_blocks(bw, torch_cuda, oracle_mod, queries, Q, big):
    """Parts are 16,896 probes here: below one, whole ones, one more, many."""
    S, C, E = 2000, 400_000, 60_000
    rng = np.random.default_rng(Q)
    parent = evgen.make_tree(S, "fork", rng)
    ev, qs = evgen.make_events(S, C, E, rng, big=big), evgen.make_queries(S, C, Q, rng)
    key = int(np.sort(ev["key"])[E // 2 + 100])
    n = Q // 2 if queries == "half" else Q
    at = rng.permutation(Q)[:n]
    qs["lo"][at] = key if queries == "point" else 0
    qs["hi"][at] = {"prefix": key, "point": key + 1, "whole": C, "half": C}[queries]
    p, e, q = evgen.to_device(torch_cuda, parent, ev, qs)
    plan = bw.Replay(p, C, E, Q)
    got = torch_cuda.empty(Q, dtype=torch_cuda.int64, device="cuda")
    want = oracle_mod.ev_sweep(parent, C, ev, qs)
    for _ in range(2):
        got.fill_(-1)
        plan.launch(p, e, q, got)
        assert plan.status() == 0
        np.testing.assert_array_equal(got.cpu().numpy(), want)
    assert plan.info()[1] == E // 512 + 1, "not the key-block path"
