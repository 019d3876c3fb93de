"""GPU parity of the key-block replay where points and columns (queried states) lie unevenly
along the tour: the row pass cuts it by both."""
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
