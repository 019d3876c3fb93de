"""GPU parity of forests of many small trees with items in few of them: the ingest finds an
item's tree far from the one before."""
from __future__ import annotations

import numpy as np
import pytest

import evgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,smax", [(1, 5), (2, 1), (33, 1), (1931, 9), (5000, 1), (700, 60)])
@pytest.mark.parametrize("events,queries", [(0.0, 0.002), (0.001, 0.02), (0.02, 1.0), (1.0, 0.05), (1.0, 1.0)])
def test_few_trees_with_items(bw, torch_cuda, oracle_mod, T, smax, events, queries):
    """`events` and `queries`: shares of the trees that have some; the first and the last always do."""
    rng = np.random.default_rng(T + smax)
    parts, so, eo, qo, keys, want = [], [0], [0], [0], [], []
    for t in range(T):
        S, C = int(rng.integers(1, smax + 1)), int(rng.integers(1, 300))
        end = t in (0, T - 1)
        E = int(rng.integers(1, 40)) if end or rng.random() < events else 0
        Q = int(rng.integers(1, 7)) if end or rng.random() < queries else 0
        parent = evgen.make_tree(S, "fork", rng)
        ev, qs = evgen.make_events(S, C, E, rng, big=t % 3 == 0), evgen.make_queries(S, C, Q, rng)
        parts.append((parent, ev, qs))
        so.append(so[-1] + S)
        eo.append(eo[-1] + E)
        qo.append(qo[-1] + Q)
        keys.append(C)
        want.append(oracle_mod.ev_sweep(parent, C, ev, qs) if Q else np.empty(0, np.int64))
    p, e, q = evgen.to_device(torch_cuda, *(np.concatenate(x) for x in zip(*parts)))
    got = bw.forest_replay(so, eo, qo, keys, p, e, q).cpu().numpy()
    np.testing.assert_array_equal(got, np.concatenate(want))
