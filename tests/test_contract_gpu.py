"""GPU parity of contracted tours (few queries a state): runs merged into nodes, nodes no
query needs dropped -- trees and forests against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import evgen

pytestmark = pytest.mark.gpu


def _tree(kind, S, C, E, Q, where, rng):
    parent = evgen.make_tree(S, kind, rng, p_extend=0.97) if kind == "fork" else evgen.make_tree(S, kind, rng)
    ev = evgen.make_events(S, C, E, rng, zipf=1.1)
    qs = evgen.make_queries(S, C, Q, rng)
    if where == "root":
        qs["state"] = 0
    elif where == "last":
        qs["state"] = S - 1
    elif where == "early":
        qs["state"] = np.sort(qs["state"] % max(1, S // 20))
    elif where == "ends":
        qs["state"] = np.sort(np.array([0, S - 1], np.uint32)[rng.integers(0, 2, Q)])
    return parent, ev, qs


@pytest.mark.parametrize("kind", ["chain", "fork", "star", "bushy"])
@pytest.mark.parametrize("S,E,Q,where", [(2, 50, 1, "any"), (300, 2000, 1, "last"), (5000, 30000, 700, "any"),
                                         (5000, 30000, 900, "root"), (5000, 30000, 900, "early"),
                                         (5000, 30000, 2500, "ends"), (5000, 10, 2500, "any"),
                                         (40000, 200_000, 3000, "any")])
def test_tree_matches_oracle(bw, torch_cuda, oracle_mod, kind, S, E, Q, where):
    rng = np.random.default_rng(S + E + Q)
    parent, ev, qs = _tree(kind, S, 3000, E, Q, where, rng)
    p, e, q = evgen.to_device(torch_cuda, parent, ev, qs)
    want = oracle_mod.ev_sweep(parent, 3000, ev, qs)
    np.testing.assert_array_equal(bw.replay(p, 3000, e, q, path="general").cpu().numpy(), want)
    if kind == "chain":
        np.testing.assert_array_equal(bw.replay(p, 3000, e, q, path="general", chain=True).cpu().numpy(), want)


@pytest.mark.parametrize("tile", [1, 2, 3, 6])
def test_forest_matches_oracle(bw, torch_cuda, oracle_mod, tile):
    rng = np.random.default_rng(77)
    trees = []
    for i in range(60):
        S = int(rng.integers(1, 4000))
        trees.append(_tree(["fork", "chain", "star", "bushy"][i % 4], S, int(rng.integers(1, 9000)),
                           int(rng.integers(0, 9 * S)), int(rng.integers(0, max(1, S // 3))),
                           ["any", "root", "last", "early"][i // 4 % 4], rng) + (int(rng.integers(9000, 70000)),))
    off = [np.concatenate([[0], np.cumsum([len(t[k]) for t in trees])]) for k in range(3)]
    C = [t[3] for t in trees]
    assert off[2][-1] * 2 <= off[0][-1]
    p, e, q = evgen.to_device(torch_cuda, *(np.concatenate([t[k] for t in trees]) for k in range(3)))
    got = bw.forest_replay(*off, C, p, e, q, tuning=dict(tile=tile, block_work=20000)).cpu().numpy()
    want = np.concatenate([oracle_mod.ev_sweep(t[0], t[3], t[1], t[2]) for t in trees])
    np.testing.assert_array_equal(got, want)


def test_bad_parent_is_rejected(bw, torch_cuda):
    rng = np.random.default_rng(3)
    parent, ev, qs = _tree("fork", 3000, 500, 9000, 100, "any", rng)
    for i, v in ((0, 0), (100, 100), (100, -1), (2999, 5000)):
        bad = parent.copy()
        bad[i] = v
        p, e, q = evgen.to_device(torch_cuda, bad, ev, qs)
        with pytest.raises(ValueError, match="bad parent"):
            bw.replay(p, 500, e, q)
