"""GPU parity of the key-block replay (large key domains) with the oracle and with the
state-block pipeline, at the edges of its blocks, tiles and rules."""
from __future__ import annotations

import numpy as np
import pytest

import evgen

pytestmark = pytest.mark.gpu

CASES = [
    # tree, S, C, E, Q, keys, queries
    ("fork", 3000, (1 << 18) + 1, 40000, 30000, "uniform", "any"),
    ("chain", 2000, 300_007, 5120, 9000, "uniform", "any"),          # events a multiple of the block
    ("star", 700, 1 << 20, 511, 3000, "uniform", "any"),             # one block
    ("bushy", 2049, 1 << 19, 70000, 8193, "uniform", "any"),
    ("fork", 5000, 400_000, 90000, 50000, "zipf", "any"),
    ("fork", 1500, 300_000, 60000, 20000, "hot", "any"),             # all events on one key
    ("fork", 1500, 300_000, 60000, 20000, "few", "any"),             # keys with many events each, at both ends
    ("fork", 9000, 300_000, 30000, 700, "uniform", "few_states"),    # most states below no query
    ("fork", 1, 300_000, 20000, 5000, "uniform", "any"),
    ("fork", 2000, 300_000, 30000, 4097, "uniform", "one_state"),
    ("fork", 2000, 300_000, 30000, 1, "uniform", "any"),
    ("fork", 40000, 300_000, 1, 2000, "uniform", "any"),
    ("fork", 30000, 500_000, 1_000_000, 300_000, "uniform", "any"),  # two steps of slots a block
]


def _case(tree, S, C, E, Q, keys, queries, big=False):
    rng = np.random.default_rng(S + C + E + Q)
    parent = evgen.make_tree(S, tree, rng)
    ev = evgen.make_events(S, C, E, rng, zipf=1.1 if keys == "zipf" else 0.0, big=big)
    if keys == "hot":
        ev["key"] = C // 3
    elif keys == "few":
        ev["key"] = np.array([0, 1, 2, C // 2, C - 2, C - 1], np.uint32)[rng.integers(0, 6, E)]
    qs = evgen.make_queries(S, C, Q, rng)
    if queries == "few_states":
        qs["state"] = np.sort(rng.choice(S, 5)[rng.integers(0, 5, Q)])
    elif queries == "one_state":
        qs["state"] = S // 2
    return parent, ev, qs


@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(map(str, c)))
def test_matches_oracle_and_state_blocks(bw, torch_cuda, oracle_mod, case):
    parent, ev, qs = _case(*case)
    C = case[2]
    p, e, q = evgen.to_device(torch_cuda, parent, ev, qs)
    want = oracle_mod.ev_sweep(parent, C, ev, qs)
    plan = bw.Replay(p, C, len(ev), len(qs))
    got = torch_cuda.empty(len(qs), dtype=torch_cuda.int64, device="cuda")
    for _ in range(2):   # the scratch is initialised by every launch
        got.fill_(-1)
        plan.launch(p, e, q, got)
        assert plan.status() == 0
        np.testing.assert_array_equal(got.cpu().numpy(), want)
    m = 512 * (len(ev) // (12 * bw.device_info()[0] * 512) + 1)
    assert plan.info()[1] == len(ev) // m + 1, "not the key-block path"
    np.testing.assert_array_equal(bw.replay(p, C, e, q, path="general").cpu().numpy(), want)


def test_wrapping_deltas_and_chain_hint(bw, torch_cuda, oracle_mod):
    parent, ev, qs = _case("chain", 900, 1 << 19, 30000, 9000, "uniform", "any", big=True)
    p, e, q = evgen.to_device(torch_cuda, parent, ev, qs)
    want = oracle_mod.ev_sweep(parent, 1 << 19, ev, qs)
    for kw in ({}, {"chain": True}):
        np.testing.assert_array_equal(bw.replay(p, 1 << 19, e, q, **kw).cpu().numpy(), want)


def test_rejected_inputs(bw, torch_cuda):
    parent, ev, qs = _case("fork", 900, 1 << 19, 30000, 9000, "uniform", "any")

    def rejected(match, **change):
        par, e, q = parent.copy(), ev.copy(), qs.copy()
        for what, (i, v) in change.items():
            if what == "parent":
                par[i] = v
            else:
                {"e": e, "q": q}[what[0]][what[2:]][i] = v
        with pytest.raises(ValueError, match=match):
            bw.replay(*(lambda a: (a[0], 1 << 19, a[1], a[2]))(evgen.to_device(torch_cuda, par, e, q)))
    rejected("event key", e_key=(77, 1 << 19))
    rejected("query bound", q_hi=(5, (1 << 19) + 1))
    rejected("not grouped", e_state=(20000, 0))
    rejected("bad parent", parent=(500, 700))
    p, e, q = evgen.to_device(torch_cuda, parent, ev, qs)
    with pytest.raises(ValueError, match="bad parent"):
        bw.replay(p, 1 << 19, e, q, chain=True)


def test_captured_launch(bw, torch_cuda, oracle_mod):
    """Kernels and memsets only: a captured launch replays on new inputs."""
    torch = torch_cuda
    C = 1 << 19
    parent, ev, qs = _case("fork", 900, C, 30000, 9000, "uniform", "any")
    p, e, q = evgen.to_device(torch, parent, ev, qs)
    plan = bw.Replay(p, C, len(ev), len(qs))
    got = torch.empty(len(qs), dtype=torch.int64, device="cuda")
    plan.launch(p, e, q, got)
    torch.cuda.synchronize()
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(g, stream=s):
        plan.launch(p, e, q, got, stream=s)
    ev["key"] = (ev["key"].astype(np.int64) * 7 + 3) % C
    e.copy_(evgen.to_device(torch, parent, ev, qs)[1])
    g.replay()
    torch.cuda.synchronize()
    np.testing.assert_array_equal(got.cpu().numpy(), oracle_mod.ev_sweep(parent, C, ev, qs))
