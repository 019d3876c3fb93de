"""GPU parity of the prepare passes where a group of 32 steps holds many events.

Groups above 512 events (2,048 in blocks of six groups a warp and more) are shared by all
warps of the CTA, up to 96 of them a block: states with none, a few, hundreds and thousands of
events, one state with almost all, contracted steps (few queries), more than 96 such groups
in a block, and blocks of one step.  Whole numbers, compared exactly with the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import evgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,E,C,Q,blocks,hot", [
    (40, 60_000, 300, 50, 0, 0.0),         # 1,500 events a state, fewer states than a group
    (3000, 200_000, 5000, 40, 3, 0.0),     # contracted: few states are asked
    (3000, 200_000, 5000, 9000, 2, 0.95),  # one state holds most events
    (9000, 200_000, 70_000, 5000, 1, 0.0), # one block, more than 96 heavy groups
    (9000, 40_000, 1, 5000, 1, 0.5),       # one key; groups around 128 events
    (700, 36_000, 4097, 700, 64, 0.0),     # groups around 512 events and more
])
def test_heavy_groups(bw, torch_cuda, oracle_mod, S, E, C, Q, blocks, hot):
    rng = np.random.default_rng(S + E)
    parent = evgen.make_tree(S, "fork", rng)
    ev, qs = evgen.make_events(S, C, E, rng, zipf=1.2), evgen.make_queries(S, C, Q, rng)
    if hot:
        st = ev["state"].copy()
        st[rng.random(E) < hot] = S // 3
        ev["state"] = np.sort(st)
    want = oracle_mod.ev_sweep(parent, C, ev, qs)
    p, e, q = evgen.to_device(torch_cuda, parent, ev, qs)
    for tile in (1, 6):
        f = bw.Forest([0, S], [0, E], [0, Q], [C], tuning=dict(tile=tile, block_work=0 if not blocks else max(1, 2 * E // blocks)))
        out = torch_cuda.empty(Q, dtype=torch_cuda.int64, device=p.device)
        f.launch(p, e, q, out)
        np.testing.assert_array_equal(out.cpu().numpy(), want)
    r = bw.Replay(p, C, E, Q, blocks=blocks)
    out = torch_cuda.empty(Q, dtype=torch_cuda.int64, device=p.device)
    r.launch(p, e, q, out)
    assert r.status() == 0
    np.testing.assert_array_equal(out.cpu().numpy(), want)


@pytest.mark.parametrize("big", [2**30 - 1, 2**30, 2**31 - 1, 2**31, -2**31, -2**31 - 1, 2**32 - 1, 2**32, 2**62, -2**63])
def test_delta_sums_around_31_bits(bw, torch_cuda, oracle_mod, big):
    """A block's sums are held in 32 bits only while its applied |delta| sum stays below 2^31."""
    rng = np.random.default_rng(abs(big) % 1000)
    S, C, E, Q = 700, 300, 9000, 300
    parent = evgen.make_tree(S, "fork", rng)
    ev, qs = evgen.make_events(S, C, E, rng), evgen.make_queries(S, C, Q, rng)
    ev["delta"] = 0
    ev["delta"][[E // 3, E // 2]] = [big, 1]
    want = oracle_mod.ev_sweep(parent, C, ev, qs)
    p, e, q = evgen.to_device(torch_cuda, parent, ev, qs)
    for blocks in (1, 4):
        r = bw.Replay(p, C, E, Q, blocks=blocks)
        out = torch_cuda.empty(Q, dtype=torch_cuda.int64, device=p.device)
        r.launch(p, e, q, out)
        assert r.status() == 0
        np.testing.assert_array_equal(out.cpu().numpy(), want)
