"""Which path a single tree over a wide key domain takes, and that both agree there: little
work over few windows of the domain stays with the state blocks."""
from __future__ import annotations

import numpy as np
import pytest

import evgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,C,E,Q,key_blocks", [
    (300, 262_145, 1000, 1_000_000, True),      # two key blocks of a million probes
    (127, 279_218, 148, 2_398_098, True),
    (6518, 471_466, 4822, 3_655_433, True),
    (300, 262_145, 1000, 100, False),           # one state block
    (1, 609_353, 23, 229, False),
    (1, 4_000_000, 2, 3, True),                 # sixteen windows
    (1, 387_896, 3, 628_384, True),
    (40_000, 300_000, 1, 2000, True),
])
def test_route(bw, torch_cuda, oracle_mod, S, C, E, Q, key_blocks):
    rng = np.random.default_rng(S + Q)
    parent = evgen.make_tree(S, "fork", rng)
    ev, qs = evgen.make_events(S, C, E, rng), evgen.make_queries(S, C, Q, rng)
    p, e, q = evgen.to_device(torch_cuda, parent, ev, qs)
    auto, general = bw.Replay(p, C, E, Q), bw.Replay(p, C, E, Q, path="general")
    got = torch_cuda.empty(Q, dtype=torch_cuda.int64, device="cuda")
    want = oracle_mod.ev_sweep(parent, C, ev, qs)
    for plan in (general, auto):
        plan.launch(p, e, q, got)
        assert plan.status() == 0
        np.testing.assert_array_equal(got.cpu().numpy(), want)
    assert (auto.workspace.numel() != general.workspace.numel()) == key_blocks
