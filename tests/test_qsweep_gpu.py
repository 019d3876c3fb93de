"""GPU parity of the query-step sweep at its own edges: many blocks."""
from __future__ import annotations

import numpy as np
import pytest

import evgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blocks", [65_535, 65_536, 70_000])
def test_many_blocks(bw, torch_cuda, oracle_mod, blocks):
    S, C, E, Q = 20_000, 16, 60_000, 360_000
    rng = np.random.default_rng(blocks)
    parent = evgen.make_tree(S, "fork", rng)
    ev, qs = evgen.make_events(S, C, E, rng), evgen.make_queries(S, C, Q, rng)
    p, e, q = evgen.to_device(torch_cuda, parent, ev, qs)
    got = bw.replay(p, C, e, q, blocks=blocks).cpu().numpy()
    np.testing.assert_array_equal(got, oracle_mod.ev_sweep(parent, C, ev, qs))
