"""GPU parity of single trees whose block holds the keys of more than 256 windows of the
sweep: one block, every key of the domain touched, int64 windows."""
from __future__ import annotations

import numpy as np
import pytest

import evgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,C,Q", [(100, 1_300_000, 6000),    # query steps: windows of 4,095 ranks
                                   (40, 3_800_000, 100)])     # Euler tiles: of 13,824
def test_many_windows(bw, torch_cuda, oracle_mod, S, C, Q):
    rng = np.random.default_rng(C)
    parent = evgen.make_tree(S, "fork", rng)
    ev, qs = evgen.make_events(S, C, C, rng, big=True), evgen.make_queries(S, C, Q, rng)
    ev["key"] = rng.permutation(C)
    p, e, q = evgen.to_device(torch_cuda, parent, ev, qs)
    got = bw.replay(p, C, e, q, blocks=1).cpu().numpy()
    np.testing.assert_array_equal(got, oracle_mod.ev_sweep(parent, C, ev, qs))
