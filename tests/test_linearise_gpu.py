"""GPU parity of the tour building at the sizes where its kernels change.

The inclusive scans sum the totals of earlier tiles in the kernel that applies them up to
2,048 tiles of 4,096 elements (twice the states), above in a kernel of their own; tours
below 2^24 states are built by chained launches.  Whole numbers, compared exactly with the chain path or the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import evgen

pytestmark = pytest.mark.gpu


def run(bw, torch, p, C, e, q, **kw):
    r = bw.Replay(p, C, e.shape[0], q.shape[0], **kw)
    out = torch.empty(q.shape[0], dtype=torch.int64, device=p.device)
    r.launch(p, e, q, out)
    assert r.status() == 0
    return out.cpu().numpy()


@pytest.mark.parametrize("S", [4 << 20, (4 << 20) + 1, (1 << 24) - 1, 1 << 24])
def test_scan_of_many_tiles(bw, torch_cuda, S):
    rng = np.random.default_rng(S)
    C, E, Q = 300, 50_000, 5000
    parent = evgen.make_tree(S, "chain", rng)
    ev, qs = evgen.make_events(S, C, E, rng, big=True), evgen.make_queries(S, C, Q, rng)
    p, e, q = evgen.to_device(torch_cuda, parent, ev, qs)
    want = run(bw, torch_cuda, p, C, e, q, chain=True, path="chain")
    np.testing.assert_array_equal(run(bw, torch_cuda, p, C, e, q), want)
