"""Lookups of the sparse index around the sizes where they change their way: key counts of
4,096 (LUTs of 2^18 buckets and more) and 65,536, 64 MiB of inputs, outputs and LUT, a million
ranges.  Compared with numpy."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lut", [1 << 16, 1 << 20, 1 << 26])
@pytest.mark.parametrize("keys", [1, 4095, 4096, 65_535, 65_536])
@pytest.mark.parametrize("n", [1, 999_999, 1_000_001, 4_200_001])
def test_lookups(bw, torch_cuda, keys, lut, n):
    torch = torch_cuda
    rng = np.random.default_rng(keys + n)
    key = np.sort(rng.choice(1 << 40, keys, replace=False).astype(np.int64))
    amount = rng.integers(-(1 << 62), 1 << 62, keys)
    perm = rng.permutation(keys)
    idx = bw.CsrIndex(torch.from_numpy(key[perm]).cuda(), torch.from_numpy(amount[perm]).cuda(), lut_budget_bytes=lut)
    assert idx.status() == 0 and idx.count() == keys
    probe = rng.integers(0, 1 << 40, n)
    hit = rng.random(n) < 0.5
    probe[hit] = key[rng.integers(0, keys, int(hit.sum()))]
    rank = np.searchsorted(key, probe)
    present = key[np.minimum(rank, keys - 1)] == probe
    got = idx.point(torch.from_numpy(probe).cuda()).cpu().numpy()
    np.testing.assert_array_equal(got, np.where(present, rank, -rank - 1))
    if n > 2_000_000:
        probe = probe[:2_200_002]
    bounds = np.sort(probe[: len(probe) // 2 * 2].reshape(-1, 2), axis=1) if n > 1 else np.array([[0, probe[0]]])
    pre = np.concatenate([[0], np.cumsum(amount)])   # wraps like the index
    r = np.searchsorted(key, bounds)
    got = idx.range(torch.from_numpy(np.ascontiguousarray(bounds)).cuda()).cpu().numpy()
    np.testing.assert_array_equal(got, np.stack([r[:, 1] - r[:, 0], pre[r[:, 1]] - pre[r[:, 0]]], axis=1))
