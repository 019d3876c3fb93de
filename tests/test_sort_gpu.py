"""The radix partition behind the index build and the grouping, at the edges of its
tiles (2,048 items), chunks and passes, against numpy."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 31, 2047, 2048, 2049, 4095, 4096, 4097, 3 * 4096 + 1, 300 * 4096 + 77]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("n_states", [1, 200, 256, 257, 70_000, 1 << 24])
def test_grouping_is_stable(bw, torch_cuda, n, n_states):
    torch = torch_cuda
    rng = np.random.default_rng(n + n_states)
    st = rng.integers(0, n_states, n) if n % 2 else np.minimum(rng.geometric(0.01, n) - 1, n_states - 1)
    ev = np.stack([st | (np.arange(n) << 32), rng.integers(-9, 9, n)], 1)
    qs = np.stack([st, np.arange(n), rng.integers(0, 9, n)], 1).astype(np.int32)
    e, q, order = bw.group_by_state(n_states, torch.from_numpy(ev).cuda(), torch.from_numpy(qs).cuda())
    want = np.argsort(st, kind="stable")
    np.testing.assert_array_equal(e.cpu().numpy(), ev[want])
    np.testing.assert_array_equal(q.cpu().numpy(), qs[want])
    np.testing.assert_array_equal(order.cpu().numpy(), want)


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("bits,distinct", [(1, 2), (8, 200), (9, 3), (40, 1 << 40), (40, 1000), (63, 1 << 62), (40, 1)])
def test_index_build(bw, torch_cuda, n, bits, distinct):
    torch = torch_cuda
    rng = np.random.default_rng(n + bits)
    keys = rng.integers(0, distinct, n) * ((1 << bits) // max(distinct, 1) if distinct < 1 << 20 else 1) & ((1 << bits) - 1)
    amounts = rng.integers(np.iinfo(np.int64).min, np.iinfo(np.int64).max, n)
    idx = bw.CsrIndex(torch.from_numpy(keys).cuda(), torch.from_numpy(amounts).cuda(), key_bits=bits,
                      lut_budget_bytes=1 << 16)
    k, pre = (x.cpu().numpy() for x in idx.arrays())
    uniq, at = np.unique(keys, return_inverse=True)
    sums = np.zeros(uniq.size, np.uint64)
    np.add.at(sums, at, amounts.astype(np.uint64))
    np.testing.assert_array_equal(k, uniq)
    np.testing.assert_array_equal(pre, np.cumsum(sums, dtype=np.uint64).astype(np.int64))
    assert idx.status() == 0
    # lookups: every key, its neighbours, and ranges between them in both directions
    probe = np.unique(np.concatenate([uniq[:500], uniq[-500:], uniq[:500] + 1, [0, (1 << bits) - 1]]))
    probe = probe[probe <= (1 << bits) - 1]
    r = np.searchsorted(uniq, probe)
    found = uniq[np.minimum(r, uniq.size - 1)] == probe
    got = idx.point(torch.from_numpy(probe).cuda()).cpu().numpy()
    np.testing.assert_array_equal(got, np.where(found, r, -r - 1))
    pair = np.stack([rng.permutation(probe), probe], 1)
    b = np.searchsorted(uniq, pair)
    p0 = np.concatenate([[0], pre])
    got = idx.range(torch.from_numpy(pair).cuda()).cpu().numpy()
    np.testing.assert_array_equal(got, np.stack([b[:, 1] - b[:, 0], p0[b[:, 1]] - p0[b[:, 0]]], 1))


def test_out_of_range_state_and_key(bw, torch_cuda):
    torch = torch_cuda
    ev = torch.zeros((5000, 2), dtype=torch.int64, device="cuda")
    ev[4999, 0] = 300
    with pytest.raises(ValueError, match="state id"):
        bw.group_by_state(300, ev)
    keys = torch.arange(5000, device="cuda")
    assert bw.CsrIndex(keys, keys, key_bits=12).status() == 1
