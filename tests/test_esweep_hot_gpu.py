"""GPU parity of the Euler-tile sweep where a state is asked much more than the others: steps of
60 queries and some (a tile's), 256 and some past it (a tile of their own), with events before,
behind and without, one block and many, dense windows, rank slices, forests, captured launches."""
from __future__ import annotations

import numpy as np
import pytest

import evgen

pytestmark = pytest.mark.gpu

COUNTS = [59, 60, 61, 255, 256, 257, 315, 316, 317, 375, 376, 1279, 2200, 5000]


def _case(S, C, E, Q, tree, hot, big, seed):
    rng = np.random.default_rng(seed)
    parent = evgen.make_tree(S, tree, rng)
    ev, qs = evgen.make_events(S, C, E, rng, big=big), evgen.make_queries(S, C, Q, rng)
    state = rng.integers(0, S, Q)
    if hot == "several":
        state[: sum(COUNTS)] = np.repeat(rng.choice(S, len(COUNTS), replace=False), COUNTS)
    elif hot is not None:
        state[: Q * 9 // 10] = hot % S
    qs["state"] = np.sort(state)
    return parent, ev, qs


@pytest.mark.parametrize("big", [False, True])
@pytest.mark.parametrize("S,C,E,Q,tree,hot", [
    (4000, 200, 60_000, 30_000, "fork", "several"),      # flat window
    (4000, 3000, 60_000, 30_000, "fork", "several"),     # chunk totals
    (4000, 60_000, 60_000, 30_000, "fork", "several"),   # rank slices (int64)
    (4000, 200_000, 90_000, 30_000, "star", "several"),
    (4000, 3000, 200, 30_000, "chain", "several"),       # hardly any events
    (4000, 8000, 60_000, 30_000, "fork", 0), (4000, 8000, 60_000, 30_000, "fork", -1),
    (4000, 32, 60_000, 30_000, "fork", 2000), (4000, 13_824, 60_000, 30_000, "bushy", 2000),
    (4000, 27_904, 60_000, 30_000, "fork", 77), (4000, 1, 60_000, 30_000, "fork", 77),
])
@pytest.mark.parametrize("blocks", [0, 1, 5])
def test_hot_states(bw, torch_cuda, oracle_mod, S, C, E, Q, tree, hot, big, blocks):
    parent, ev, qs = _case(S, C, E, Q, tree, hot, big, C + E)
    p, e, q = evgen.to_device(torch_cuda, parent, ev, qs)
    got = bw.replay(p, C, e, q, blocks=blocks).cpu().numpy()
    np.testing.assert_array_equal(got, oracle_mod.ev_sweep(parent, C, ev, qs))


@pytest.mark.parametrize("big", [False, True])
def test_forest_of_hot_states(bw, torch_cuda, oracle_mod, big):
    parts, so, eo, qo, keys, want = [], [0], [0], [0], [], []
    for t, (S, C, E, Q, tree, hot) in enumerate([(1, 300, 900, 4000, "chain", 0), (900, 5000, 20_000, 27_000, "fork", "several"),
                                                 (50, 70_000, 30_000, 9000, "fork", 49), (2, 17, 0, 316, "chain", 1),
                                                 (300, 29_000, 12_000, 20, "star", None)]):
        parent, ev, qs = _case(S, C, E, Q, tree, hot, big, t)
        parts.append((parent, ev, qs))
        for off, n in ((so, S), (eo, E), (qo, Q)):
            off.append(off[-1] + n)
        keys.append(C)
        want.append(oracle_mod.ev_sweep(parent, C, ev, qs))
    p, e, q = evgen.to_device(torch_cuda, *(np.concatenate(x) for x in zip(*parts)))
    got = bw.forest_replay(so, eo, qo, keys, p, e, q).cpu().numpy()
    np.testing.assert_array_equal(got, np.concatenate(want))


def test_captured_launch(bw, torch_cuda, oracle_mod):
    """A captured launch replays on new inputs: first without a state asked much, then with."""
    torch = torch_cuda
    S, C, E, Q = 4000, 3000, 60_000, 30_000
    plain, hot = _case(S, C, E, Q, "fork", None, False, 1), _case(S, C, E, Q, "fork", "several", False, 1)
    p, e, q = evgen.to_device(torch, *plain)
    f, s = bw.Forest([0, S], [0, E], [0, Q], [C]), torch.cuda.Stream()
    out = torch.empty(Q, dtype=torch.int64, device="cuda")
    f.capture(p, e, q, out, s)
    for parent, ev, qs in (plain, hot, plain):
        for dst, src in zip((p, e, q), evgen.to_device(torch, parent, ev, qs)):
            dst.copy_(src)
        out.fill_(-1)
        torch.cuda.synchronize()
        f.replay(s)
        assert f.status(s) == 0
        np.testing.assert_array_equal(out.cpu().numpy(), oracle_mod.ev_sweep(parent, C, ev, qs))
