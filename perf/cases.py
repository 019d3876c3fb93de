"""The framework's work as a user has it done: replays of version chains, trees and
forests, the sparse-key index, grouping of ungrouped logs and the served store, from
the smallest calls to the sizes of the configured workloads (workloads.py), made on
the GPU from a seed.

``listed()`` gives the named cases, ``draw(rng)`` one more of the same ranges,
``prepare`` the inputs and the handles a program keeps, ``run`` one pass through the
public entry points, ``work`` what a pass cannot do without, ``exact`` the answers
from plain torch (a list-ranked Euler tour and a wavelet matrix with prefix sums)."""
import importlib
import math
from statistics import NormalDist

import numpy as np
import torch

bw = importlib.import_module("biworlddb-artifact_gb300")

# Deltas: cents of a trip or a sale (workloads.py), or the products amount x factor of
# the reference-native workloads, which mostly leave the int32 range.
CENTS, PRODUCTS = "cents", "products"


def listed():
    return [
        # one short history asked a few questions: one call, the answers checked
        dict(name="chain_small", kind="chain", states=501, events=25_003, queries=251, keys=4096, deltas=CENTS,
             width=256, plan=False),
        # the plain chain as configured, through a plan that is kept
        dict(name="chain_plain", kind="chain", states=20_000, events=1_000_000, queries=10_000, keys=4096,
             deltas=CENTS, width=256, plan=True),
        # the same history a hundred times as long
        dict(name="chain_large", kind="chain", states=2_000_000, events=100_000_000, queries=1_000_000, keys=4096,
             deltas=CENTS, width=256, plan=True),
        # a reference-native chain: factor edits that touch a whole support, deltas
        # beyond 32 bits, two queries a state
        dict(name="chain_native", kind="native", states=300_000, edits=4000, support=1700, queries=599_998,
             keys=3429, deltas=PRODUCTS),
        # the trip-log tree, more queries than events
        dict(name="tree_trip", kind="tree", states=300_000, events=40_000_000, queries=50_000_000, keys=65536,
             deltas=CENTS, width=0, extend=0.9),
        # a smaller log as it arrives: events and queries in arrival order, grouped on
        # the device, replayed, the answers put back in arrival order
        dict(name="tree_ungrouped", kind="ungrouped", states=30_011, events=4_000_037, queries=5_000_011, keys=65536,
             deltas=CENTS, width=0, extend=0.9),
        # a few dozen uneven trees in one launch
        dict(name="forest_small", kind="forest", trees=61, median=2000, cap=20_000, per_state=8, queries=1000,
             bits_lo=10, bits_hi=18, graph=False),
        # the batched uneven trees as configured, one graph launch
        dict(name="forest_batched", kind="forest", trees=4096, median=2000, cap=200_000, per_state=8, queries=1000,
             bits_lo=10, bits_hi=18, graph=True),
        # index build over sparse 40-bit keys
        dict(name="csr_build", kind="csr_build", distinct=10_000_000, items=20_000_000, lut_mib=64),
        # point and range rank lookups in that index, half present and half absent
        dict(name="csr_lookup", kind="csr_lookup", distinct=10_000_000, items=20_000_000, lookups=100_000_000,
             lut_mib=64),
        # a version tree over sparse keys: index, rank mapping and range answers
        dict(name="versioned", kind="versioned", states=100_000, distinct=10_000_000, events=20_000_000,
             lookups=100_000_000, ranges=True),
        # requests to a served store, all pending at once: queries, commits and forks
        dict(name="served", kind="served", states=30_000, events=4_000_000, keys=65536, requests=200_000),
    ]


def _log(rng, lo, hi):
    """A whole number of [lo, hi], spread over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["chain", "chain", "native", "tree", "tree", "ungrouped", "forest", "forest", "csr_build",
                       "csr_lookup", "versioned", "served"])
    if kind == "chain":
        events = _log(rng, 25_000, 60_000_000)
        return dict(kind=kind, states=_log(rng, 300, max(301, events // 8)), events=events,
                    queries=_log(rng, 200, max(201, events // 40)), keys=_log(rng, 500, 32768), deltas=CENTS,
                    width=rng.choice([64, 256, 1024]), plan=rng.random() < 0.7)
    if kind == "native":
        states = _log(rng, 5000, 300_000)
        return dict(kind=kind, states=states, edits=max(1, states // rng.randint(60, 120)),
                    support=rng.randint(300, 1700), queries=rng.choice([1, 2]) * (states - 1),
                    keys=rng.randint(1800, 4000), deltas=PRODUCTS)
    if kind in ("tree", "ungrouped"):
        events = _log(rng, 200_000, 20_000_000 if kind == "tree" else 4_000_000)
        return dict(kind=kind, states=_log(rng, 2000, max(2001, min(300_000, events // 16))), events=events,
                    queries=_log(rng, 2000, events), keys=_log(rng, 4000, 65536), deltas=CENTS,
                    width=rng.choice([0, 1024]), extend=rng.choice([0.7, 0.9, 0.99]))
    if kind == "forest":
        lo = rng.randint(8, 16)
        return dict(kind=kind, trees=_log(rng, 16, 2048), median=_log(rng, 200, 2000),
                    cap=rng.choice([20_000, 100_001]), per_state=rng.choice([2, 8, 12]),
                    queries=_log(rng, 50, 1000), bits_lo=lo, bits_hi=rng.randint(lo, 18), graph=rng.random() < 0.5)
    if kind == "csr_build":
        distinct = _log(rng, 50_000, 10_000_000)
        return dict(kind=kind, distinct=distinct, items=int(distinct * rng.uniform(1.0, 2.0)),
                    lut_mib=rng.choice([16, 64, 256]))
    if kind == "csr_lookup":
        distinct = _log(rng, 50_000, 10_000_000)
        return dict(kind=kind, distinct=distinct, items=int(distinct * rng.uniform(1.0, 2.0)),
                    lookups=_log(rng, 500_000, 80_000_000), lut_mib=rng.choice([16, 64, 256]))
    if kind == "versioned":
        distinct = _log(rng, 300_000, 3_000_000)
        events = int(distinct * rng.uniform(1.0, 2.0))
        return dict(kind=kind, states=_log(rng, 2000, 100_000), distinct=distinct, events=events,
                    lookups=_log(rng, 200_000, 5 * events), ranges=rng.random() < 0.5)
    states = _log(rng, 2000, 30_000)
    return dict(kind=kind, states=states, events=states * rng.randint(20, 130), keys=_log(rng, 4096, 65536),
                requests=_log(rng, 10_000, 200_000))


# ---------------------------------------------------------------------- inputs
def _gen(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1_000_003 + salt)


def _rand(g, n):
    return torch.rand(n, generator=g, device="cuda", dtype=torch.float64)


def _ints(g, lo, hi, n):
    return torch.randint(lo, hi, (n,), generator=g, device="cuda", dtype=torch.int64)


def _zipf(g, n, C, s):
    """Zipf ranks scattered over the domain by a permutation."""
    cdf = torch.cumsum(torch.arange(1, C + 1, device="cuda", dtype=torch.float64) ** (-s), 0)
    cdf = cdf / cdf[-1].clone()
    perm = torch.randperm(C, generator=g, device="cuda")
    return perm[torch.searchsorted(cdf, _rand(g, n)).clamp_(max=C - 1)]


def _deltas(g, n, what, signs=True):
    d = torch.empty(n, device="cuda", dtype=torch.float64).log_normal_(7.0, 1.0, generator=g).round_().long()
    if what == PRODUCTS:
        d = d * _ints(g, 2, 8, n) * _ints(g, 300, 3000, n)
    if signs:
        d = torch.where(_rand(g, n) < 0.1, -d, d)
    return d


def _grouped(g, n, S):
    """n states of [0, S), uniform, in ascending order."""
    return torch.repeat_interleave(torch.bincount(_ints(g, 0, S, n), minlength=S))


def _chain_parent(S):
    return torch.arange(-1, S - 1, device="cuda", dtype=torch.int32)


def _fork_parent(g, S, extend):
    v = torch.arange(S, device="cuda")
    fork = (_rand(g, S) >= extend) & (v >= 2)
    return torch.where(fork, (_rand(g, S) * v).long(), v - 1).int()


def _intervals(g, n, C, width):
    """[lo, hi): both ends uniform (width 0), or lo uniform and a geometric width."""
    if width == 0:
        a, b = _ints(g, 0, C + 1, n), _ints(g, 0, C + 1, n)
        return torch.minimum(a, b), torch.maximum(a, b)
    lo = _ints(g, 0, C, n)
    w = torch.empty(n, device="cuda", dtype=torch.float64).geometric_(1.0 / width, generator=g).long()
    return lo, (lo + w).clamp_(max=C)


def _events(state, key, delta):
    return torch.stack([state | (key << 32), delta], 1)


def _queries(state, lo, hi):
    return torch.stack([state.int(), lo.int(), hi.int()], 1)


def _tree_inputs(c, seed):
    """parent, (event state, key, delta), (query state, lo, hi), all grouped by state."""
    g = _gen(seed)
    S, C = c["states"], c["keys"]
    if c["kind"] == "native":
        # row edits at every state, and every few states an edit of a whole support
        n, sup = c["edits"], min(c["support"], C)
        fs = torch.randperm(S - 1, generator=g, device="cuda")[:n] + 1
        off = _ints(g, 0, C - sup + 1, n)
        es = torch.cat([torch.arange(S, device="cuda"), fs.repeat_interleave(sup)])
        ek = torch.cat([_ints(g, 0, C, S), (off[:, None] + torch.arange(sup, device="cuda")).reshape(-1)])
        order = torch.argsort(es, stable=True)
        es, ek = es[order], ek[order]
        ed = _deltas(g, es.numel(), c["deltas"])
        qs = 1 + torch.arange(c["queries"], device="cuda") * (S - 1) // c["queries"]
        return _chain_parent(S), (es, ek, ed), (qs, *_intervals(g, c["queries"], C, 0))
    parent = _chain_parent(S) if c["kind"] == "chain" else _fork_parent(g, S, c["extend"])
    s = 1.1 if c["kind"] == "chain" else 1.2
    ev = (_grouped(g, c["events"], S), _zipf(g, c["events"], C, s), _deltas(g, c["events"], c["deltas"]))
    return parent, ev, (_grouped(g, c["queries"], S), *_intervals(g, c["queries"], C, c["width"]))


def _forest_sizes(c):
    """States per tree: the quantiles of a lognormal (sigma 1.6) about the median."""
    T, nd = c["trees"], NormalDist()
    z = [nd.inv_cdf((i + 0.5) / T) for i in range(T)]
    return np.array([min(c["cap"], max(2, round(c["median"] * math.exp(1.6 * x)))) for x in z], dtype=np.int64)


def _forest_inputs(c, seed):
    """Offsets and key domains (host), parent, events and queries (device, concatenated)."""
    rng, g = np.random.default_rng(seed), _gen(seed)
    T, Q = c["trees"], c["queries"]
    size = rng.permutation(_forest_sizes(c))
    bits = rng.integers(c["bits_lo"], c["bits_hi"] + 1, size=T)
    soff = np.concatenate([[0], np.cumsum(size)])
    S = int(soff[-1])
    E = S * c["per_state"]
    d_soff, d_size = torch.from_numpy(soff).cuda(), torch.from_numpy(size).cuda()
    tree = torch.repeat_interleave(d_size)
    local = torch.arange(S, device="cuda") - d_soff[tree]
    fork = (_rand(g, S) >= 0.95) & (local >= 2)
    parent = torch.where(fork, (_rand(g, S) * local).long(), local - 1).int()
    gs = _grouped(g, E, S)
    eoff = torch.searchsorted(gs, d_soff).cpu().numpy()
    et = tree[gs]
    key = torch.empty(E, device="cuda", dtype=torch.int64)
    eb = torch.from_numpy(bits).cuda()[et]
    for b in range(c["bits_lo"], c["bits_hi"] + 1):
        at = torch.nonzero(eb == b).reshape(-1)
        key[at] = _zipf(g, at.numel(), 1 << b, 1.1)
    del eb, et
    events = _events(local[gs], key, _deltas(g, E, CENTS))
    qt = torch.arange(T, device="cuda").repeat_interleave(Q)
    qs = torch.sort(qt + _rand(g, T * Q).clamp_(max=1 - 2.0 ** -30))[0] - qt
    qs = torch.minimum((qs * d_size[qt]).long(), d_size[qt] - 1)
    C = torch.from_numpy(1 << bits).cuda()[qt]
    a, b = ((_rand(g, T * Q) * (C + 1)).long() for _ in range(2))
    queries = _queries(qs, torch.minimum(a, b), torch.maximum(a, b))
    return soff, eoff, np.arange(T + 1, dtype=np.int64) * Q, (1 << bits).astype(np.uint32), parent, events, queries


def _sparse(c, seed):
    """Distinct even keys of [0, 2^40), items on them (each at least once), and a
    function that draws lookup keys, half present and half absent (odd)."""
    g = _gen(seed)
    K, step = c["distinct"], (1 << 39) // c["distinct"]
    distinct = (torch.arange(K, device="cuda") * step + _ints(g, 0, step, K)) * 2
    n = c.get("items", c.get("events"))
    pick = torch.cat([torch.randperm(K, generator=g, device="cuda"), _ints(g, 0, K, n - K)])

    def mixed(m):
        return torch.where(_rand(g, m) < 0.5, distinct[_ints(g, 0, K, m)], _ints(g, 0, 1 << 39, m) * 2 + 1)
    return g, distinct[pick], _deltas(g, n, CENTS), mixed


def _lookups(c, seed):
    g, keys, amounts, mixed = _sparse(c, seed)
    a, b = mixed(c["lookups"]), mixed(c["lookups"])
    return keys, amounts, mixed(c["lookups"]), torch.stack([torch.minimum(a, b), torch.maximum(a, b)], 1)


def _versioned(c, seed):
    g, keys, deltas, mixed = _sparse(c, seed)
    parent = _fork_parent(g, c["states"], 0.9)
    es, qs = _grouped(g, keys.numel(), c["states"]), _grouped(g, c["lookups"], c["states"])
    a = mixed(c["lookups"])
    b = mixed(c["lookups"]) if c["ranges"] else a
    lo, hi = (torch.minimum(a, b), torch.maximum(a, b)) if c["ranges"] else (a, None)
    return parent, es, keys, deltas, qs, lo, hi


def _served(c, seed):
    """An initial tree and a request log: 90 % queries, 8 % commits of 1-64 events to a
    live leaf, 2 % forks of any version (workloads.serving)."""
    tree = dict(c, kind="tree", extend=0.9, queries=1, width=0, deltas=CENTS)
    parent, (es, ek, ed), _ = _tree_inputs(tree, seed)
    events = _events(es, ek, ed).cpu().numpy().view(bw.workloads.EVENT_DTYPE).reshape(-1)
    parent = parent.cpu().numpy()
    rng = np.random.default_rng(seed + 7)
    n, S, C = c["requests"], c["states"], c["keys"]
    u = rng.random(n)
    req = np.zeros(n, dtype=bw.workloads.REQUEST_DTYPE)
    kind = np.where(u < 0.9, 0, np.where(u < 0.98, 1, 2))
    made = np.cumsum(kind != 0) - (kind != 0)
    req["kind"] = kind
    req["version"] = rng.random(n) * (S + made)
    req["lo"] = rng.integers(0, C, size=n)
    req["hi"] = np.minimum(req["lo"] + rng.geometric(1 / 1024, size=n), C)
    leaf = np.ones(S, dtype=bool)
    leaf[parent[1:]] = False
    leaves = np.nonzero(leaf)[0].tolist()
    for i in np.nonzero(kind)[0].tolist():
        new = S + int(made[i])
        if kind[i] == 1:        # the leaf is extended
            j = int(u[i] * 1e9) % len(leaves)
            req["version"][i], leaves[j] = leaves[j], new
        else:
            leaves.append(new)
        req["new_version"][i] = new
    req["lo"][kind != 0] = req["hi"][kind != 0] = 0
    req["n_events"] = np.where(kind == 1, rng.integers(1, 65, size=n), 0)
    req["events_off"] = np.where(kind == 1, np.cumsum(req["n_events"]) - req["n_events"], 0)
    cev = np.zeros(int(req["n_events"].sum()), dtype=bw.workloads.EVENT_DTYPE)
    cev["state"] = np.repeat(req["new_version"], req["n_events"])
    g = _gen(seed, 9)
    cev["key"] = _zipf(g, cev.size, C, 1.2).cpu().numpy()
    cev["delta"] = _deltas(g, cev.size, CENTS).cpu().numpy()
    return parent, events, req, cev


# ---------------------------------------------------------------------- cases
def prepare(case, seed):
    c, k = case, case["kind"]
    st = {"case": c}
    if k in ("chain", "native", "tree", "ungrouped"):
        parent, ev, qs = _tree_inputs(c, seed)
        st["parent"], st["events"], st["queries"] = parent, _events(*ev), _queries(*qs)
        if k == "ungrouped":
            g = _gen(seed, 5)
            st["events"] = st["events"][torch.randperm(c["events"], generator=g, device="cuda")]
            st["queries"] = st["queries"][torch.randperm(c["queries"], generator=g, device="cuda")]
        elif k != "chain" or c["plan"]:
            st["plan"] = bw.Replay(parent, c["keys"], st["events"].shape[0], c["queries"], chain=k != "tree",
                                   wide=c["deltas"] == PRODUCTS)
            st["answers"] = torch.empty(c["queries"], dtype=torch.int64, device="cuda")
    elif k == "forest":
        *shape, parent, events, queries = _forest_inputs(c, seed)
        st["in"] = (parent, events, queries, torch.empty(len(queries), dtype=torch.int64, device="cuda"))
        st["plan"] = bw.Forest(*shape)
        if c["graph"]:
            st["plan"].capture(*st["in"], torch.cuda.Stream())
    elif k == "csr_build":
        _, st["keys"], st["amounts"], _ = _sparse(c, seed)
    elif k == "csr_lookup":
        keys, amounts, st["points"], st["bounds"] = _lookups(c, seed)
        st["index"] = bw.CsrIndex(keys, amounts, lut_budget_bytes=c["lut_mib"] << 20)
    elif k == "versioned":
        parent, es, keys, deltas, qs, lo, hi = _versioned(c, seed)
        st["in"] = (parent, es.int(), keys, deltas, qs.int(), lo, hi)
    else:
        parent, events, st["requests"], st["commits"] = _served(c, seed)
        made = int((st["requests"]["kind"] != 0).sum())
        st["server"] = bw.Server(parent, c["keys"], events, max_versions=c["states"] + made,
                                 max_events=len(events) + len(st["commits"]), hbm_cap_bytes=20 << 30)
    return st


def run(state):
    c, k = state["case"], state["case"]["kind"]
    if k == "ungrouped":
        ev, qs, order = bw.group_by_state(c["states"], state["events"], state["queries"])
        answers = bw.replay(state["parent"], c["keys"], ev, qs)
        return bw.scatter_device_answers(answers, order, c["queries"])
    if k in ("chain", "native", "tree"):
        if "plan" not in state:
            return bw.replay(state["parent"], c["keys"], state["events"], state["queries"], chain=True)
        state["plan"].launch(state["parent"], state["events"], state["queries"], state["answers"])
        return state["answers"]
    if k == "forest":
        if c["graph"]:
            state["plan"].replay()
        else:
            state["plan"].launch(*state["in"])
        return state["in"][3]
    if k == "csr_build":
        keys, pre = bw.CsrIndex(state["keys"], state["amounts"], lut_budget_bytes=c["lut_mib"] << 20).arrays()
        return keys, pre
    if k == "csr_lookup":
        return state["index"].point(state["points"]), state["index"].range(state["bounds"])
    if k == "versioned":
        return bw.versioned_sparse_replay(*state["in"])[0]
    state["server"].reset()
    return state["server"].run(state["requests"], state["commits"])[0]


def work(case):
    """Bytes: each input once, each output once.  Sums of int64: no floating operations."""
    c, k = case, case["kind"]
    if k == "forest":
        S = int(_forest_sizes(c).sum())
        n = 4 * S + 16 * S * c["per_state"] + 20 * c["trees"] * c["queries"]
    elif k == "native":
        n = 4 * c["states"] + 16 * (c["states"] + c["edits"] * min(c["support"], c["keys"])) + 20 * c["queries"]
    elif k in ("chain", "tree", "ungrouped"):
        n = 4 * c["states"] + 16 * c["events"] + 20 * c["queries"]
    elif k == "csr_build":
        n = 16 * c["items"] + 16 * c["distinct"]
    elif k == "csr_lookup":
        n = (8 + 8 + 16 + 16) * c["lookups"]
    elif k == "versioned":
        n = 4 * c["states"] + 20 * c["events"] + (28 if c["ranges"] else 20) * c["lookups"]
    else:   # requests, their answers and latencies, the commits' events (32.5 each on 8 %)
        n = int(44 * c["requests"] + 0.08 * 32.5 * 16 * c["requests"])
    return {"bytes": n, "flops": 0}


# ---------------------------------------------------------------------- the exact answers
def _tour(parent):
    """First and last position of every state's subtree in an Euler tour of 2S steps
    (the trees of a forest one after another), by list ranking."""
    S = parent.numel()
    v = torch.arange(S, device="cuda")
    order = torch.argsort(parent, stable=True)          # children of a state side by side
    p = parent[order]
    first = torch.full((S + 1,), -1, device="cuda", dtype=torch.int64)
    head = torch.ones(S, dtype=torch.bool, device="cuda")
    head[1:] = p[1:] != p[:-1]
    first[p[head]] = order[head]                         # roots write the spare last entry
    sib = torch.full((S,), -1, device="cuda", dtype=torch.int64)
    sib[order[:-1]] = torch.where(head[1:], -1, order[1:])
    up = torch.where(parent >= 0, S + parent, 2 * S)
    nxt = torch.cat([torch.where(first[:S] >= 0, first[:S], S + v), torch.where(sib >= 0, sib, up),
                     torch.tensor([2 * S], device="cuda")])
    dist = torch.ones(2 * S + 1, device="cuda", dtype=torch.int64)
    dist[2 * S] = 0
    for _ in range(int(2 * S).bit_length()):
        dist = dist + dist[nxt]
        nxt = nxt[nxt]
    return 2 * S - dist[:S], 2 * S - dist[S:2 * S]


def _dominance(pos, key, val, qpos, qkeys, C):
    """For every k of qkeys: the sum of val over pos <= qpos and key < k (pos in any
    order), by a wavelet matrix over the keys with the values' prefix sums."""
    order = torch.argsort(pos)
    key, val = key[order].int(), val[order]
    r = torch.searchsorted(pos[order], qpos, right=True)
    del order
    probes = [[torch.zeros_like(r), r, k, torch.zeros_like(r)] for k in qkeys]
    zero = torch.zeros(1, device="cuda", dtype=torch.int64)
    for bit in range(int(C).bit_length() - 1, -1, -1):
        low = (key >> bit & 1) == 0
        Z = torch.cat([zero, torch.cumsum(low, 0)])
        W = torch.cat([zero, torch.cumsum(torch.where(low, val, 0), 0)])
        for x in probes:
            l, e, k, s = x
            one = (k >> bit & 1) == 1
            s += torch.where(one, W[e] - W[l], 0)
            zl, ze = Z[l], Z[e]
            x[0], x[1] = torch.where(one, Z[-1] + l - zl, zl), torch.where(one, Z[-1] + e - ze, ze)
        del W, Z
        key, val = torch.cat([key[low], key[~low]]), torch.cat([val[low], val[~low]])
    return [x[3] for x in probes]


def _answers(parent, ev, qs, C):
    """Range sums over the root paths; parent, states and bounds global, C above all keys."""
    (es, ek, ed), (st, lo, hi) = ev, qs
    tin, tout = _tour(parent)
    pos = torch.cat([tin[es], tout[es]])
    below_lo, below_hi = _dominance(pos, torch.cat([ek, ek]), torch.cat([ed, -ed]), tin[st], (lo, hi), C)
    return torch.where(hi > lo, below_hi - below_lo, 0)


def _unpack(events, queries):
    s = events[:, 0]
    q = queries.long()
    return (s & 0xffffffff, s >> 32, events[:, 1]), (q[:, 0], q[:, 1], q[:, 2])


def _index(keys, amounts):
    uniq, at = torch.unique(keys, return_inverse=True)
    return uniq, torch.cumsum(torch.zeros_like(uniq).index_add_(0, at, amounts), 0)


def exact(case, seed):
    c, k = case, case["kind"]
    if k in ("chain", "native", "tree"):
        parent, ev, qs = _tree_inputs(c, seed)
        return _answers(parent.long(), ev, qs, c["keys"])
    if k == "ungrouped":
        st = prepare(c, seed)
        return _answers(st["parent"].long(), *_unpack(st["events"], st["queries"]), c["keys"])
    if k == "forest":
        soff, eoff, qoff, keys, parent, events, queries = _forest_inputs(c, seed)
        base = torch.from_numpy(soff[:-1]).cuda()
        (es, ek, ed), (st, lo, hi) = _unpack(events, queries)
        del events
        up = torch.repeat_interleave(base, torch.from_numpy(np.diff(soff)).cuda())
        es = es + torch.repeat_interleave(base, torch.from_numpy(np.diff(eoff)).cuda())
        st = st + base.repeat_interleave(c["queries"])
        parent = torch.where(parent < 0, -1, parent + up)
        return _answers(parent, (es, ek, ed), (st, lo, hi), 1 << c["bits_hi"])
    if k == "csr_build":
        _, keys, amounts, _ = _sparse(c, seed)
        return _index(keys, amounts)
    if k == "csr_lookup":
        keys, amounts, points, bounds = _lookups(c, seed)
        uniq, pre = _index(keys, amounts)
        pre = torch.cat([torch.zeros(1, device="cuda", dtype=torch.int64), pre])
        r = torch.searchsorted(uniq, points)
        found = uniq[r.clamp(max=uniq.numel() - 1)] == points
        b = torch.searchsorted(uniq, bounds)
        return torch.where(found, r, -r - 1), torch.stack([b[:, 1] - b[:, 0], pre[b[:, 1]] - pre[b[:, 0]]], 1)
    if k == "versioned":
        parent, es, keys, deltas, qs, lo, hi = _versioned(c, seed)
        uniq, ek = torch.unique(keys, return_inverse=True)
        a = torch.searchsorted(uniq, lo)
        b = torch.searchsorted(uniq, hi if c["ranges"] else lo, right=not c["ranges"])
        return _answers(parent.long(), (es, ek, deltas), (qs, a, b), uniq.numel())
    parent, events, req, cev = _served(c, seed)
    made = req["kind"] != 0
    up = lambda a: torch.from_numpy(a.astype(np.int64)).cuda()  # noqa: E731
    ev = tuple(up(np.concatenate([events[f], cev[f]])) for f in ("state", "key", "delta"))
    q = req["kind"] == 0
    got = _answers(up(np.concatenate([parent, req["version"][made].astype(np.int32)])), ev,
                   tuple(up(req[f][q]) for f in ("version", "lo", "hi")), c["keys"])
    out = np.zeros(len(req), dtype=np.int64)
    out[q] = got.cpu().numpy()
    return out
