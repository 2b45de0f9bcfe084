"""Measured cases: what users of this library have it do, through its public entry points.

A user reads automata (random ones in experiments, structured ones in
conjecture checks), picks a plan (the reference's config JSON) and asks for
the shortest reset length of each, one automaton after another
(`Context.solve`, what the command line does with a file) or many at once
(`Context.solve_batch`).  Beside that they call the kernel-level helpers on
sets of their own, and train the distance model behind `LearnedBeam`.

Searches return the bounds, whether a word came with them and its length, per
automaton.  The words themselves are left out: any shortest reset word is a
right answer, which of them is found depends on the order in which blocks of a
kernel finish, and the library has applied each word to all states before it
returns it.

Every automaton comes from the case's seed through SplitMix64.  One context
serves all the cases of a process, as a program keeps one for its lifetime.
"""
from __future__ import annotations

import json
import math
import random

import numpy as np
import torch

import synchrowords_gb300 as sw
from synchrowords_gb300.generate import batch, random_dfa, splitmix64

EXACT = json.dumps({"algorithms": [{"name": "Exact", "config": {}}]})

# the Beam and Exact entries of the reference's configs/exact.json
BEAM_EXACT = json.dumps({
    "upper_bound": "1ULL * (AUT_N - 1) * (AUT_N - 1) + 1",
    "algorithms": [
        {"name": "Beam", "config": {"presort": "indeg", "dynamic": True,
                                    "min_beam_size": "AUT_N * std::log2(AUT_N)",
                                    "max_beam_size": "AUT_N * AUT_N * std::log2(AUT_N)",
                                    "beam_exact_ratio": 0.01}},
        {"name": "Exact", "config": {"dfs_min_list_size": "8192", "bfs_small_list_size": "AUT_N * AUT_K",
                                     "dfs": True, "dfs_shortcut": True, "max_memory_mb": "12 * 1024"}}]})

# a bound of the caller's own: random automata reset far below 4 n, and a forward beam that lost its way stops there
LEARNED_EXACT = json.dumps({
    "upper_bound": "4 * AUT_N",
    "algorithms": [
        {"name": "LearnedBeam", "config": {"beam_size": "4096", "order": "model"}},
        {"name": "Exact", "config": {"dfs_min_list_size": "8192", "bfs_small_list_size": "AUT_N * AUT_K",
                                     "dfs": True, "dfs_shortcut": True, "max_memory_mb": "12 * 1024"}}]})

# the reference's configs/readme_config.json
README = json.dumps({
    "upper_bound": "1ULL * AUT_N * AUT_N * AUT_N / 6", "threads": 1, "gpu": False,
    "algorithms": [
        {"name": "Brute", "config": {"max_n": "20"}},
        {"name": "Eppstein", "config": {"transition_tables": False, "find_word": True}},
        {"name": "Beam", "config": {"presort": "indeg", "beam_size": "10"}},
        {"name": "Reduce", "config": {"min_n": "80", "list_size_threshold": "AUT_N * 16"}},
        {"name": "Exact", "config": {"dfs_min_list_size": "10000", "bfs_small_list_size": "AUT_N * 16",
                                     "dfs": True, "dfs_shortcut": True, "max_memory_mb": "2 * 1024"}}]})

PLANS = {"exact": EXACT, "beam_exact": BEAM_EXACT, "learned_exact": LEARNED_EXACT, "readme": README}


def listed():
    return [
        # the smallest call: small random automata one after another, where
        # launches and synchronisations per BFS level are the time
        {"name": "solve_n48", "kind": "solve", "plan": "exact", "n": 48, "k": 2, "count": 8},
        # the reference's middle size, one automaton at a time
        {"name": "solve_n200", "kind": "solve", "plan": "exact", "n": 200, "k": 2, "count": 4},
        # Cerny's automaton and relatives of it (a rotation and one merging
        # letter): hundreds of BFS levels of small lists
        {"name": "solve_cyclic_n28", "kind": "cyclic", "plan": "exact", "n": 28, "k": 2, "count": 4},
        # the file of the reference's README: every algorithm of its example
        # plan, three letters, the automaton reduced before the search
        {"name": "readme_n100_k3", "kind": "solve", "plan": "readme", "n": 100, "k": 3, "count": 6},
        # a served batch of small automata of one size
        {"name": "batch_n48", "kind": "batch", "plan": "exact", "n": 48, "k": 2, "count": 64},
        # a served batch of uneven automata, n in [32, 160], two or three letters
        {"name": "batch_uneven", "kind": "uneven", "plan": "exact", "n": 160, "k": 3, "count": 256},
        # the benchmark's own workload
        {"name": "batch_n200", "kind": "batch", "plan": "exact", "n": 200, "k": 2, "count": 16},
        # large automata with the reference's beam bound
        {"name": "beam_exact_n300", "kind": "batch", "plan": "beam_exact", "n": 300, "k": 2, "count": 2},
        # the learned bound: scoring on the tensor cores, then the exact search
        {"name": "learned_exact_n256", "kind": "solve", "plan": "learned_exact", "n": 256, "k": 2, "count": 3},
        # a caller's own search: which sets of a new layer contain a set seen before
        {"name": "subsets_check_n200", "kind": "subsets_check", "n": 200, "count": 1 << 16, "queries": 1 << 15,
         "proper": False},
        # a caller's own layer: sort and deduplicate (ragged size)
        {"name": "sort_unique_n150", "kind": "sort_unique", "n": 150, "count": 300007, "queries": 0, "proper": False},
        # one epoch over four automata's pairs, with the ranking term
        {"name": "train_b512", "kind": "train", "n": 96, "k": 2, "count": 2048, "automata": 4, "batch": 512,
         "rank": 1.0},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["solve", "solve", "cyclic", "readme", "batch", "batch", "uneven", "beam_exact", "learned_exact",
                       "subsets_check", "sort_unique", "train"])
    if kind == "solve":
        k = rng.choice([2, 2, 3, 4])
        n = _log_uniform(rng, 16, int(200 / math.log2(k)))
        return {"kind": "solve", "plan": "exact", "n": n, "k": k, "count": 8 if n < 100 else 4}
    if kind == "cyclic":
        return {"kind": "cyclic", "plan": "exact", "n": rng.randint(9, 31), "k": 2, "count": 4}
    if kind == "readme":
        k = rng.choice([2, 3])
        return {"kind": "solve", "plan": "readme", "n": _log_uniform(rng, 24, 120 if k == 2 else 100), "k": k, "count": 6}
    if kind == "batch":
        k = rng.choice([2, 2, 3])
        n = _log_uniform(rng, 16, int(200 / math.log2(k)))
        return {"kind": "batch", "plan": "exact", "n": n, "k": k, "count": rng.randint(33, 300) if n < 100 else rng.randint(5, 16)}
    if kind == "uneven":
        return {"kind": "uneven", "plan": "exact", "n": rng.randint(64, 160), "k": 3, "count": _log_uniform(rng, 16, 256)}
    if kind == "beam_exact":
        return {"kind": "batch", "plan": "beam_exact", "n": _log_uniform(rng, 128, 290), "k": 2, "count": 2}
    if kind == "learned_exact":
        return {"kind": "solve", "plan": "learned_exact", "n": _log_uniform(rng, 96, 250), "k": 2, "count": 3}
    if kind == "subsets_check":
        return {"kind": kind, "n": rng.randint(40, 400), "count": _log_uniform(rng, 1000, 1 << 17),
                "queries": _log_uniform(rng, 1000, 1 << 15), "proper": rng.random() < 0.5}
    if kind == "sort_unique":
        return {"kind": kind, "n": rng.randint(100, 400), "count": _log_uniform(rng, 1000, 1 << 19), "queries": 0,
                "proper": False}
    return {"kind": "train", "n": rng.randint(64, 128), "k": 2, "count": _log_uniform(rng, 700, 4096),
            "automata": rng.randint(1, 4), "batch": rng.choice([256, 512, 1024]), "rank": rng.choice([0.0, 1.0])}


_ctx = None


def _context():
    global _ctx
    if _ctx is None:
        _ctx = sw.Context(0)
    return _ctx


# ---- inputs -----------------------------------------------------------------
def _cyclic(n, d, swap):
    """Letter `swap`: q -> q + 1 mod n; the other letter: 0 -> d, others fixed (d = 1: Cerny's automaton)."""
    t = [0] * (2 * n)
    for q in range(n):
        t[2 * q + swap] = (q + 1) % n
        t[2 * q + 1 - swap] = q
    t[1 - swap] = d
    return t


def _merge_levels(n, k, t):
    """Shortest merge length of every pair of states (0 on the diagonal, -1 if the pair never merges)."""
    t = np.asarray(t).reshape(n, k)
    level = np.where(np.eye(n, dtype=bool), 0, -1)
    depth = 0
    while True:
        depth += 1
        new = np.zeros((n, n), dtype=bool)
        for a in range(k):
            new |= level[np.ix_(t[:, a], t[:, a])] >= 0
        new &= level < 0
        if not new.any():
            return level
        level[new] = depth


def _automata(case, seed):
    n, k, count = case["n"], case["k"], case["count"]
    if case["kind"] == "uneven":
        return batch(count, seed, (32, n), (2, k))
    g = splitmix64(seed)
    if case["kind"] == "cyclic":
        steps = [d for d in range(1, n) if math.gcd(d, n) == 1]
        return [(n, 2, _cyclic(n, 1 if i == 0 else steps[next(g) % len(steps)], next(g) % 2)) for i in range(count)]
    out = []
    while len(out) < count:
        t = random_dfa(n, k, next(g))
        # about one binary automaton in n has no reset word; a beam would search for one up to its bound
        if "beam" not in case["plan"] and "learned" not in case["plan"] or (_merge_levels(n, k, t) >= 0).all():
            out.append((n, k, t))
    return out


def _images(g, delta, count, lengths):
    """Images of the full set under `count` random words (word i of lengths[i] letters), a 0/1 matrix on the GPU."""
    n, k = delta.shape
    by_letter = delta.t().contiguous()
    x = torch.ones(count, n, dtype=torch.int32, device="cuda")
    for step in range(int(lengths.max())):
        to = by_letter[torch.randint(0, k, (count,), generator=g, device="cuda")]
        y = (torch.zeros_like(x).scatter_add_(1, to, x) > 0).int()
        x = torch.where((lengths > step)[:, None], y, x)
    return x


def _layer(g, delta, count):
    """A layer before its duplicates are dropped, shuffled: three quarters of the rows distinct, the others copies.
    The sets are images under words of nine letters with a tenth of their states gone, as varied as deep layers."""
    distinct = count - count // 4
    have = torch.zeros(0, delta.shape[0], dtype=torch.int32, device="cuda")
    weight = torch.randint(1, 1 << 40, (delta.shape[0],), generator=g, device="cuda")
    while len(have) < distinct:
        x = _images(g, delta, count, torch.full((count,), 9, device="cuda"))
        x = torch.cat([have, x * (torch.rand(x.shape, generator=g, device="cuda") < 0.9)])
        _, group = torch.unique(x.double() @ weight.double(), return_inverse=True)
        first = torch.full((len(x),), len(x), device="cuda").scatter_reduce_(
            0, group, torch.arange(len(x), device="cuda"), "amin")
        have = x[torch.sort(first[first < len(x)]).values[:distinct]]
    rows = torch.cat([have, have[torch.randint(0, distinct, (count - distinct,), generator=g, device="cuda")]])
    return rows[torch.randperm(count, generator=g, device="cuda")]


def _pack(x, words):
    """0/1 matrix -> rows of `words` uint64, state q = bit q % 64 of word q // 64."""
    b = np.packbits(x.to(torch.uint8).cpu().numpy(), axis=1, bitorder="little")
    out = np.zeros((x.shape[0], words * 8), dtype=np.uint8)
    out[:, :b.shape[1]] = b
    return out.view(np.uint64)


def _delta(n, k, seed):
    return torch.tensor(random_dfa(n, k, seed), device="cuda").reshape(n, k)


def _train_inputs(case, seed):
    g = torch.Generator("cuda").manual_seed(seed)
    rng = np.random.default_rng(seed)
    autos, sets, dense, labels, groups = [], [], [], [], []
    for i in range(case["automata"]):
        n = case["n"] + 7 * i
        delta = _delta(n, case["k"], seed + 1000 + i)
        depth = torch.sort(torch.randint(1, 25, (case["count"],), generator=g, device="cuda")).values
        x = _images(g, delta, case["count"], depth)
        autos.append((n, case["k"], delta.flatten().tolist()))
        sets.append(_pack(x, 8))
        dense.append(x.cpu().numpy())
        d = depth.cpu().numpy()
        labels.append((30 - d + rng.integers(-3, 4, d.size)).astype(np.float32))
        groups.append(d.astype(np.uint32))
    parts = [rng.normal(0, (2.0 / 16) ** 0.5 / 4, 16 * 64), np.zeros(64), rng.normal(0, (2.0 / 64) ** 0.5, 64 * 128),
             np.zeros(128), rng.normal(0, (2.0 / 128) ** 0.5, 128 * 128), np.zeros(128),
             rng.normal(0, (1.0 / 128) ** 0.5 / 10, 128), np.array([20.0])]
    return autos, sets, dense, labels, groups, np.concatenate(parts).astype(np.float32)


def prepare(case, seed):
    kind, ctx = case["kind"], _context()
    state = {"case": case, "ctx": ctx}
    if kind in ("solve", "cyclic", "batch", "uneven"):
        state["automata"] = _automata(case, seed)
        state["plan"] = PLANS[case["plan"]]
    elif kind in ("subsets_check", "sort_unique"):
        g = torch.Generator("cuda").manual_seed(seed)
        n = case["n"]
        delta = _delta(n, 2, seed)
        words = (n + 63) // 64
        if kind == "sort_unique":
            state["sets"] = _pack(_layer(g, delta, case["count"]), words)
        else:  # the sets of one layer (twenty letters) and new sets of the layer before
            for name, rows, length in (("sets", case["count"], 20), ("checks", case["queries"], 19)):
                state[name] = _pack(_images(g, delta, rows, torch.full((rows,), length, device="cuda")), words)
    else:
        autos, sets, _, labels, groups, params = _train_inputs(case, seed)
        state.update(autos=autos, sets=sets, labels=labels, groups=groups if case["rank"] else None, params=params)
    return state


# ---- one pass ---------------------------------------------------------------
def _answers(results):
    return {"bounds": np.array([[r.lower, r.upper] for r in results], dtype=np.int64),
            "non_synchro": np.array([r.non_synchro for r in results]),
            "word_length": np.array([-1 if r.word is None else len(r.word) for r in results], dtype=np.int64)}


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind in ("solve", "cyclic"):
        return _answers([ctx.solve(d, n, k, state["plan"]) for n, k, d in state["automata"]])
    if kind in ("batch", "uneven"):
        return _answers(ctx.solve_batch(state["automata"], state["plan"]))
    if kind == "subsets_check":
        return ctx.subsets_check(case["n"], state["sets"], state["checks"], proper=case["proper"])
    if kind == "sort_unique":
        return ctx.sort_unique(case["n"], state["sets"]).view(np.int64)
    params, loss = ctx.mlp_train(state["params"], state["autos"], state["sets"], state["labels"], epochs=1,
                                 batch=case["batch"], lr=1e-3, seed=1, groups_per_automaton=state["groups"],
                                 rank_weight=case["rank"])
    return {"params": params, "loss": loss}


# ---- what a pass cannot do without ------------------------------------------
def work(case):
    kind, n = case["kind"], case["n"]
    if kind in ("solve", "cyclic", "batch", "uneven"):
        # the tables in, a word of about n letters and the bounds out; how many
        # sets the search between them visits depends on the automaton
        return {"bytes": case["count"] * (4 * n * case["k"] + 4 * n + 16), "flops": 0}
    words = (n + 63) // 64
    if kind == "subsets_check":
        return {"bytes": 8 * words * (case["count"] + case["queries"]) + case["queries"], "flops": 0}
    if kind == "sort_unique":
        return {"bytes": 2 * 8 * words * case["count"], "flops": 0}
    pairs = case["automata"] * case["count"]
    wide = n * 64 + 64 * 128 + 128 * 128 + 128  # multiply-adds of one set's forward pass
    return {"bytes": pairs * (64 + 4 + 4) + 2 * 4 * sw.MLP_PARAMS, "flops": 6 * pairs * wide}


# ---- the training case in 64 bits -------------------------------------------
def _features(n, k, t):
    """The model's 16 features per state, standardised over the states."""
    t = np.asarray(t).reshape(n, k)
    indeg = np.zeros((n, k))
    for a in range(k):
        np.add.at(indeg[:, a], t[:, a], 1)
    total = indeg.sum(1)
    pi = np.full(n, 1.0 / n)
    for _ in range(100):
        nx = np.full(n, 0.01 / n)
        for q in range(n):
            for a in range(k):
                nx[t[q, a]] += 0.99 * pi[q] / k
        pi = nx
    rank = np.zeros(n)
    rank[np.argsort(-pi, kind="stable")] = np.arange(n) / max(1, n - 1)
    # the strongly connected component that no letter leaves: what every state of it reaches
    reach = np.eye(n, dtype=bool)
    for _ in range(n):
        more = reach.copy()
        for a in range(k):
            more |= reach[t[:, a]]
        if (more == reach).all():
            break
        reach = more
    v = 0
    while True:  # a state whose reachable set is smallest lies in a sink component
        w = min(np.flatnonzero(reach[v]), key=lambda u: (reach[u].sum(), u))
        if reach[w].sum() == reach[v].sum():
            break
        v = w
    sink = reach[v]
    pair = _merge_levels(n, k, t)
    pair[pair < 0] = n * n
    off = pair + np.where(np.eye(n, dtype=bool), 1 << 40, 0)
    f = np.zeros((n, 16))
    f[:, 0], f[:, 1], f[:, 2], f[:, 3] = 1, total / k, indeg.min(1), indeg.max(1)
    f[:, 4], f[:, 5], f[:, 6], f[:, 7] = off.min(1), pi * n, sink, pair.sum(1) / (n - 1)
    f[:, 8] = total[t].sum(1) / k ** 2
    two = np.zeros(n)
    for a in range(k):
        np.add.at(two, t[:, a], total)
    f[:, 9] = two / k ** 2
    f[:, 10] = sum(indeg[t[:, a], a] > 1 for a in range(k)) / k
    f[:, 11], f[:, 12], f[:, 13] = np.log2(1 + total), rank, 64.0 / n
    f[:, 14] = sink & (indeg.max(1) > 1)
    f[:, 15] = sink[t].sum(1) / k
    for j in range(1, 16):
        if j != 13:
            sd = f[:, j].std()
            f[:, j] = (f[:, j] - f[:, j].mean()) / sd if sd > 1e-6 else 0.0
    return f


def _train_exact(case, seed):
    autos, _, dense, labels, groups, params = _train_inputs(case, seed)
    p = params.astype(np.float64)
    shapes = [(16, 64), (64,), (64, 128), (128,), (128, 128), (128,), (128,), (1,)]
    at = np.cumsum([0] + [math.prod(s) for s in shapes])
    m, v = np.zeros_like(p), np.zeros_like(p)
    order = list(range(len(autos)))
    g = splitmix64(1)
    for a in range(len(order), 1, -1):
        j = next(g) % a
        order[a - 1], order[j] = order[j], order[a - 1]
    losses = []
    for a in order:
        n, k, t = autos[a]
        f = _features(n, k, t)
        for o in range(0, case["count"], case["batch"]):
            phi, c, w1, b1, w2, b2, w3, b3 = [p[at[i]:at[i + 1]].reshape(s) for i, s in enumerate(shapes)]
            bits = dense[a][o:o + case["batch"]].astype(np.float64)
            want = labels[a][o:o + case["batch"]].astype(np.float64)
            rows = len(want)
            ep = f @ phi + c
            e = np.maximum(ep, 0)
            x = bits @ e
            p1 = x @ w1 + b1
            h1 = np.maximum(p1, 0)
            p2 = h1 @ w2 + b2
            h2 = np.maximum(p2, 0)
            y = h2 @ w3 + b3[0]
            loss = np.mean((y - want) ** 2)
            dy = 2 * (y - want) / rows
            if case["rank"]:
                grp = groups[a][o:o + case["batch"]]
                below = (grp[:, None] == grp[None, :]) & (want[:, None] < want[None, :])
                z = y[:, None] - y[None, :]
                loss += case["rank"] / rows * np.sum(np.logaddexp(0, z) * below)
                s = below / (1 + np.exp(-z))
                dy = dy + case["rank"] / rows * (s.sum(1) - s.sum(0))
            losses.append(loss)
            d2 = np.outer(dy, w3) * (p2 > 0)
            d1 = (d2 @ w2.T) * (p1 > 0)
            de = (bits.T @ (d1 @ w1.T)) * (ep > 0)
            grad = np.concatenate([x.ravel() for x in (f.T @ de, de.sum(0), x.T @ d1, d1.sum(0), h1.T @ d2, d2.sum(0),
                                                       h2.T @ dy, np.array([dy.sum()]))])
            step = len(losses)
            m = 0.9 * m + 0.1 * grad
            v = 0.999 * v + 0.001 * grad ** 2
            p = p - 1e-3 * (m / (1 - 0.9 ** step)) / (np.sqrt(v / (1 - 0.999 ** step)) + 1e-8)
    return {"params": p, "loss": float(np.mean(losses))}


def exact(case, seed):
    """Searches, subset checks and sorted sets are whole numbers; the trained parameters and the loss in 64 bits."""
    return _train_exact(case, seed) if case["kind"] == "train" else None
