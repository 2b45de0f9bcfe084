"""Dominance reductions through Reduce and distance pairs, whose layers are
pruned in full: labels and layer sizes at widths and alphabets around the
kernel's chunk (1024, 4096 rows) and word edges, against a plain search."""
import numpy as np
import pytest

from synchrowords_gb300.generate import random_dfa

pytestmark = pytest.mark.gpu


def maximal_layers(d, n, k, depth, forward):
    """Layer sizes of the pruned search: children that hold (forward: are held
    by, backward) an earlier kept set or a sibling are dropped."""
    full = (1 << n) - 1
    ind = [[sum(1 for p in range(n) if d[p * k + a] == q) for a in range(k)] for q in range(n)]

    def step(s, a):
        if forward:
            r = 0
            for q in range(n):
                if s >> q & 1:
                    r |= 1 << d[q * k + a]
            return r
        return sum(1 << q for q in range(n) if s >> d[q * k + a] & 1)

    inside = (lambda a, b: a & ~b == 0) if forward else (lambda a, b: b & ~a == 0)  # a dominates b
    # the states of the one component nothing leaves
    reach = {0}
    todo = [0]
    while todo:
        q = todo.pop()
        for a in range(k):
            p = d[q * k + a]
            if p not in reach:
                reach.add(p)
                todo.append(p)
    sink = reach
    for q in sorted(reach):
        r, t = {q}, [q]
        while t:
            u = t.pop()
            for a in range(k):
                p = d[u * k + a]
                if p not in r:
                    r.add(p)
                    t.append(p)
        if len(r) < len(sink):
            sink = r
    layer = [full] if forward else [1 << q for q in sorted(sink) if max(ind[q]) > 1]
    seen = list(layer)
    out = []
    for _ in range(depth):
        kids = sorted({step(s, a) for s in layer for a in range(k)})
        kids = [c for c in kids if not any(inside(v, c) for v in seen)]
        layer = [c for c in kids if not any(o != c and inside(o, c) for o in kids)]
        seen += layer
        out.append(len(layer))
    return out


@pytest.mark.parametrize("n,k", [(20, 2), (33, 3), (64, 2), (65, 3), (130, 2), (200, 2), (257, 2), (390, 2), (449, 2), (512, 2)])
def test_pruned_layer_sizes(ctx, n, k):
    import json
    import synchrowords_gb300 as sw
    d = random_dfa(n, k, 900 + n)
    # a search cut off by its bound after `depth` levels reports what it kept
    depth = 9 if k == 3 else 12
    plan = json.dumps({"upper_bound": str(depth), "algorithms": [{"name": "Exact", "config": {"reductions": "always"}}]})
    with sw.Context(0) as c:
        r = c.solve(d, n, k, plan)
    if r.non_synchro or r.stats["bfs_steps"] + r.stats["ibfs_steps"] < depth:
        pytest.skip("no search of the full depth")
    f = maximal_layers(d, n, k, r.stats["bfs_steps"], True)
    b = maximal_layers(d, n, k, r.stats["ibfs_steps"], False)
    assert r.stats["subsets_kept"] == sum(f) + sum(b)


@pytest.mark.parametrize("n", [100, 170])
def test_reductions_do_not_change_lengths(ctx, n):
    import json
    always = json.dumps({"algorithms": [{"name": "Exact", "config": {"reductions": "always"}}]})
    plain = json.dumps({"algorithms": [{"name": "Exact", "config": {}}]})
    for seed in range(4):
        d = random_dfa(n, 2, 40 + seed)
        a, p = ctx.solve(d, n, 2, always), ctx.solve(d, n, 2, plain)
        assert (a.non_synchro, a.lower, a.upper) == (p.non_synchro, p.lower, p.upper)
