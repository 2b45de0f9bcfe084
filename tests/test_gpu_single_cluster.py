"""A solve's first levels on one thread-block cluster and their hand-over to
the streamed search: searches that end on the cluster, that leave it for each
reason (work limit, length limit, memory budget), at every set width, against
the same search without it (a plan with "reductions": "always" never starts
there) and against known lengths."""
import json

import pytest

import oracle
from synchrowords_gb300.generate import cerny, random_dfa

pytestmark = pytest.mark.gpu


def plan(**exact):
    return json.dumps({"algorithms": [{"name": "Exact", "config": exact}]})


@pytest.mark.parametrize("n", [2, 3, 12, 33, 34])
def test_deep_searches(ctx, n):
    # C_33 resets at the launch's length limit (1024), C_34 one merge past it
    r = ctx.solve(cerny(n), n, 2, plan())
    assert (r.lower, r.upper) == ((n - 1) ** 2,) * 2
    assert len(oracle.apply_word(cerny(n), n, 2, r.word)) == 1
    assert r.stats["bfs_steps"] + r.stats["ibfs_steps"] == (n - 1) ** 2


@pytest.mark.parametrize("n,k", [(1, 2), (5, 1), (63, 2), (64, 3), (65, 2), (128, 2), (129, 3), (150, 2), (192, 2), (193, 2),
                                 (256, 2), (256, 16), (40, 16)])
def test_same_lengths_without_the_cluster(ctx, n, k):
    for seed in range(3):
        d = random_dfa(n, k, 7000 + 31 * n + seed)
        r, s = ctx.solve(d, n, k, plan()), ctx.solve(d, n, k, plan(reductions="always"))
        assert (r.non_synchro, r.lower, r.upper) == (s.non_synchro, s.lower, s.upper)
        if n == 1:
            assert r.upper == 0  # the plan's bound n^3 / 6 is zero: nothing is searched
        elif not r.non_synchro and r.lower == r.upper:  # else both stopped at the plan's memory budget
            assert len(r.word) == r.upper and len(oracle.apply_word(d, n, k, r.word)) == 1


@pytest.mark.parametrize("mb", [1, 2, 4])
def test_memory_budget_decides_as_without_the_cluster(ctx, mb):
    # the levels that pass a quarter of the budget bring the reductions on; past it the search ends with a lower bound
    for seed in range(3):
        d = random_dfa(120, 2, 7700 + seed)
        full = ctx.solve(d, 120, 2, plan())
        for dfs in (True, False):
            r = ctx.solve(d, 120, 2, plan(max_memory_mb=mb, dfs=dfs))
            assert r.lower <= full.lower <= r.upper
            if r.lower == r.upper:
                assert r.upper == full.upper
