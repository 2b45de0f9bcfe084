"""Automata whose letters are permutations but for one state: layers of sets of
few sizes, most of whose children are duplicates."""
import json
import random
import time

import pytest

import oracle
import synchrowords_gb300 as sw
from synchrowords_gb300.generate import random_dfa

pytestmark = pytest.mark.gpu


def near_permutations(n, k, seed):
    g = random.Random(seed)
    d = [0] * (n * k)
    for a in range(k):
        p = list(range(n))
        g.shuffle(p)
        d[a::k] = p
    d[0] = d[k * (n - 1)]
    return d


def seconds(call, runs=4):
    best = 1e9
    for _ in range(runs):
        t = time.perf_counter()
        call()
        best = min(best, time.perf_counter() - t)
    return best


@pytest.mark.parametrize("n,k,seed", [(60, 16, 2), (40, 8, 3)])
def test_reduced_levels_without_their_count(n, k, seed):
    d = near_permutations(n, k, seed)
    plan = json.dumps({"algorithms": [{"name": "Exact", "config": {"reductions": "always", "dfs": False,
                                                                   "max_memory_mb": 40}}]})
    with sw.Context(0) as c:
        plain = c.solve(d, n, k, plan)

        def counted():  # under the profiler every level's count is read back before its checks
            c.profile_begin()
            r = c.solve(d, n, k, plan)
            c.profile_end()
            assert (r.lower, r.upper) == (plain.lower, plain.upper)

        assert seconds(lambda: c.solve(d, n, k, plan)) < 1.25 * seconds(counted) + 1e-3


def beam_plan(beam, upper):
    return json.dumps({"upper_bound": str(upper), "algorithms": [
        {"name": "Beam", "config": {"presort": "indeg", "beam_size": str(beam)}}]})


# one set to the largest beam of one launch; the layers whose bins hold too many to be compared in pairs among them
@pytest.mark.parametrize("n,k,beam", [(20, 2, 1), (33, 2, 130), (60, 16, 500), (64, 2, 4000), (65, 3, 257), (128, 2, 896),
                                      (200, 2, 1528), (300, 2, 500), (400, 2, 300), (512, 3, 150)])
def test_beam_matches_oracle(ctx, n, k, beam):
    d, upper = near_permutations(n, k, n + beam), 60
    r = ctx.solve(d, n, k, beam_plan(beam, upper))
    b = oracle.beam(d, n, k, oracle.BeamParams(beam_size=beam, presort_indeg=True), upper=upper)
    assert r.upper == b.upper
    if b.upper < upper:
        assert len(r.word) == r.upper and len(oracle.apply_word(d, n, k, r.word)) == 1


def test_beam_words(ctx):
    for n, k, beam in ((12, 2, 300), (14, 3, 400), (16, 4, 500), (24, 8, 800), (40, 16, 1000)):  # all reset within the bound
        d = near_permutations(n, k, n)
        r = ctx.solve(d, n, k, beam_plan(beam, n * n))
        b = oracle.beam(d, n, k, oracle.BeamParams(beam_size=beam, presort_indeg=True), upper=n * n)
        assert r.upper == b.upper < n * n
        assert len(r.word) == r.upper and len(oracle.apply_word(d, n, k, r.word)) == 1


def test_beam_levels_of_similar_sets(ctx):
    # ranked in pairs within its bins a level took 50 times as long as a random automaton's
    n, k, beam = 128, 2, 3000
    plan = beam_plan(beam, 25)
    times = [seconds(lambda: ctx.solve(d, n, k, plan)) for d in (random_dfa(n, k, 7), near_permutations(n, k, 5))]
    assert times[1] < 6 * times[0]
