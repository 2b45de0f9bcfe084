"""Batches of automata whose levels one CTA takes: sizes on both sides of that
launch's limit, alone and among larger ones, searches past its regions, and
hundreds of levels."""
import json

import pytest

import oracle
import synchrowords_gb300 as sw
from synchrowords_gb300.generate import cerny, random_dfa

pytestmark = pytest.mark.gpu
PLAIN = json.dumps({"algorithms": [{"name": "Exact", "config": {}}]})


def synchronizes(n, k, d):
    merged = {(q, q) for q in range(n)}
    while True:
        more = {(p, q) for p in range(n) for q in range(n) for a in range(k) if (d[p * k + a], d[q * k + a]) in merged}
        if more <= merged:
            return len(merged) == n * n
        merged |= more


def check(c, automata):
    for (n, k, d), r in zip(automata, c.solve_batch(automata, PLAIN)):
        assert r.non_synchro == (n < 20 and not synchronizes(n, k, d)) or n >= 20
        if r.non_synchro:
            continue
        ref = oracle.exact(d, n, k)
        assert (r.lower, r.upper) == (ref.lower, ref.upper), (n, k)
        if r.word is not None:
            assert len(r.word) == r.upper and len(oracle.apply_word(d, n, k, r.word)) == 1


@pytest.mark.parametrize("sizes", [[(2, 2), (3, 2), (5, 3)], [(31, 2), (20, 3), (15, 4)], [(32, 2)], [(16, 4)], [(16, 2), (32, 2)],
                                   [(10, 2), (70, 2), (130, 2)], [(10, 2)] * 3 + [(60, 2)] * 2])
def test_sizes(sizes):
    automata = [(n, k, random_dfa(n, k, 50 * s + n)) for s in range(8) for n, k in sizes]
    with sw.Context(0) as c:
        check(c, automata)
        check(c, automata[::2])
        check(c, automata)


def test_deep_and_many():
    with sw.Context(0) as c:
        check(c, [(n, 2, cerny(n)) for n in range(2, 32)])
        check(c, [(8, 2, random_dfa(8, 2, s)) for s in range(400)])
        check(c, [(n, 2, cerny(n)) for n in range(20, 40)])


def test_launch_time():
    # a launch of four CTAs each spent 2.6 ms on these, one of one CTA 0.7
    with sw.Context(0) as c:
        automata = [(10, 2, random_dfa(10, 2, s)) for s in range(2000)]
        ms = []
        for _ in range(4):
            c.solve_batch(automata, PLAIN)
            ms.append(c.last_batch_profile()["device_ms"])
        assert min(ms) < 1.5
