"""Automata without a reset word: found out by the host while the search runs, in
about the time that takes."""
import json

import pytest

from synchrowords_gb300.generate import random_dfa
from test_gpu_near_permutations import seconds

pytestmark = pytest.mark.gpu
PLAIN = json.dumps({"algorithms": [{"name": "Exact", "config": {}}]})


def rotation(n, d):
    """q -> q + 1 and 0 -> d: no reset word when d divides n (d > 1)."""
    t = [0] * (2 * n)
    for q in range(n):
        t[2 * q], t[2 * q + 1] = (q + 1) % n, q
    t[1] = d
    return t


@pytest.mark.parametrize("n,d", [(4, 2), (9, 3), (28, 2), (64, 2), (128, 2), (200, 2), (256, 2)])
def test_rotations(ctx, n, d):
    r = ctx.solve(rotation(n, d), n, 2, PLAIN)
    assert r.non_synchro
    # searched to its end it takes hundreds of levels, 2 to 7 ms; the host's check takes 0.02 to 0.3
    assert seconds(lambda: ctx.solve(rotation(n, d), n, 2, PLAIN)) < 1e-3


def test_between_others(ctx):
    automata = [(28, 2, rotation(28, 2)), (48, 2, random_dfa(48, 2, 1)), (64, 2, rotation(64, 2)), (27, 2, rotation(27, 2)),
                (100, 2, random_dfa(100, 2, 3))]
    first = [ctx.solve(d, n, k, PLAIN) for n, k, d in automata]
    again = [ctx.solve(d, n, k, PLAIN) for n, k, d in automata] + list(ctx.solve_batch(automata, PLAIN))
    assert [r.non_synchro for r in first] == [True, False, True, False, False]
    for r, f in zip(again, 2 * first):
        assert (r.non_synchro, r.non_synchro or (r.lower, r.upper)) == (f.non_synchro, f.non_synchro or (f.lower, f.upper))
