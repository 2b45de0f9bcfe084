"""Reduce's list stays on the device: relabelling across row widths and the
word traced through it, against the oracle and the automaton itself."""
import json

import pytest

import oracle
from synchrowords_gb300.generate import random_dfa

pytestmark = pytest.mark.gpu


def lifted(core, n, k, seed):
    """A random automaton of `core` states under n - core states that lead into it."""
    d = random_dfa(core, k, seed)
    s = seed
    for q in range(core, n):
        for _ in range(k):
            s = (s * 6364136223846793005 + 1442695040888963407) % (1 << 64)
            d.append((s >> 33) % (core if q % 3 else q))
    perm = sorted(range(n), key=lambda q: (q * 7919 + seed) % n)
    out = [0] * (n * k)
    for q in range(n):
        for a in range(k):
            out[perm[q] * k + a] = perm[d[q * k + a]]
    return out


# original and reduced widths in words: 1-1, 2-1, 2-1 (63..65 states kept), 3-2, 5-1, 8-2
@pytest.mark.parametrize("core,n,k", [(30, 64, 2), (40, 65, 2), (63, 128, 2), (64, 128, 2), (65, 129, 2), (50, 320, 3),
                                      (100, 512, 2)])
@pytest.mark.parametrize("threshold", [0, 1, 40, 2000])
def test_reduced_search(ctx, core, n, k, threshold):
    d = lifted(core, n, k, 3 * n + core)
    plan = json.dumps({"upper_bound": "AUT_N * AUT_N", "algorithms": [
        {"name": "Reduce", "config": {"min_n": "2", "list_size_threshold": str(threshold)}},
        {"name": "Exact", "config": {}}]})
    r = ctx.solve(d, n, k, plan)
    ex = oracle.exact(d, n, k, upper=n * n)
    assert (r.non_synchro, r.lower, r.upper) == (ex.non_synchro, ex.lower, ex.upper)
    assert len(r.word) == r.upper and len(oracle.apply_word(d, n, k, r.word)) == 1
