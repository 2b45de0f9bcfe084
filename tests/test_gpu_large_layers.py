"""Layers of millions of sets: their buckets are as fine as the checks need, and
the answers those of another route."""
import json

import pytest

import oracle
import synchrowords_gb300 as sw
from synchrowords_gb300.generate import random_dfa

pytestmark = pytest.mark.gpu
PLAIN = json.dumps({"algorithms": [{"name": "Exact", "config": {"max_memory_mb": 40000}}]})
BEAM = json.dumps({"upper_bound": "AUT_N", "algorithms": [
    {"name": "Beam", "config": {"presort": "indeg", "beam_size": "20000"}},
    {"name": "Exact", "config": {"max_memory_mb": 40000, "reductions": "always"}}]})


@pytest.mark.parametrize("n,k,seed", [(280, 2, 22), (280, 2, 23), (320, 2, 1)])  # up to 2^22 children and past it
def test_lengths_and_rows_tested(n, k, seed):
    d = random_dfa(n, k, seed)
    with sw.Context(0) as c:
        c.solve(d, n, k, PLAIN)
        c.profile_begin()
        r = c.solve(d, n, k, PLAIN)
        subset_query = c.profile_end()["subset_query"]
        other = c.solve(d, n, k, BEAM)
    assert (r.lower, r.upper) == (other.lower, other.upper) and r.lower == r.upper
    assert len(r.word) == r.upper and len(oracle.apply_word(d, n, k, r.word)) == 1
    # bytes of rows read a pair asked about: 0.0006 to 0.0015; with 2^16 buckets 0.0013 to 0.0048
    assert subset_query["bytes"] < (0.0009 if n == 320 else 0.0025) * r.stats["logical_pairs"]
