"""Beam in one launch: bounds and words against the oracle's beam, from a beam
of one set to the largest that fits, over several launches' worth of levels,
and one size past it."""
import json

import pytest

import oracle
from synchrowords_gb300.generate import cerny, random_dfa

pytestmark = pytest.mark.gpu


def plan(**cfg):
    return json.dumps({"upper_bound": "AUT_N * AUT_N", "algorithms": [
        {"name": "Beam", "config": {key: str(v) for key, v in cfg.items()}}]})


CASES = [("random", 5, 2, 1), ("random", 33, 2, 31), ("random", 64, 2, 32), ("random", 65, 3, 33),
         ("random", 100, 3, 10), ("random", 129, 2, 1000), ("random", 200, 2, 1528), ("random", 255, 2, 2040),
         ("random", 300, 2, 100), ("random", 512, 2, 64), ("random", 64, 2, 4000),
         ("random", 300, 2, 2468),  # past the capacity: the launches over the whole GPU
         ("cerny", 18, 2, 3), ("cerny", 26, 2, 7)]  # 289 and 625 levels: over one launch's


@pytest.mark.parametrize("kind,n,k,beam", CASES)
@pytest.mark.parametrize("presort", ["indeg", "none"])
def test_beam_matches_oracle(ctx, kind, n, k, beam, presort):
    d = cerny(n) if kind == "cerny" else random_dfa(n, k, 7 * n + beam)
    r = ctx.solve(d, n, k, plan(presort=presort, beam_size=beam))
    b = oracle.beam(d, n, k, oracle.BeamParams(beam_size=beam, presort_indeg=presort == "indeg"), upper=n * n)
    assert r.upper == b.upper
    if b.upper < n * n:
        assert len(r.word) == r.upper and len(oracle.apply_word(d, n, k, r.word)) == 1


@pytest.mark.parametrize("max_iter", [0, 1, 255, 256, 257, 600])
def test_beam_stops_at_max_iter(ctx, max_iter):
    n, k, beam = 26, 2, 5
    d = cerny(n)
    r = ctx.solve(d, n, k, plan(beam_size=beam, max_iter=max_iter))
    b = oracle.beam(d, n, k, oracle.BeamParams(beam_size=beam, max_iter=max_iter), upper=n * n)
    assert r.upper == b.upper
