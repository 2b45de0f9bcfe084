"""The learned beam when the model tells no sets apart: the kept sets are those
the order of equal scores names, in about the time of a model that does."""
import json
import time

import numpy as np
import pytest

import synchrowords_gb300 as sw
from synchrowords_gb300.generate import random_dfa
from test_gpu_learned_select import host_beam

pytestmark = pytest.mark.gpu


def plan(width, upper):
    return json.dumps({"upper_bound": upper, "algorithms": [
        {"name": "LearnedBeam", "config": {"beam_size": str(width), "order": "model"}}]})


@pytest.mark.parametrize("n,k,width,seed", [(40, 2, 1, 3), (64, 2, 127, 4), (65, 3, 129, 5), (130, 2, 1023, 6),
                                            (200, 2, 3000, 7), (150, 4, 4096, 9), (449, 2, 500, 10)])
def test_kept_sets_with_equal_scores(n, k, width, seed):
    equal = np.zeros(sw.MLP_PARAMS, dtype=np.float32)
    d = random_dfa(n, k, seed)
    with sw.Context(0, model=None) as c:
        c.set_model(equal)
        r = c.solve(d, n, k, plan(width, "2 * AUT_N"))
        assert r.upper == host_beam(c, equal, d, n, k, width, 2 * n)


def test_equal_scores_take_no_longer():
    if not sw.DEFAULT_MODEL.exists():
        pytest.skip("no packaged model")
    n, k = 150, 4
    d = random_dfa(n, k, 9)
    ms = []
    with sw.Context(0) as c:
        for params in (c.get_model(), np.zeros(sw.MLP_PARAMS, dtype=np.float32)):
            c.set_model(params)
            c.solve(d, n, k, plan(4096, "18"))  # shorter than either finds: the same 17 levels
            t = time.perf_counter()
            r = c.solve(d, n, k, plan(4096, "18"))
            ms.append(1e3 * (time.perf_counter() - t))
            assert r.upper == 18
    # one CTA: a level of 16 384 equal scores takes up to 16 more passes of ~10 us; ranked pair by pair it took 40 ms
    assert ms[1] < 5 * ms[0] + 1
