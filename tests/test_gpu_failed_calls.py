"""Calls that end for want of device memory leave their context usable: the
next calls on it give what a fresh context gives."""
import ctypes
import json

import numpy as np
import pytest

import synchrowords_gb300 as sw
from synchrowords_gb300.generate import random_dfa

pytestmark = pytest.mark.gpu


@pytest.fixture
def fail_growth(native_lib):
    """fail_growth(s): after s more growths of a device buffer, one fails."""
    yield native_lib.sw_testing_fail_growth
    native_lib.sw_testing_fail_growth(-1)


def test_error_stays_with_its_call(fail_growth):
    sets = np.array([[5], [3], [5], [9]], dtype=np.uint64)
    with sw.Context(0) as c:
        fail_growth(0)
        with pytest.raises(sw.SynchroError):
            c.sort_unique(40, sets)
        assert len(c.sort_unique(40, sets)) == 3


def plan(*algorithms, **top):
    return json.dumps({**top, "algorithms": [{"name": name, "config": config} for name, config in algorithms]})


PLANS = {
    "plain": plan(("Exact", {})),
    "always": plan(("Exact", {"reductions": "always"})),
    "reduce": plan(("Eppstein", {}), ("Beam", {"presort": "indeg", "beam_size": "10"}),
                   ("Reduce", {"min_n": "40", "list_size_threshold": "AUT_N * 16"}), ("Exact", {})),
    # the bounded phase, in chunks
    "bounded": plan(("Beam", {"presort": "indeg", "beam_size": "AUT_N * 4"}),
                    ("Exact", {"max_memory_mb": "4", "dfs_min_list_size": "512"})),
}


def answers(results):
    return [(r.non_synchro, r.lower, r.upper, r.word is not None) for r in results]


# at n = 200 the lists pass 2^16 children and the size where the dominance checks order them
@pytest.mark.parametrize("name,n,k,seed", [("plain", 200, 2, 12), ("always", 65, 3, 1), ("always", 200, 2, 12),
                                           ("reduce", 100, 3, 4), ("bounded", 120, 2, 7700)])
def test_solves_after_a_failed_growth(fail_growth, name, n, k, seed):
    big, small = random_dfa(n, k, seed), random_dfa(70, 2, 5)
    with sw.Context(0) as c:
        want = answers([c.solve(big, n, k, PLANS[name]), c.solve(small, 70, 2, PLANS["always"])])
    failed = 0
    for successes in range(500):
        with sw.Context(0) as c:
            fail_growth(successes)
            try:
                c.solve(big, n, k, PLANS[name])
            except sw.SynchroError:
                failed += 1
            else:
                break
            finally:
                fail_growth(-1)
            assert answers([c.solve(small, 70, 2, PLANS["always"])]) == want[1:]
            assert answers([c.solve(big, n, k, PLANS[name]), c.solve(small, 70, 2, PLANS["always"])]) == want
    assert 10 < failed < 500


def test_batches_after_a_failed_growth(fail_growth):
    automata = [(n, 2, random_dfa(n, 2, 300 + n)) for n in (40, 70, 101, 130, 170, 190, 200)]
    with sw.Context(0) as c:
        want = answers(c.solve_batch(automata, PLANS["plain"]))
    failed = 0
    for successes in range(0, 400, 3):
        with sw.Context(0) as c:
            fail_growth(successes)
            try:
                c.solve_batch(automata, PLANS["plain"])
            except sw.SynchroError:
                failed += 1
            else:
                break
            finally:
                fail_growth(-1)
            assert answers(c.solve_batch(automata, PLANS["plain"])) == want
    assert 3 < failed < 130


@pytest.mark.parametrize("name", ["plain", "reduce"])
def test_later_calls_leave_the_record_of_a_failed_one(native_lib, fail_growth, name):
    n, k = 100, 3
    d = np.array(random_dfa(n, k, 4), dtype=np.uint32)
    sets = np.arange(1, 200, dtype=np.uint64).reshape(-1, 1)
    with sw.Context(0) as c:
        record = sw._Result()
        fail_growth(5)
        assert native_lib.sw_solve_json(c._h, d.ctypes.data_as(sw._U32P), n, k, PLANS[name].encode(),
                                        ctypes.byref(record)) != 0
        fail_growth(-1)
        before = bytes(record)
        c.subsets_check(60, sets, sets)
        assert bytes(record) == before


@pytest.mark.parametrize("what", ["forward", "gradient"])
def test_scores_after_a_failed_growth(fail_growth, what):
    rng = np.random.default_rng(2)
    small, big = (40, 2, random_dfa(40, 2, 1)), (300, 2, random_dfa(300, 2, 2))
    params = rng.normal(0, 0.1, sw.MLP_PARAMS).astype(np.float32)
    labels = rng.normal(10, 3, 300).astype(np.float32)

    def call(c, automaton):
        n, k, d = automaton
        sets = np.packbits(np.random.default_rng(n).random((300, 512)) < 0.2, axis=1, bitorder="little").view(np.uint64)
        if what == "forward":
            return c.mlp_forward(params, d, n, k, sets)
        return c.mlp_gradient(params, d, n, k, sets, labels)[0]

    with sw.Context(0) as c:
        want = [call(c, small), call(c, big)]
    failed = 0
    for successes in range(200):
        with sw.Context(0) as c:
            call(c, small)
            fail_growth(successes)
            try:
                call(c, big)
            except sw.SynchroError:
                failed += 1
            else:
                break
            finally:
                fail_growth(-1)
            for automaton, w in zip((small, big), want):
                np.testing.assert_allclose(call(c, automaton), w, rtol=1e-4, atol=1e-4 * np.abs(w).max())
    assert 3 < failed < 200


def test_learned_plans_after_a_failed_growth(fail_growth):
    learned = plan(("LearnedBeam", {"beam_size": "1024", "order": "model"}), ("Exact", {}), upper_bound="4 * AUT_N")
    n, d = 130, random_dfa(130, 2, 6)
    with sw.Context(0) as c:
        want = answers([c.solve(d, n, 2, learned)])
    failed = 0
    for successes in range(300):
        with sw.Context(0) as c:
            fail_growth(successes)
            try:
                c.solve(d, n, 2, learned)
            except sw.SynchroError:
                failed += 1
            else:
                break
            finally:
                fail_growth(-1)
            assert answers([c.solve(d, n, 2, learned)]) == want
    assert 10 < failed < 300


@pytest.mark.parametrize("what", ["forward", "beam"])
def test_a_scoring_wait_that_ran_out_is_reported(native_lib, what):
    n, d = 130, random_dfa(130, 2, 6)
    rows = np.packbits(np.random.default_rng(1).random((100, 512)) < 0.1, axis=1, bitorder="little").view(np.uint64)
    learned = plan(("LearnedBeam", {"beam_size": "256", "order": "model"}), upper_bound="4 * AUT_N")

    def call(c):
        return c.mlp_forward(c.get_model(), d, n, 2, rows).tolist() if what == "forward" else c.solve(d, n, 2, learned).upper

    with sw.Context(0) as c:
        want = call(c)
        assert native_lib.sw_testing_plant_error(c._h, 4) == 0  # what the kernel stores (mlp::kErrorWait)
        with pytest.raises(sw.SynchroError, match="tensor-core wait"):
            call(c)
        assert call(c) == want
