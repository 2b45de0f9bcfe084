"""The learned beam's kept sets against a beam run on the host with the same
scores: one to all of a layer's children kept, and on both sides of the largest
layer that is selected from rather than sorted."""
import json

import numpy as np
import pytest

import oracle
import synchrowords_gb300 as sw
from synchrowords_gb300.generate import random_dfa

pytestmark = pytest.mark.gpu


def pack(sets, n):
    return np.packbits(np.pad(sets, ((0, 0), (0, 512 - n))), axis=1, bitorder="little").view(np.uint64)


def tie_order(sets, n):
    """Order of equal scores: the first 64 states as a number (state 0 highest),
    then a 32-bit mix of the rest."""
    words = (n + 63) // 64
    rows = np.packbits(np.pad(sets, ((0, 0), (0, 64 * words - n))), axis=1, bitorder="big").view(">u8").astype(np.uint64)
    h = np.full(len(rows), 0x9E3779B97F4A7C15, np.uint64)
    for w in range(1, words):
        x = rows[:, w] ^ (h + np.uint64(0x632BE59BD9B4E019 * (w + 1) % 2**64))
        x ^= x >> np.uint64(31)
        x *= np.uint64(0x94D049BB133111EB)
        x ^= x >> np.uint64(29)
        h = (h ^ x) * np.uint64(0xBF58476D1CE4E5B9)
    mix = (h ^ (h >> np.uint64(32))) & np.uint64(0xFFFFFFFF)
    return rows[:, 0], mix if words > 1 else np.zeros(len(rows), np.uint64)


def host_beam(ctx, params, d, n, k, width, upper):
    """Length at which the beam first holds a singleton, or upper."""
    delta = np.asarray(d).reshape(n, k)
    layer = np.ones((1, n), bool)
    for length in range(1, upper):
        children = np.zeros((k * len(layer), n), bool)
        for a in range(k):
            rows, states = np.nonzero(layer)
            children[a * len(layer) + rows, delta[states, a]] = True
        children = np.unique(children, axis=0)
        if (children.sum(axis=1) == 1).any():
            return length
        if len(children) > width:
            score = np.asarray(ctx.mlp_forward(params, d, n, k, pack(children, n)), dtype=np.float32)
            first, mix = tie_order(children, n)
            children = children[np.lexsort((mix, first, score))[:width]]
        layer = children
    return upper


@pytest.mark.parametrize("n,k,width,seed", [(40, 2, 1, 3), (64, 2, 33, 4), (65, 3, 100, 5), (130, 2, 1023, 6),
                                            (200, 2, 1025, 7), (256, 2, 4096, 8), (150, 4, 4096, 9),
                                            (150, 4, 4097, 9)])  # 16384 children, and more
def test_kept_sets(n, k, width, seed):
    if not sw.DEFAULT_MODEL.exists():
        pytest.skip("no packaged model")
    ctx = sw.Context(0)
    d = random_dfa(n, k, seed)
    plan = json.dumps({"upper_bound": "2 * AUT_N", "algorithms": [
        {"name": "LearnedBeam", "config": {"beam_size": str(width), "order": "model"}}]})
    r = ctx.solve(d, n, k, plan)
    assert r.upper == host_beam(ctx, ctx.get_model(), d, n, k, width, 2 * n)
    if r.upper < 2 * n:
        assert len(r.word) == r.upper and len(oracle.apply_word(d, n, k, r.word)) == 1
    ctx.close()
