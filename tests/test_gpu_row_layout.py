"""Conversion between the reference bit layout and device rows, on the device:
bits of states >= n in a caller's rows take no part, at every position a row
can end in its last word."""
import numpy as np
import pytest

from bitsets import from_rows, image, preimage, random_sets, to_rows
from synchrowords_gb300.generate import random_dfa

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 63, 64, 65, 150, 511, 512])
@pytest.mark.parametrize("count", [1, 255, 5000])
def test_bits_past_the_last_state_are_ignored(ctx, n, count):
    rng = np.random.default_rng(n + count)
    delta = random_dfa(n, 2, 5 * n + count)
    sets = random_sets(rng, n, count, 0.3)
    rows = to_rows(sets, n)
    dirty = rows.copy()
    if n % 64:
        dirty[:, -1] |= np.uint64(((1 << 64) - 1) ^ ((1 << (n % 64)) - 1))
    for inverse, fn in ((False, lambda s: image(delta, 2, 1, s)), (True, lambda s: preimage(delta, n, 2, 1, s))):
        got = ctx.apply_transition(delta, n, 2, 1, inverse, dirty)
        assert (got == ctx.apply_transition(delta, n, 2, 1, inverse, rows)).all()
        assert from_rows(got[:50], n) == [fn(s) for s in sets[:50]]
    assert (ctx.sort_unique(n, dirty) == ctx.sort_unique(n, rows)).all()
