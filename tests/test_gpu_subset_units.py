"""How a subset check is cut into units: whole super-tiles, parts of them, and
listed (32 queries, super-tile) pairs, on lists at the edges of each, against
every pair tested on the CPU."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def draw(rng, n, count, density):
    words = (n + 63) // 64
    bits = rng.random((count, 64 * words)) < density
    bits[:, n:] = False
    return np.packbits(bits, axis=1, bitorder="little").view(np.uint64)


def brute(sets, checks, proper):
    out = np.zeros(len(checks), bool)
    for a in range(0, len(sets), 1 << 16):
        part = sets[a:a + (1 << 16)]
        for i, c in enumerate(checks):
            if out[i]:
                continue
            inside = ~(part & ~c).any(axis=1)
            if proper:
                inside &= (part != c).any(axis=1)
            out[i] = inside.any()
    return out


# super-tiles of 1024 rows: 1 unit; ragged; 2^14 pairs (16 super-tiles x 1024
# groups is the last unlisted size) and one past; more than 1024 super-tiles
@pytest.mark.parametrize("n,sets,checks", [(200, 1, 1), (200, 1023, 33), (64, 1025, 31), (130, 4097, 65),
                                           (40, 16384, 32768), (40, 16385, 32768), (200, 33000, 17000),
                                           (48, 1050000, 520), (300, 20000, 30000)])
@pytest.mark.parametrize("proper", [False, True])
def test_units(ctx, n, sets, checks, proper):
    rng = np.random.default_rng(n + sets + checks)
    S = draw(rng, n, sets, 0.3 if n > 60 else 0.4)
    Q = draw(rng, n, checks, 0.9)
    Q[::7] = S[rng.integers(0, sets, len(Q[::7]))]           # equal to a set
    Q[3::7] = S[rng.integers(0, sets, len(Q[3::7]))] | draw(rng, n, len(Q[3::7]), 0.05)  # around one
    sample = rng.permutation(checks)[:400]
    got = np.asarray(ctx.subsets_check(n, S, Q, proper=proper)).astype(bool)
    assert (got[sample] == brute(S, Q[sample], proper)).all()
