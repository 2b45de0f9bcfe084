"""The dominance checks on lists of their own, around the sizes at which their
chunks, the ordering of the rows and the check itself change, on both sides,
proper and not, with counts on the host and on the device, against a product of
the lists as matrices."""
import ctypes

import numpy as np
import pytest
import torch

import synchrowords_gb300 as sw
from test_gpu_near_permutations import near_permutations

pytestmark = pytest.mark.gpu


def pack(x):
    """0/1 matrix -> device rows: state q is bit 63 - q % 64 of word q / 64."""
    words = (x.shape[1] + 63) // 64
    b = np.packbits(np.pad(x, ((0, 0), (0, 64 * words - x.shape[1]))), axis=1, bitorder="big")
    return np.ascontiguousarray(b).view(">u8").astype(np.uint64)


def check(lib, c, n, forward, proper, S, Q, live=False, masked=False):
    s, q = pack(S if forward else 1 - S), pack(Q if forward else 1 - Q)
    flags, ms = np.zeros(len(q), dtype=np.uint32), ctypes.c_float()
    at = lambda a: a.ctypes.data_as(ctypes.c_void_p)
    assert lib.sw_testing_dominated(c._h, n, int(forward), int(proper), at(s), len(s), at(q), len(q), int(live),
                                    int(masked), at(flags), ctypes.byref(ms)) == 0
    return flags, ms.value


def reference(forward, proper, S, Q):
    """Which rows of Q hold a row of S (forward) or lie in one (a proper one)."""
    s, q = (torch.tensor(np.ascontiguousarray(x), device="cuda", dtype=torch.float16) for x in (S, Q))
    sizes_s, sizes_q = s.float().sum(1), q.float().sum(1)
    hit = torch.zeros(len(q), dtype=torch.bool, device="cuda")
    for i in range(0, len(s), 4096):
        part, sizes = s[i:i + 4096], sizes_s[i:i + 4096]
        common = q @ part.T  # whole numbers below 2048: exact in 16 bits
        inside = common == (sizes.half()[None, :] if forward else sizes_q.half()[:, None])
        if proper:
            inside &= sizes[None, :] != sizes_q[:, None]
        hit |= inside.any(1)
    return hit.cpu().numpy().astype(np.uint32)


def lists(rng, n, m, q, share):
    """m and q sets of about a tenth or two fifths of the states, a third of the second list made from the first."""
    S = (rng.random((m, n)) < rng.choice([0.05, 0.1, 0.2, 0.4], (m, 1))).astype(np.uint8)
    Q = (rng.random((q, n)) < rng.choice([0.05, 0.1, 0.2, 0.4], (q, 1))).astype(np.uint8)
    S[:, 0], Q[:, 1] = 1, 1  # no set is empty
    some = rng.choice(q, q // 3, replace=False)
    base = S[rng.integers(0, m, len(some))]
    Q[some] = base | (rng.random((len(some), n)) < 0.02) if share else base
    return S, Q


@pytest.mark.parametrize("n,m,q", [
    (40, 1, 1), (64, 33, 1024), (40, 1025, 700), (64, 900, 1025), (200, 8192, 3000), (200, 3000, 8193), (384, 8193, 500),
    (384, 500, 8193), (130, 32768, 2000), (130, 2000, 32769), (130, 32769, 2000), (60, 2500, 32769), (300, 40001, 3001),
    (300, 3001, 40001), (448, 9000, 9000), (449, 8191, 2000), (512, 8193, 4097), (512, 4097, 8193), (512, 33000, 1500),
    (512, 1500, 33000), (60, 3000, 65536), (130, 3000, 65536), (130, 3000, 65537)])
def test_flags(native_lib, n, m, q):
    rng = np.random.default_rng(n + m + q)
    with sw.Context(0) as c:
        for forward in (True, False):
            S, Q = lists(rng, n, m, q, True)
            if not forward:
                S, Q = 1 - S, 1 - Q
            for proper in (False, True):
                want = reference(forward, proper, S, Q)
                for live in (False, True):
                    assert (check(native_lib, c, n, forward, proper, S, Q, live)[0] == want).all()
    assert m == 1 or want.any() and not want.all()


@pytest.mark.parametrize("n", [130, 512])
@pytest.mark.parametrize("m", [1023, 8200, 40000])
def test_siblings(native_lib, n, m):
    rng = np.random.default_rng(m)
    S, Q = lists(rng, n, m // 2, m - m // 2, True)
    rows = np.unique(np.concatenate([S, Q]), axis=0)
    with sw.Context(0) as c:
        for forward in (True, False):
            R = rows if forward else 1 - rows
            assert (check(native_lib, c, n, forward, True, R, R)[0] == reference(forward, True, R, R)).all()


def test_large_forward_lists_take_the_faster_check(native_lib):
    n, k = 42, 3
    d = np.array(near_permutations(n, k, 2)).reshape(n, k)
    layer = np.ones((1, n), dtype=np.uint8)
    while len(layer) < 200_000:
        images = np.zeros((k * len(layer), n), dtype=np.uint8)
        for a in range(k):
            for q in range(n):
                images[a * len(layer):(a + 1) * len(layer), d[q, a]] |= layer[:, q]
        layer = np.unique(images, axis=0)[::-1]
    layer = np.ascontiguousarray(layer[:300_000])
    with sw.Context(0) as c:
        sliced_or_masked = check(native_lib, c, n, True, True, layer, layer)[1]
        masked = check(native_lib, c, n, True, True, layer, layer, masked=True)[1]
    assert sliced_or_masked < 1.3 * masked
