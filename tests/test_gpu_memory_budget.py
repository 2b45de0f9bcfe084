"""Device memory of a search against its max_memory_mb."""
import ctypes
import json

import pytest

import synchrowords_gb300 as sw
from synchrowords_gb300.generate import random_dfa

pytestmark = pytest.mark.gpu

USED, USED_HIGH = 7, 8  # CU_MEMPOOL_ATTR_USED_MEM_CURRENT, _HIGH


class Pool:
    """The device's default memory pool, from which a solve takes its buffers."""

    def __init__(self):
        self.lib, self.pool, device = ctypes.CDLL("libcuda.so.1"), ctypes.c_void_p(), ctypes.c_int()
        assert self.lib.cuDeviceGet(ctypes.byref(device), 0) == 0
        assert self.lib.cuDeviceGetDefaultMemPool(ctypes.byref(self.pool), device) == 0

    def get(self, attribute):
        v = ctypes.c_uint64()
        assert self.lib.cuMemPoolGetAttribute(self.pool, attribute, ctypes.byref(v)) == 0
        return v.value

    def peak(self, call):
        """Bytes at the peak of the call beyond those held before it."""
        zero = ctypes.c_uint64(0)
        before = self.get(USED)
        assert self.lib.cuMemPoolSetAttribute(self.pool, USED_HIGH, ctypes.byref(zero)) == 0
        call()
        return self.get(USED_HIGH) - before


# The budget counts each visited row and each child's three copies.  Lists take
# a quarter more than their rows, twice (a visited list and the one it is merged
# into), children at most as much; hashed lists with their tables stay within
# the budget.  Beside that the first levels' cluster, the subset check's list
# and its masks take up to 100 MB.
@pytest.mark.parametrize("mb", [100, 300, 1000])
@pytest.mark.parametrize("reductions", ["always", "memory"])
@pytest.mark.parametrize("beam", [False, True])
def test_peak(mb, reductions, beam):
    d, algorithms = random_dfa(300, 2, 5), [{"name": "Exact", "config": {
        "max_memory_mb": mb, "reductions": reductions, "dfs": beam, "dfs_min_list_size": "8192"}}]
    if beam:
        algorithms.insert(0, {"name": "Beam", "config": {"presort": "indeg", "beam_size": "AUT_N * 4"}})
    with sw.Context(0) as c:
        c.solve(random_dfa(60, 2, 1), 60, 2, json.dumps({"algorithms": algorithms[-1:]}))
        peak = Pool().peak(lambda: c.solve(d, 300, 2, json.dumps({"algorithms": algorithms})))
    assert peak < (2.5 * mb + 100) * 2**20


def test_a_smaller_budget_gives_back_what_a_larger_left(native_lib):
    d = random_dfa(300, 2, 5)
    plan = lambda mb: json.dumps({"algorithms": [{"name": "Exact", "config": {"max_memory_mb": mb, "dfs": False}}]})
    with sw.Context(0) as c:
        small = c.solve(d, 300, 2, plan(40))
        c.solve(d, 300, 2, plan(400))
        again = c.solve(d, 300, 2, plan(40))
    assert (small.lower, small.upper) == (again.lower, again.upper)
