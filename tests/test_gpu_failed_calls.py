"""Calls that end for want of device memory leave their context usable: the
next calls on it give what a fresh context gives."""
import numpy as np
import pytest

import synchrowords_gb300 as sw

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
