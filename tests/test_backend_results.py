"""What a result array keeps alive: large results are views of the call's own
array (their unused pages were never written), small ones that fill little of
it are copies of their own size."""

import numpy as np
import pytest

from microsimulator_b200 import abi
from microsimulator_b200.backend import _HEAP_BYTES, _filled


@pytest.mark.parametrize("capacity,count,copied", [
    (1000, 0, True), (1000, 249, True), (1000, 250, False), (1000, 1000, False),
    (_HEAP_BYTES // abi.CELL_CONTACT_DTYPE.itemsize, 100, True),
    (_HEAP_BYTES // abi.CELL_CONTACT_DTYPE.itemsize + 1, 100, False),
])
def test_results_keep_little_more_than_themselves(capacity, count, copied):
    array = np.zeros(capacity, dtype=abi.CELL_CONTACT_DTYPE)
    array["first_id"][:count] = np.arange(count)
    result = _filled(array, count)
    assert len(result) == count and np.array_equal(result["first_id"], np.arange(count))
    assert np.shares_memory(result, array) != copied or count == 0
    if copied:
        assert result.base is None
