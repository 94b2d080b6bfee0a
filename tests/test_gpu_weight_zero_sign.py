"""Row means and weight sums that are zero are +0.0, as sums from 0.0 are,
whatever the signs of the zeros summed and however long the row."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("longest", [1, 2, 3, 8, 9, 40])
def test_sums_of_negative_zeros(longest):
    from numba_celltree_gb300.regrid import WeightMatrix

    lengths = np.arange(longest, 0, -1)  # alone (1) and beside longer rows of a warp
    rows = np.repeat(np.arange(longest), lengths)
    cols = np.arange(len(rows)) % 7
    w = np.ones(len(rows))
    m = WeightMatrix.from_intersections(rows, cols, w, longest, 7)
    mean = m.mean(np.full(7, -0.0))
    assert np.array_equal(mean, np.zeros(longest)) and not np.signbit(mean).any()
    ws = WeightMatrix.from_intersections(rows, cols, -0.0 * w, longest, 7).weight_sum.cpu().numpy()
    assert np.array_equal(ws, np.zeros(longest)) and not np.signbit(ws).any()
