"""Row pointers and row means of WeightMatrix at the edges of the kernel's row
classes: rows of up to 8 entries on 8 lanes, longer ones on a warp in steps of
128, 4 to 32 rows per warp by the number of rows."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 2, 7, 8, 9, 31, 32, 33, 127, 128, 129, 255, 257, 1000]


def _case(lengths, n_cols=97, seed=0):
    rng = np.random.default_rng(seed)
    lengths = np.asarray(lengths, dtype=np.int64)
    rows = np.repeat(np.arange(len(lengths)), lengths)
    return rows, rng.integers(0, n_cols, len(rows)), rng.random(len(rows)) + 0.5, rng.normal(size=n_cols)


@pytest.mark.parametrize("n_rows", [1, 3, 4, 5, 1000, 80_000, 160_000, 320_000, 1_300_000])
def test_rows_of_every_length(n_rows):
    from numba_celltree_gb300.regrid import WeightMatrix

    rng = np.random.default_rng(n_rows)
    lengths = rng.integers(0, 4, n_rows)
    at = rng.permutation(n_rows)[: len(LENGTHS)]
    lengths[at] = LENGTHS[: len(at)]
    lengths[-1] = 0 if n_rows % 2 else lengths[-1]  # an empty last row too
    rows, cols, w, x = _case(lengths)
    m = WeightMatrix.from_intersections(rows, cols, w, n_rows, len(x))
    ptr = np.concatenate([[0], np.cumsum(lengths)])
    assert np.array_equal(m.row_ptr.cpu().numpy(), ptr)
    mean, ws = m.mean(x), m.weight_sum.cpu().numpy()
    num = np.zeros(n_rows, dtype=np.longdouble)
    den = np.zeros(n_rows, dtype=np.longdouble)
    mag = np.zeros(n_rows)
    np.add.at(num, rows, w.astype(np.longdouble) * x[cols])
    np.add.at(den, rows, w.astype(np.longdouble))
    np.add.at(mag, rows, np.abs(w * x[cols]))
    held = lengths > 0
    assert np.array_equal(np.isnan(mean), ~held)
    u = 2.0**-53  # a sum of n rounded terms is off by at most n u times the sum of their magnitudes
    n = lengths[held]
    den_h = den[held].astype(float)
    assert (np.abs(ws[held] - den_h) <= n * u * den_h).all()
    assert (np.abs(mean[held] - (num[held] / den[held]).astype(float)) <= (2 * n + 4) * u * mag[held] / den_h).all()


def test_no_pairs_and_bad_indices():
    from numba_celltree_gb300.regrid import WeightMatrix

    m = WeightMatrix.from_intersections([], [], [], 5, 3)
    assert np.array_equal(m.row_ptr.cpu().numpy(), np.zeros(6, dtype=np.int64))
    assert np.isnan(m.mean(np.ones(3))).all()
    rows, cols, w, x = _case([3, 0, 200])
    for k in (0, 4, 150):  # a column out of range in a short and in a long row
        bad = cols.copy()
        bad[k] = len(x)
        with pytest.raises(ValueError):
            WeightMatrix.from_intersections(rows, bad, w, 3, len(x)).mean(x)
    for r in (-1, 3):
        bad = rows.copy()
        bad[0 if r < 0 else -1] = r
        with pytest.raises(ValueError, match="out of range"):
            WeightMatrix.from_intersections(bad, cols, w, 3, len(x))
    with pytest.raises(ValueError, match="non-decreasing"):
        WeightMatrix.from_intersections(rows[::-1].copy(), cols, w, 3, len(x))
