"""Small matrices of many left columns: the three-launch form of the small path
(small.cu) up to the columns that two accumulators of an SM hold, against the
oracle."""
import numpy as np
import pytest

import oracle
from gb_b200 import _lib, la
from gb_b200.matrix import MacaulayMatrix

pytestmark = pytest.mark.gpu

COLUMNS = 14400  # two accumulators
LEFT = 12288


def banded(nru, nrl, ncr, p, seed, per_row=12, rest_len=6):
    """Known pivots with a few entries near their lead and in the right block, rows to
    reduce with entries in every part of the left block."""
    rng = np.random.default_rng(seed)
    nc = nru + ncr
    rows = []
    for i in range(nru):
        near = i + 1 + rng.choice(60, size=per_row // 2, replace=False)
        right = nru + rng.choice(ncr, size=min(ncr, rest_len), replace=False)
        rows.append((i, 0, np.unique(np.concatenate([near[near < nru], right]))))
    for _ in range(nrl):
        lead = int(rng.integers(0, max(1, nru // 4)))
        left = lead + 1 + rng.choice(nru - 1 - lead, size=per_row, replace=False)
        right = nru + rng.choice(ncr, size=min(ncr, rest_len), replace=False)
        rows.append((lead, 1, np.unique(np.concatenate([left, right]))))
    rows.sort(key=lambda r: (r[0], r[1]))
    cols = [np.concatenate([[lead], rest]) for lead, _, rest in rows]
    ptr = np.concatenate([[0], np.cumsum([len(c) for c in cols])])
    vals = rng.integers(1, p, size=ptr[-1])
    vals[ptr[:-1]] = 1
    assert ptr[-1] == sum(map(len, cols)) and max(map(max, cols)) < nc
    return MacaulayMatrix(p, nru, ncr, ptr, np.concatenate(cols), vals)


def launches(m):
    lib = _lib.load()
    before = lib.gbgpu_kernel_launches()
    got = la.linear_algebra(m)
    return got, lib.gbgpu_kernel_launches() - before


@pytest.mark.parametrize("p", [3, 251, 65521, 65537, 2147483647])
@pytest.mark.parametrize("nru,nrl,ncr", [
    (6999, 40, 200), (7001, 40, 200), (7001, 40, 199), (8000, 127, 200), (8000, 200, 127),
    (12001, 1500, 20), (LEFT, 90, COLUMNS - LEFT)])
def test_few_rows_after_many_left_columns(nru, nrl, ncr, p):
    m = banded(nru, nrl, ncr, p, seed=nru + nrl)
    want, _ = oracle.oracle_la(m)
    got, n = launches(m)
    assert n == 3
    assert got.equals(want), got.first_difference(want)


@pytest.mark.parametrize("nru,nrl,ncr", [
    (8000, 128, 128), (LEFT, 90, COLUMNS - LEFT + 1), (LEFT + 1, 20, 30)])
def test_other_matrices_leave_it(nru, nrl, ncr):
    m = banded(nru, nrl, ncr, 65521, seed=nru + nrl)
    want, _ = oracle.oracle_la(m)
    got, n = launches(m)
    assert n > 3
    assert got.equals(want), got.first_difference(want)


@pytest.mark.parametrize("ncr,small", [(1, True), (COLUMNS - 700, True), (COLUMNS - 699, False),
                                       (300000, False)])
def test_known_pivots_alone(ncr, small):
    """Nothing to reduce: an empty answer, and only the checks of the general path
    (no copy through pinned memory) once the rows are long."""
    m = banded(700, 0, ncr, 65521, seed=ncr)
    got, n = launches(m)
    assert (n == 1) == small
    assert got.np == 0 and got.nnz == 0
    m.vals[m.row_ptr[699]] = 2
    with pytest.raises(_lib.GbgpuError) as ei:
        la.linear_algebra(m)
    assert ei.value.code == _lib.GBGPU_EINVAL
