"""The small path's unreduced 64-bit sums at their largest: every known pivot adds a
product to every right column, up to the most left columns the path takes, against
plain integers."""
import numpy as np
import pytest

from gb_b200 import _lib, la
from gb_b200.matrix import MacaulayMatrix

pytestmark = pytest.mark.gpu


def rref(M, p):
    """Rows of the reduced echelon form, descending leads (Python integers)."""
    M, out = M.astype(object), []
    for c in range(M.shape[1]):
        i = next((i for i in range(len(out), len(M)) if M[i, c]), None)
        if i is None:
            continue
        k = len(out)
        M[[k, i]] = M[[i, k]]
        M[k] = M[k] * pow(int(M[k, c]), -1, p) % p
        for r in range(len(M)):
            if r != k and M[r, c]:
                M[r] = (M[r] - M[r, c] * M[k]) % p
        out.append(k)
    return M[: len(out)][::-1]


@pytest.mark.parametrize("p", [251, 65521, 65537, 2147483647])
@pytest.mark.parametrize("ncl", [1, 1000, 1025, 3001, 7001, 12288])
@pytest.mark.parametrize("entry", ["ones", "largest"])
def test_every_pivot_in_every_sum(ncl, entry, p):
    """Pivots [e_i | p - 1 .. p - 1]; rows of ones have the largest multipliers (p - 1),
    rows of p - 1 the smallest, and end in random right parts."""
    nrl, ncr = 9, 11
    rng = np.random.default_rng(ncl)
    right = rng.integers(1, p, size=(nrl, ncr))
    piv_cols = np.concatenate([np.arange(ncl)[:, None], np.tile(ncl + np.arange(ncr), (ncl, 1))], 1)
    piv_vals = np.full((ncl, 1 + ncr), p - 1)
    piv_vals[:, 0] = 1
    left = np.full(ncl, 1 if entry == "ones" else p - 1)
    left[0] = 1
    row_cols = np.tile(np.arange(ncl + ncr), (nrl, 1))
    row_vals = np.concatenate([np.tile(left, (nrl, 1)), right], 1)
    # the rows to reduce have lead 0, as the first pivot, which comes before them
    cols = np.concatenate([piv_cols[0], row_cols.ravel(), piv_cols[1:].ravel()])
    vals = np.concatenate([piv_vals[0], row_vals.ravel(), piv_vals[1:].ravel()])
    lens = np.concatenate([[1 + ncr], np.full(nrl, ncl + ncr), np.full(ncl - 1, 1 + ncr)])
    ptr = np.concatenate([[0], np.cumsum(lens)])
    m = MacaulayMatrix(p, ncl, ncr, ptr, cols, vals)
    lib = _lib.load()
    before = lib.gbgpu_kernel_launches()
    got = la.linear_algebra(m)
    assert lib.gbgpu_kernel_launches() - before == (1 if ncl <= 1024 else 3)
    total = sum(int(x) for x in left) * (p - 1)
    want = rref(np.array([[(int(x) - total) % p for x in row] for row in right], dtype=object), p)
    assert got.np == len(want)
    dense = np.zeros(want.shape, dtype=object)
    for i in range(got.np):
        b, e = got.row_ptr[i], got.row_ptr[i + 1]
        dense[i, got.cols[b:e] - ncl] = got.vals[b:e]
    assert np.array_equal(dense, want)
