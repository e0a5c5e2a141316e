"""Interreduction on both its paths (row by row, and one dense back
substitution) at the edges of the rule between them and of the blocks of 128 and
1024 pivots, against a plain Gauss-Jordan."""
import ctypes as C

import numpy as np
import pytest

from gb_b200 import _lib

pytestmark = pytest.mark.gpu


def basis(nr, nc, row_len, p, seed):
    """rows with distinct leads in any order, columns after the lead in any order"""
    rng = np.random.default_rng(seed)
    leads = rng.permutation(rng.choice(nc, size=nr, replace=False))
    cols, vals, ptr = [], [], [0]
    for lead in leads:
        k = min(row_len, nc - 1 - int(lead))
        rest = int(lead) + 1 + rng.choice(nc - 1 - int(lead), size=k, replace=False) if k else []
        cols.append(np.concatenate([[lead], rest]).astype(np.int32))
        vals.append(np.concatenate([[1], rng.integers(1, p, size=k)]).astype(np.int32))
        ptr.append(ptr[-1] + k + 1)
    return np.array(ptr, dtype=np.int64), np.concatenate(cols), np.concatenate(vals), leads


def reduced(ptr, cols, vals, leads, nc, p):
    """rows in ascending lead order, each reduced by all others"""
    M = np.zeros((len(leads), nc), dtype=np.int64)
    for i in range(len(leads)):
        M[i, cols[ptr[i]:ptr[i + 1]]] = vals[ptr[i]:ptr[i + 1]]
    order = np.argsort(leads)
    M, leads = M[order], leads[order]
    for i in range(len(leads) - 1, -1, -1):
        f = M[:i, leads[i]]
        rows = np.flatnonzero(f)
        M[rows] = (M[rows] - f[rows, None] * M[i][None, :] % p) % p
    return M


def run(nr, nc, p, ptr, cols, vals, form):
    opt = _lib.Options(form, 0, 1, 0, None)
    rows = _lib.Rows()
    lib = _lib.load()
    _lib.check(lib.gbgpu_interreduce(p, nr, nc, ptr.ctypes.data, cols.ctypes.data, vals.ctypes.data,
                                     C.byref(opt), C.byref(rows)))
    n = rows.np
    rp = np.ctypeslib.as_array(C.cast(rows.row_ptr, C.POINTER(C.c_int64)), (n + 1,)).copy()
    cs = np.ctypeslib.as_array(C.cast(rows.cols, C.POINTER(C.c_int32)), (rp[-1],)).copy()
    vs = np.ctypeslib.as_array(C.cast(rows.vals, C.POINTER(C.c_int32)), (rp[-1],)).copy()
    lib.gbgpu_rows_free(C.byref(rows))
    return rp, cs, vs


@pytest.mark.parametrize("p", [3, 251, 32003, 65537, 2147483647])
@pytest.mark.parametrize("nr,nc,row_len", [
    (127, 200, 120), (128, 129, 128), (256, 513, 60), (385, 999, 3), (640, 641, 640),
    (300, 40000, 1500), (1025, 2501, 12), (1300, 20000, 1)])
def test_interreduce_both_paths(p, nr, nc, row_len):
    ptr, cols, vals, leads = basis(nr, nc, row_len, p, nr + nc)
    want = reduced(ptr, cols, vals, leads, nc, p)
    rp, cs, vs = run(nr, nc, p, ptr, cols, vals, _lib.FORM_AUTO)
    assert len(rp) == nr + 1
    got = np.zeros_like(want)
    row = np.repeat(np.arange(nr), np.diff(rp))
    got[row, cs] = vs
    assert np.array_equal(got, want)
    assert all(np.array_equal(a, b) for a, b in
               zip((rp, cs, vs), run(nr, nc, p, ptr, cols, vals, _lib.FORM_PLAIN)))
