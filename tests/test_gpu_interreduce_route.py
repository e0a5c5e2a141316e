"""Which path an interreduction takes (api.cu): rows that meet enough pivots, and are
enough for the prime's limbs, are reduced by one dense back substitution.  Told by the
kernel launches of the call; the answers are those of the row form."""
import numpy as np
import pytest

from gb_b200 import _lib
from test_gpu_interreduce import run

pytestmark = pytest.mark.gpu

TOTAL, PER_ROW = 3000, 4  # entries at pivot columns from which on the path is dense


def basis(nr, hits, p, seed):
    """Row i has lead i; `hits` entries at pivot columns, leads included, and a few
    right of all leads."""
    rng = np.random.default_rng(seed)
    nc = nr + 40
    more = np.zeros(nr, dtype=int)
    for _ in range(hits - nr):
        i = rng.integers(0, nr - 1)
        while more[i] >= nr - 1 - i:
            i = rng.integers(0, nr - 1)
        more[i] += 1
    cols = [np.concatenate([[i], i + 1 + rng.choice(nr - 1 - i, size=more[i], replace=False),
                            nr + rng.choice(40, size=5, replace=False)]) for i in range(nr)]
    ptr = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int64)
    vals = rng.integers(1, p, size=ptr[-1]).astype(np.int32)
    vals[ptr[:-1]] = 1
    return nc, ptr, np.concatenate(cols).astype(np.int32), vals


def launches(nr, nc, p, ptr, cols, vals, form):
    lib = _lib.load()
    before = lib.gbgpu_kernel_launches()
    answer = run(nr, nc, p, ptr, cols, vals, form)
    return answer, lib.gbgpu_kernel_launches() - before


@pytest.mark.parametrize("p", [2, 251, 65521, 65537, 2147483647])
@pytest.mark.parametrize("nr,hits", [(127, TOTAL), (128, TOTAL - 1), (128, TOTAL), (159, TOTAL),
                                     (160, TOTAL - 1), (160, TOTAL), (900, PER_ROW * 900 - 1),
                                     (900, PER_ROW * 900)])
def test_path_by_rows_entries_and_prime(nr, hits, p):
    case = basis(nr, hits, p, seed=nr)
    rows, plain = launches(nr, case[0], p, *case[1:], _lib.FORM_PLAIN)
    auto, n = launches(nr, case[0], p, *case[1:], _lib.FORM_AUTO)
    assert all(np.array_equal(a, b) for a, b in zip(auto, rows))
    asked = p > 2 and nr >= (128 if p < 65536 else 160)  # counts its entries: one launch
    dense = asked and hits >= max(TOTAL, PER_ROW * nr)
    if dense:
        assert n > plain + 1
    else:
        assert n == plain + asked
