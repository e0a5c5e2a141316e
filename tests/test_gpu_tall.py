"""Tall right blocks whose rows come to the cluster echelon in turns (plain.cu), at
the edges of a turn (1111 rows of one panel, 1109 of three, less the pivots kept),
of the panels and of the rule, by a call and by a plan, against the oracle."""
import numpy as np
import pytest

import oracle
from gb_b200 import _lib, la, synth
from gb_b200.matrix import MacaulayMatrix

pytestmark = pytest.mark.gpu


def matrix(D, p):
    """One left column: the pivot [1 | 0] and the rows [1 | D_i]."""
    n, m = D.shape
    row, col = np.nonzero(D)
    count = np.bincount(row, minlength=n) + 1
    ptr = np.concatenate([[0, 1], 1 + np.cumsum(count)])
    cols = np.zeros(ptr[-1], dtype=np.int32)
    vals = np.ones(ptr[-1], dtype=np.int32)
    rest = np.ones(ptr[-1], dtype=bool)
    rest[ptr[:-1]] = False
    cols[rest], vals[rest] = col + 1, D[row, col]
    return MacaulayMatrix(p, 1, m, ptr, cols, vals)


def block(n, m, rank, p, kind, seed):
    rng = np.random.default_rng(seed)
    D = synth.dense_lowrank(n, m, rank, p, seed=seed)
    if kind == "late":  # turn after turn one column more; its first rows are zero
        for j in range(m):
            D[: n * (m - 1 - j) // m, j] = 0
    elif kind == "sparse":  # most rows zero, columns without an entry
        D[rng.random(n) < 0.9] = 0
        D[:, rng.random(m) < 0.3] = 0
    elif kind == "zero":
        D[:] = 0
    return D


SHAPES = [(1111, 1, 1), (1112, 1, 1), (1111, 16, 16), (1112, 16, 9), (1111, 17, 17),
          (1109, 48, 48), (1110, 48, 47), (1110, 49, 49), (2170, 48, 48), (2206, 16, 16),
          (2207, 16, 5), (3000, 33, 20), (7100, 2, 2), (7400, 48, 40), (7770, 1, 1), (7771, 1, 1)]


@pytest.mark.parametrize("kind", ["dense", "late", "sparse", "zero"])
@pytest.mark.parametrize("p", [2, 251, 65521, 65537, 2147483647])
def test_tall_blocks_match_oracle(p, kind):
    for n, m, rank in SHAPES:
        mat = matrix(block(n, m, rank, p, kind, n + m), p)
        want, _ = oracle.oracle_la(mat)
        got = la.linear_algebra(mat)
        assert got.equals(want), (n, m, got.first_difference(want))
        plan = la.Plan(mat, form=_lib.FORM_PLAIN)
        plan.run()
        got = plan.result()
        plan.close()
        assert got.equals(want), (n, m, got.first_difference(want))
