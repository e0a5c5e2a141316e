"""The cluster echelon of small blocks (tiny.cuh) at the sizes where its panels,
owners, sweeps and warps change, against the oracle: a Macaulay
matrix whose Schur complement is the block itself, alone and in a batch call."""
import numpy as np
import pytest

import oracle
from gb_b200 import la, synth

pytestmark = pytest.mark.gpu

# (rows, columns, rank): one row and column; around a 16-column panel; around a
# warp's 16 rows; panels that wrap around the eight CTAs; around a sweep of 256
# rows; tall, wide and large blocks
SHAPES = [(1, 1, 1), (1, 40, 1), (2, 15, 2), (7, 16, 5), (16, 17, 16), (20, 31, 9), (33, 33, 33),
          (40, 48, 17), (49, 49, 48), (100, 191, 64), (129, 130, 120), (255, 60, 60),
          (257, 100, 99), (1030, 20, 19), (12, 1500, 12), (60, 800, 33), (220, 225, 220),
          (400, 700, 370)]
PRIMES = [2, 3, 251, 65521, 65537, 2147483647]


def block(n, m, rank, p, kind, seed):
    D = synth.dense_lowrank(n, m, rank, p, seed=seed)
    rng = np.random.default_rng(seed)
    if kind == "sparse":  # many rows untouched by a pivot, empty panels
        D = np.where(rng.random((n, m)) < 0.08, D, 0)
        D[:, rng.integers(0, m):][:, :20] = 0
    elif kind == "largest":  # every residue p - 1 or 0
        D = np.where(rng.random((n, m)) < 0.7, p - 1, 0)
    return D


@pytest.mark.parametrize("kind", ["dense", "sparse", "largest"])
@pytest.mark.parametrize("p", PRIMES)
def test_tiny_echelon_matches_oracle(p, kind):
    mats = [synth.dense_block_macaulay(block(n, m, r, p, kind, 3 * n + m), p)
            for n, m, r in SHAPES]
    want = [oracle.oracle_la(m)[0] for m in mats]
    for (n, m, r), mat, w in zip(SHAPES, mats, want):
        got = la.linear_algebra(mat)
        assert got.equals(w), (n, m, r, got.first_difference(w))
    answers, status = la.reduce_batch(mats)
    assert not any(status)
    for s, a, w in zip(SHAPES, answers, want):
        assert a.equals(w), (s, a.first_difference(w))
