"""The synchronisation of the one-launch small-matrix kernel (small.cu): read from
its source on the CPU, and the batches and invalid matrices that depend on it on
the GPU, against the oracle."""
import os
import re

import pytest

import oracle
from gb_b200 import _lib, la, synth
from gb_b200.matrix import MacaulayMatrix

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "gb_b200", "csrc")
PRIMES = [2, 251, 65521, 65537, 2147483647]


def body_of(source, name):
    """The braces of the function `name` in csrc/`source`, comments left out."""
    with open(os.path.join(CSRC, source)) as fh:
        text = re.sub(r"//[^\n]*", "", fh.read())
    at = text.index("{", re.search(rf"\b{name}\([^;{{]*\)\s*{{", text).start())
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == "{") - (text[i] == "}")
        if depth == 0:
            return text[at:i + 1]
    raise AssertionError(name)


def test_clusters_meet_before_the_first_remote_store():
    """A CTA's shared memory may be written by another one only after it is known
    to run: a cluster barrier before the first store, in the kernel's own text."""
    body = body_of("small.cu", "k_small")
    assert body.index("cluster_sync()") < body.index("remote_st(")


@pytest.mark.gpu
@pytest.mark.parametrize("count", [1, 18, 19, 37, 149, 300])
def test_batches_around_the_clusters_of_the_device(count):
    """One matrix, as many as clusters of eight (and of four, two, one) fit, and
    more: the first entry of every cluster comes from the queue."""
    mats = [synth.random_macaulay(5 + i % 23, 1 + i % 17, 4 + i % 31, PRIMES[i % len(PRIMES)],
                                  density=0.3, seed=count + i) for i in range(count)]
    want = [oracle.oracle_la(m)[0] for m in mats]
    for _ in range(3):
        answers, status = la.reduce_batch(mats)
        assert not any(status)
        for i, (a, w) in enumerate(zip(answers, want)):
            assert a.equals(w), (i, a.first_difference(w))


def test_the_checks_verdict_is_uniform_where_barriers_depend_on_it():
    """Between the read that opens the branch with block barriers and the next
    cluster barrier nothing writes the word that was read."""
    body = body_of("small.cu", "small_prep")
    part = body[body.index("const bool good"):]
    part = part[:part.index("cluster_sync()")]
    assert "__syncthreads()" in part and "__ldcg(a.err) == 0" in part
    assert not re.search(r"atomic\w+\(\s*a\.err\s*,|\*a\.err\s*=|a\.err\[0\]\s*=", part)


def without_pivots(m, columns):
    """`m` with the rows of the given left columns' pivots led by column 0 instead:
    every row is valid, the columns have no pivot."""
    cols = m.cols.copy()
    for i in range(m.nr):
        b, e = m.row_ptr[i], m.row_ptr[i + 1]
        if cols[b] in columns:
            assert 0 not in cols[b:e]
            cols[b] = 0
    return MacaulayMatrix(m.p, m.ncl, m.ncr, m.row_ptr, cols, m.vals)


@pytest.mark.gpu
@pytest.mark.parametrize("p", [251, 65521, 2147483647])
@pytest.mark.parametrize("nru,nrl,ncr", [(3, 1, 2), (130, 40, 60), (900, 30, 90), (1400, 20, 50),
                                         (300, 200, 50)])
def test_missing_pivots_of_valid_rows(nru, nrl, ncr, p):
    """One launch and three, alone and beside valid matrices: the call is refused
    with that reason, and the next one is answered."""
    m = synth.random_macaulay(nru, nrl, ncr, p, density=0.05, seed=nru + nrl)
    want, _ = oracle.oracle_la(m)
    for columns in ({nru - 1}, set(range(1, nru))):
        bad = without_pivots(m, columns)
        with pytest.raises(_lib.GbgpuError) as ei:
            la.linear_algebra(bad)
        assert ei.value.code == _lib.GBGPU_EINVAL and "pivot" in str(ei.value)
        assert la.linear_algebra(m).equals(want)
        answers, status = la.reduce_batch([bad, m] * 5)
        assert list(status) == [_lib.GBGPU_EINVAL, 0] * 5
        assert all(a is None for a in answers[::2])
        assert all(a.equals(want) for a in answers[1::2])
