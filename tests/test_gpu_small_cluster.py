"""The synchronisation of the one-launch small-matrix kernel (small.cu): read from
its source on the CPU, and the batches and invalid matrices that depend on it on
the GPU, against the oracle."""
import os
import re

import pytest

import oracle
from gb_b200 import la, synth

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
