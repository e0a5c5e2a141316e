"""The tile shape of a tensor-core product (tc_shape.h), compiled for the host: what a
tuning file may change and what it may not."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "gb_b200", "csrc")
BIG, MID = 0, 2
SMS = 148


@pytest.fixture(scope="module")
def shape(tmp_path_factory):
    d = tmp_path_factory.mktemp("shape")
    (d / "q.cpp").write_text("""
#include <cstdio>
#include "tc_shape.h"
int main() {
    long long L, M, N, K, batch, sms, tuned;
    while (scanf("%lld %lld %lld %lld %lld %lld %lld", &L, &M, &N, &K, &batch, &sms, &tuned) == 7)
        printf("%d\\n", gbgpu::tc_shape((int)L, M, N, (int)K, batch, (int)sms, (int)tuned));
}
""")
    subprocess.run(["g++", "-std=c++17", "-I" + CSRC, str(d / "q.cpp"), "-o", str(d / "q")], check=True)

    def ask(queries):
        text = "\n".join(" ".join(map(str, q)) for q in queries)
        out = subprocess.run([str(d / "q")], input=text, capture_output=True, text=True, check=True)
        return [int(x) for x in out.stdout.split()]

    return ask


def waves(L, M, N, batch):
    cols = 256 if L == 1 else 128
    tiles = -(-M // 128) * -(-N // cols) * batch
    return -(-tiles // SMS)


SIZES = [(128, 64), (130, 65), (512, 512), (1024, 1024), (2520, 1220), (2520, 2500), (3032, 1476),
         (1216, 9472), (2368, 9472), (4736, 3072), (4096, 4096), (5000, 20000), (8192, 8192)]
DEPTHS = [1, 128, 200, 256, 937, 1536, 2000, 4000, 8192]


@pytest.mark.parametrize("batch", [1, 7])
@pytest.mark.parametrize("L", [1, 2, 3, 4])
def test_tuning_reaches_the_products_it_was_timed_on(shape, L, batch):
    """At most three waves of tiles: the same shape with any table.  More: the
    table's (the wide shape without one); three and four limbs have one shape."""
    for M, N in SIZES:
        for K in DEPTHS:
            none, big, mid = shape([(L, M, N, K, batch, SMS, t) for t in (-1, BIG, MID)])
            if L > 2:
                assert none == big == mid == BIG
            elif waves(L, M, N, batch) <= 3:
                assert none == big == mid, (M, N, K)
            else:
                assert (none, big, mid) == (BIG, BIG, MID), (M, N, K)


def test_measured_choices(shape):
    """The sizes both shapes were timed at: two limbs, then one."""
    got = shape([(2, 512, 512, 128, 1, SMS, -1), (2, 1024, 1024, 1024, 1, SMS, -1),
                 (2, 2520, 1220, 200, 1, SMS, -1), (2, 2520, 1220, 937, 1, SMS, -1),
                 (2, 2520, 1220, 4000, 1, SMS, -1), (2, 3032, 1476, 2000, 1, SMS, -1),
                 (2, 5000, 20000, 256, 1, SMS, -1), (1, 2520, 2500, 200, 1, SMS, -1),
                 (1, 2520, 2500, 2000, 1, SMS, -1)])
    assert got == [MID, MID, MID, MID, BIG, BIG, BIG, MID, BIG]
