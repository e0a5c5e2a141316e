"""Plans of small right blocks: the cluster echelon up to the entries that one SM held,
the rounds of the sparse-row form beyond, against the oracle."""
import pytest

import oracle
from gb_b200 import _lib, la, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [2, 32003, 2147483647])
@pytest.mark.parametrize("nrl,ncr,rounds", [(100, 545, False), (50, 1105, False), (110, 502, False),
                                            (110, 503, True), (120, 600, True)])
def test_plan_route_by_block(nrl, ncr, rounds, p):
    m = synth.random_macaulay(150, nrl, ncr, p, density=0.1, seed=nrl + ncr, dup_rows=7)
    want, _ = oracle.oracle_la(m)
    plan = la.Plan(m, form=_lib.FORM_PLAIN)
    plan.run()
    got, stats = plan.result(), plan.stats()
    plan.close()
    assert got.equals(want), got.first_difference(want)
    assert (stats["echelon_rounds"] > 0) == rounds
