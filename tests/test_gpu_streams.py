"""What a finished plan leaves behind does not slow later calls down."""
import ctypes as C
import time

import pytest

from gb_b200 import _lib, la, synth

pytestmark = pytest.mark.gpu


def fastest(torch):
    """A pass of a small product: two launches, one allocation."""
    lib = _lib.load()
    A, B, D = (torch.zeros((64, 64), dtype=torch.int32, device="cuda") for _ in range(3))
    opt = _lib.Options(_lib.FORM_TENSOR, 0, 1, 0, torch.cuda.current_stream().cuda_stream)
    best = 1.0
    for _ in range(400):
        t0 = time.perf_counter()
        _lib.check(lib.gbgpu_dense_submul(251, 64, 64, 64, A.data_ptr(), 64, B.data_ptr(), 64,
                                          D.data_ptr(), 64, C.byref(opt)))
        torch.cuda.synchronize()
        best = min(best, time.perf_counter() - t0)
    return best


def plans(m, form, n):
    alive = [la.Plan(m, form=form) for _ in range(n)]
    for plan in alive:
        plan.run()
        plan.result()
    for plan in alive:
        plan.close()


@pytest.mark.parametrize("form", [_lib.FORM_PLAIN, _lib.FORM_TENSOR])
@pytest.mark.parametrize("nrl,ncr", [(60, 90), (200, 400)])
def test_calls_are_as_fast_after_plans_that_ran_side_by_side(nrl, ncr, form):
    """Parked streams with freed blocks of the pool make every stream-ordered allocation
    dearer, 2.7 us a stream: the product's fastest pass (about 45 us) after one plan and
    after twelve that were alive at once."""
    torch = pytest.importorskip("torch")
    m = synth.random_macaulay(300, nrl, ncr, 251, density=0.1, seed=1)
    plans(m, form, 1)
    before = fastest(torch)
    plans(m, form, 12)
    after = fastest(torch)
    assert after <= 1.2 * before, (before, after)
