"""What a finished plan leaves behind does not slow later calls down."""
import ctypes as C
import time

import pytest

from gb_b200 import _lib, la, synth

pytestmark = pytest.mark.gpu


def test_calls_are_as_fast_after_plans_that_ran_side_by_side():
    """Streams kept alive make every stream-ordered allocation dearer: a small
    product (two launches, one allocation) alone and after twelve plans that were
    alive at once, each the fastest of many passes.  Eight parked streams cost a pass
    of about 45 us another 20."""
    torch = pytest.importorskip("torch")
    lib = _lib.load()
    A, B, D = (torch.zeros((64, 64), dtype=torch.int32, device="cuda") for _ in range(3))
    opt = _lib.Options(_lib.FORM_TENSOR, 0, 1, 0, torch.cuda.current_stream().cuda_stream)

    def fastest():
        best = 1.0
        for _ in range(400):
            t0 = time.perf_counter()
            _lib.check(lib.gbgpu_dense_submul(251, 64, 64, 64, A.data_ptr(), 64, B.data_ptr(), 64,
                                              D.data_ptr(), 64, C.byref(opt)))
            torch.cuda.synchronize()
            best = min(best, time.perf_counter() - t0)
        return best

    def plans(n):
        m = synth.random_macaulay(200, 60, 90, 251, density=0.1, seed=1)
        alive = [la.Plan(m) for _ in range(n)]
        for plan in alive:
            plan.run()
            plan.result()
        for plan in alive:
            plan.close()

    plans(1)
    before = fastest()
    plans(12)
    after = fastest()
    assert after <= 1.2 * before, (before, after)
