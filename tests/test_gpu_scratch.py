"""Device memory of the echelon: what a round uses serves the next one, so the
scratch of a block does not grow with its number of rounds."""
import ctypes as C

import pytest

from gb_b200 import _lib

pytestmark = pytest.mark.gpu

PANEL = 128  # columns of a round


def pool_peak(torch, call):
    """Bytes of the device's stream-ordered pool in use at the most during call()."""
    rt = pytest.importorskip("cuda.bindings.runtime")
    driver = pytest.importorskip("cuda.bindings.driver")
    err, pool = rt.cudaDeviceGetDefaultMemPool(0)
    assert err == rt.cudaError_t.cudaSuccess
    torch.cuda.synchronize()
    high = rt.cudaMemPoolAttr.cudaMemPoolAttrUsedMemHigh
    err, base = rt.cudaMemPoolGetAttribute(pool, rt.cudaMemPoolAttr.cudaMemPoolAttrUsedMemCurrent)
    assert err == rt.cudaError_t.cudaSuccess
    assert rt.cudaMemPoolSetAttribute(pool, high, driver.cuuint64_t(0))[0] == rt.cudaError_t.cudaSuccess
    call()
    torch.cuda.synchronize()
    err, peak = rt.cudaMemPoolGetAttribute(pool, high)
    assert err == rt.cudaError_t.cudaSuccess
    return int(peak) - int(base)


def limbs(p):
    return (int(p - 1).bit_length() + 7) // 8


@pytest.mark.parametrize("p", [251, 65521, 2147483647])
@pytest.mark.parametrize("rows,cols", [(60000, 1024), (60000, 3072)])
def test_rref_scratch_does_not_grow_with_rounds(rows, cols, p):
    """A dense block: every round has one panel, all rows but its pivots are left."""
    torch = pytest.importorskip("torch")
    g = torch.Generator(device="cuda")
    g.manual_seed(cols)
    D = torch.randint(0, p, (rows, cols), device="cuda", dtype=torch.int64, generator=g).to(torch.int32)
    piv = torch.zeros(cols, dtype=torch.int32, device="cuda")
    opt = _lib.Options(_lib.FORM_TENSOR, 0, 1, 0, torch.cuda.current_stream().cuda_stream)
    rank = C.c_int32()
    lib = _lib.load()

    def call():
        _lib.check(lib.gbgpu_dense_rref(p, rows, cols, D.data_ptr(), cols, C.byref(rank),
                                        piv.data_ptr(), C.byref(opt)))

    peak = pool_peak(torch, call)
    assert rank.value == cols
    # the rows in answer order; a round's pivot columns of all rows (4 bytes), with the
    # limb planes of the round's product (rows x 128 and 128 x cols, each held while it
    # grows to the next larger one); the back substitution's inverses, its row block and
    # limb planes (blocks of 1024 pivots)
    order = 4 * rows * cols
    rounds = 4 * rows * PANEL + 2 * limbs(p) * PANEL * (rows + cols + 256)
    back = 8 * 3 * 1024 * cols + 4 * 1024 * cols + 2 * limbs(p) * 2 * 1024 * (cols + 1024)
    lists = 64 * (rows + cols) + 4 * PANEL * PANEL * (cols // PANEL)
    assert peak <= order + rounds + back + lists + (16 << 20), (peak, order, rounds, back, lists)
