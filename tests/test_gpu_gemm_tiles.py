"""The tensor-core GEMM's epilogue forms and tile shapes at their edges: aligned
and unaligned D (16-byte accesses or single ones), row and column tails, narrow
and wide tiles, one and several K panels of tiles; every entry exact, nothing
outside D written."""
import ctypes as C

import numpy as np
import pytest

from gb_b200 import _lib

pytestmark = pytest.mark.gpu


def exact_submul(D, A, B, p):
    A, B = A.astype(np.int64), B.astype(np.int64)
    lo = (A @ (B & 0xFFFF)) % p
    hi = (A @ (B >> 16)) % p
    return ((D.astype(np.int64) - lo - ((hi << 16) % p)) % p).astype(np.int32)


@pytest.mark.parametrize("p", [251, 65521, 1000003, 2147483647])
@pytest.mark.parametrize("M,N,K", [
    (1, 1, 1), (31, 33, 127), (128, 64, 128), (129, 65, 129), (127, 257, 130), (260, 3, 40),
    (1300, 1201, 96), (1031, 1413, 300)])
@pytest.mark.parametrize("off,extra", [(0, 0), (4, 4), (1, 0), (0, 1), (3, 6)])
def test_submul_edges(p, M, N, K, off, extra):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(M + 7 * N + K)
    ldd = (N + 3) // 4 * 4 + extra
    A = rng.integers(0, p, size=(M, K), dtype=np.int64).astype(np.int32)
    B = rng.integers(0, p, size=(K, N), dtype=np.int64).astype(np.int32)
    D = rng.integers(0, p, size=(M, N), dtype=np.int64).astype(np.int32)
    A[0, :], B[:, 0] = p - 1, p - 1
    buf = np.full(off + M * ldd + 8, -7, dtype=np.int32)
    view = buf[off:off + M * ldd].reshape(M, ldd)
    view[:, :N] = D
    dA, dB, dbuf = (torch.from_numpy(x).cuda() for x in (A, B, buf))
    opt = _lib.Options(_lib.FORM_TENSOR, 0, 1, 0, torch.cuda.current_stream().cuda_stream)
    _lib.check(_lib.load().gbgpu_dense_submul(p, M, N, K, dA.data_ptr(), K, dB.data_ptr(), N,
                                              dbuf.data_ptr() + 4 * off, ldd, C.byref(opt)))
    view[:, :N] = exact_submul(D, A, B, p)
    assert np.array_equal(dbuf.cpu().numpy(), buf)


def run(p, D, A, B, torch):
    M, K, N = A.shape[0], A.shape[1], B.shape[1]
    dA, dB, dD = (torch.from_numpy(x.astype(np.int32)).cuda() for x in (A, B, D))
    opt = _lib.Options(_lib.FORM_TENSOR, 0, 1, 0, torch.cuda.current_stream().cuda_stream)
    _lib.check(_lib.load().gbgpu_dense_submul(p, M, N, K, dA.data_ptr(), K, dB.data_ptr(), N,
                                              dD.data_ptr(), N, C.byref(opt)))
    return dD.cpu().numpy()


@pytest.mark.parametrize("p", [251, 65521])
@pytest.mark.parametrize("M,N,K", [(1112, 1220, 200), (2520, 1221, 937), (2083, 799, 2200),
                                   (1752, 2756, 500), (3032, 1476, 2000)])
def test_submul_few_waves(p, M, N, K):
    """sizes on both sides of the rule between the tile shapes (products below
    2^32 K: exact in doubles)"""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(M + N + K)
    A, B, D = (rng.integers(0, p, size=s).astype(np.float64) for s in ((M, K), (K, N), (M, N)))
    assert np.array_equal(run(p, D, A, B, torch), ((D - A @ B) % p).astype(np.int32))


@pytest.mark.parametrize("p,panel", [(251, 32768), (65521, 16384), (16777213, 10880),
                                     ((1 << 24) + 43, 8192), (2147483647, 8192)])
def test_submul_full_accumulators(p, panel):
    """every operand p - 1, a whole panel of K and the start of the next:
    A B = K mod p everywhere"""
    torch = pytest.importorskip("torch")
    K = panel + 64
    D = np.random.default_rng(K).integers(0, p, size=(130, 70))
    A, B = np.full((130, K), p - 1), np.full((K, 70), p - 1)
    assert np.array_equal(run(p, D, A, B, torch), ((D - K) % p).astype(np.int32))
