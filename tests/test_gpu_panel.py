"""The echelon's panel factorization and its application at their edges (rows of
a panel around 16 and 256, panels cut by the last column, one and many panels,
dependent rows, staircase leads), through the dense RREF, against a plain
Gauss-Jordan."""
import ctypes as C

import numpy as np
import pytest

from gb_b200 import _lib

pytestmark = pytest.mark.gpu


def rref(D, p):
    A = D.astype(np.int64) % p
    r, piv = 0, []
    for c in range(A.shape[1]):
        nz = np.flatnonzero(A[r:, c])
        if nz.size == 0:
            continue
        A[[r, r + nz[0]]] = A[[r + nz[0], r]]
        A[r] = A[r] * pow(int(A[r, c]), p - 2, p) % p
        f = A[:, c].copy()
        f[r] = 0
        rows = np.flatnonzero(f)
        A[rows] = (A[rows] - f[rows, None] * A[r][None, :] % p) % p
        piv.append(c)
        r += 1
        if r == A.shape[0]:
            break
    return A, piv


def block(kind, m, n, p, seed):
    rng = np.random.default_rng(seed)
    D = rng.integers(0, p, size=(m, n), dtype=np.int64)
    if kind == "stairs":  # leads spread over the columns: many panels a round
        for i in range(m):
            D[i, : rng.integers(0, n)] = 0
    elif kind == "multiples":  # many dependent rows in one panel
        base = D[: max(1, m // 5)]
        D = base[rng.integers(0, base.shape[0], m)] * rng.integers(1, p, (m, 1)) % p
    elif kind == "gaps":  # columns without a pivot inside the panels
        D[:, rng.random(n) < 0.4] = 0
        D[rng.random((m, n)) < 0.5] = 0
    return D


@pytest.mark.parametrize("kind", ["dense", "stairs", "multiples", "gaps"])
@pytest.mark.parametrize("p", [2, 3, 251, 65521, 65537, 2147483647])
@pytest.mark.parametrize("m,n", [(1, 130), (15, 17), (17, 128), (129, 129), (255, 300), (257, 127),
                                 (330, 400)])
def test_dense_rref_panels(kind, p, m, n):
    torch = pytest.importorskip("torch")
    D = block(kind, m, n, p, m + n)
    want, piv = rref(D, p)
    dev = torch.from_numpy(D.astype(np.int32)).cuda()
    pc = torch.zeros(min(m, n), dtype=torch.int32, device="cuda")
    rank = C.c_int32()
    opt = _lib.Options(_lib.FORM_AUTO, 0, 1, 0, torch.cuda.current_stream().cuda_stream)
    _lib.check(_lib.load().gbgpu_dense_rref(p, m, n, dev.data_ptr(), n, C.byref(rank),
                                            pc.data_ptr(), C.byref(opt)))
    assert rank.value == len(piv)
    assert pc.cpu().numpy()[: rank.value].tolist() == piv
    assert np.array_equal(dev.cpu().numpy(), want)
