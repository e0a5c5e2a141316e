"""The echelon's round bookkeeping at its edges (more rows than one batch of a
warp, more panels than are counted in shared memory, clean and dirty panels,
rows left for a next round), through the dense RREF, against a plain
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
    """dense rows; or rows of a few entries near a lead, with `lead_of(i)` rows
    sharing it: two a panel (all dirty), one (all clean), or a mix"""
    rng = np.random.default_rng(seed)
    if kind == "dense":
        return rng.integers(0, p, size=(m, n), dtype=np.int64)
    D = np.zeros((m, n), dtype=np.int64)
    share = {"clean": 1, "dirty": 2, "mixed": 3}[kind]
    groups = (m + share - 1) // share
    for i in range(m):
        g = i % groups
        lead = g * n // groups
        if kind == "mixed" and g % 2:
            lead = min(n - 1, lead + i // groups)
        D[i, lead] = rng.integers(1, p)
        at = lead + 1 + rng.integers(0, 130, size=6)
        at = at[at < n]
        D[i, at] = rng.integers(0, p, size=at.size)
    return D[rng.permutation(m)]


@pytest.mark.parametrize("kind,m,n,p", [
    ("dense", 8200, 40, 65521), ("dense", 9000, 131, 2147483647), ("dense", 1025, 140, 251),
    ("clean", 1030, 5000, 65521), ("dirty", 1030, 5000, 2147483647), ("mixed", 900, 4097, 65521),
    ("dirty", 620, 40000, 65521), ("mixed", 700, 40003, 2147483647), ("clean", 310, 40001, 251)])
def test_dense_rref_rounds(kind, m, n, p):
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


@pytest.mark.parametrize("p", [3, 251, 65521, 65537, (1 << 24) + 43, 2147483647])
@pytest.mark.parametrize("rows,n", [
    ((2, 33, 64), 400), ((65, 16, 128), 397), ((31, 32, 17, 127, 63), 645), ((130, 1, 129), 500)])
def test_chunks_of_every_size(rows, n, p):
    """panel q has rows[q] rows of its own, so its chunk finds up to that many pivots"""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n + len(rows))
    D = np.zeros((sum(rows), n), dtype=np.int64)
    at = 0
    for q, r in enumerate(rows):
        D[at:at + r, 128 * q:] = rng.integers(0, p, size=(r, n - 128 * q))
        at += r
    D = D[rng.permutation(at)]
    want, piv = rref(D, p)
    dev = torch.from_numpy(D.astype(np.int32)).cuda()
    pc = torch.zeros(min(D.shape), dtype=torch.int32, device="cuda")
    rank = C.c_int32()
    opt = _lib.Options(_lib.FORM_AUTO, 0, 1, 0, torch.cuda.current_stream().cuda_stream)
    _lib.check(_lib.load().gbgpu_dense_rref(p, *D.shape, dev.data_ptr(), n, C.byref(rank),
                                            pc.data_ptr(), C.byref(opt)))
    assert rank.value == len(piv)
    assert pc.cpu().numpy()[: rank.value].tolist() == piv
    assert np.array_equal(dev.cpu().numpy(), want)
