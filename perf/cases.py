"""Performance cases: the calls a user of the library makes, over the sizes they
are made at.

The library does the linear algebra of gb's F4 rounds over GF(p), so most cases
are whole reductions: the small matrices of early rounds and small systems (one
call, host rows in and out), batches of them, and the large staircase matrices
through a device-resident plan whose answer is delivered into the caller's
pinned host buffers at the prime's own coefficient width.  The rest are the
dense-block operations that can be called by themselves (the exact modular
product and the reduced echelon form of a block in device memory) and the final
interreduction of a basis.  Primes are of the three coefficient widths (8, 16
and 31 bits).  Values are uniform in [1, p) for sparse rows and in [0, p) for
dense blocks, which is how F4's coefficients look after the first reductions.

Kinds (the "kind" entry of a case):

* ``reduce``      ``gbgpu_reduce`` on one host matrix
* ``plan``        ``gbgpu_plan_run_into_v`` on a plan, pinned output buffers
* ``images``      ``gbgpu_reduce_batch`` on the images of one integer matrix modulo
                  the largest primes below 2^31 (the multi-modular driver's call)
* ``batch``       ``gbgpu_reduce_batch`` on independent uneven staircases
* ``interreduce`` ``gbgpu_interreduce`` on rows with distinct leads
* ``gemm``        ``gbgpu_dense_submul``, D <- D - A B mod p in place
* ``rref``        ``gbgpu_dense_rref`` on a copy of the block (it works in place)
"""
import ctypes as C
import math

import numpy as np
import torch

from gb_b200 import _lib, la, synth
from gb_b200.matrix import ReducedRows

P8, P15, P16, P31 = 251, 32003, 65521, 2147483647


def listed():
    return [
        # an la call of a small F4 run: quadratic system in 7 variables, rows of about
        # 36 terms; latency, launches and copies count
        {"name": "round_small", "kind": "reduce", "gen": "random", "nru": 300, "nrl": 141,
         "ncr": 191, "density": 0.08, "p": P15},
        # a middle F4 round in one call, host rows in and out
        {"name": "round_middle", "kind": "reduce", "gen": "staircase", "nru": 2001, "nrl": 517,
         "ncr": 2203, "dmin": 0.02, "dmax": 0.05, "p": P15},
        # the images a rational reduction needs, several primes a call
        {"name": "images_31bit", "kind": "images", "nru": 400, "nrl": 100, "ncr": 300,
         "dmin": 0.02, "dmax": 0.05, "bound": 64, "n": 16},
        # independent matrices of uneven size in one call
        {"name": "batch_uneven", "kind": "batch", "rows_min": 500, "rows_max": 5000, "n": 12,
         "dmin": 0.01, "dmax": 0.10, "p": P15},
        # the standalone A|B/C|D matrix of the benchmark
        {"name": "staircase_16bit", "kind": "plan", "nru": 20000, "nrl": 5000, "ncr": 20000,
         "dmin": 0.02, "dmax": 0.05, "p": P16},
        # a later round over a 31-bit prime
        {"name": "staircase_31bit", "kind": "plan", "nru": 6007, "nrl": 2003, "ncr": 9001,
         "dmin": 0.02, "dmax": 0.05, "p": P31},
        # and over an 8-bit prime
        {"name": "staircase_8bit", "kind": "plan", "nru": 10000, "nrl": 2500, "ncr": 10000,
         "dmin": 0.02, "dmax": 0.05, "p": P8},
        # the final basis: rows with distinct leads, reduced by one another
        {"name": "interreduce", "kind": "interreduce", "nr": 800, "nc": 3001, "row_len": 60,
         "p": P15},
        # dense Schur updates: one, two and four limbs, one of them ragged
        {"name": "gemm_8bit", "kind": "gemm", "m": 8192, "n": 8192, "k": 8192, "p": P8},
        {"name": "gemm_16bit_ragged", "kind": "gemm", "m": 5003, "n": 7001, "k": 3001, "p": P16},
        {"name": "gemm_31bit", "kind": "gemm", "m": 8192, "n": 8192, "k": 8192, "p": P31},
        # the echelon form of a dense D block
        {"name": "rref_16bit", "kind": "rref", "m": 8192, "n": 8192, "rank": 6144, "p": P16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: a kind by about the share of calls it has in use, its sizes
    over the whole range that the listed ones stand for."""
    kind = rng.choice(["reduce", "reduce", "plan", "plan", "images", "batch", "interreduce",
                       "gemm", "gemm", "rref"])
    p = rng.choice([P8, P15, P16, P31])
    if kind == "reduce":
        rows = _log(rng, 60, 4000)
        nrl = max(1, int(rows * rng.uniform(0.15, 0.4)))
        ncr = max(8, int(rows * rng.uniform(0.4, 1.2)))
        if rows <= 700:
            return {"kind": kind, "gen": "random", "nru": rows - nrl, "nrl": nrl, "ncr": ncr,
                    "density": round(rng.uniform(0.04, 0.2), 3), "p": p}
        return {"kind": kind, "gen": "staircase", "nru": rows - nrl, "nrl": nrl, "ncr": ncr,
                "dmin": 0.02, "dmax": 0.05, "p": p}
    if kind == "plan":
        rows = _log(rng, 1500, 10000 if p == P31 else 20000)
        nrl = max(1, int(rows * rng.uniform(0.15, 0.25)))
        return {"kind": kind, "nru": rows - nrl, "nrl": nrl,
                "ncr": int((rows - nrl) * rng.uniform(0.8, 1.3)), "dmin": 0.02, "dmax": 0.05,
                "p": p}
    if kind == "images":
        rows = rng.randint(100, 700)
        nrl = max(1, rows // 5)
        return {"kind": kind, "nru": rows - nrl, "nrl": nrl, "ncr": int(rows * 0.6),
                "dmin": 0.02, "dmax": 0.05, "bound": 64, "n": rng.choice([8, 16])}
    if kind == "batch":
        return {"kind": kind, "rows_min": 500, "rows_max": _log(rng, 1000, 5000),
                "n": rng.randint(4, 12), "dmin": 0.01, "dmax": 0.10, "p": p}
    if kind == "interreduce":
        nr = _log(rng, 50, 1000)
        return {"kind": kind, "nr": nr, "nc": int(nr * rng.uniform(2.0, 5.0)),
                "row_len": rng.randint(10, 80), "p": p}
    if kind == "gemm":
        hi = 6000 if p == P31 else 8192
        return {"kind": kind, "m": _log(rng, 200, hi), "n": _log(rng, 200, hi),
                "k": _log(rng, 128, hi), "p": p}
    m, n = _log(rng, 300, 4096), _log(rng, 300, 4096)
    return {"kind": kind, "m": m, "n": n, "rank": max(1, int(min(m, n) * rng.uniform(0.5, 1.0))),
            "p": p}


# --------------------------------------------------------------------------
# inputs


def _staircase(c, seed, nru=None, nrl=None, ncr=None, dmin=None, dmax=None, p=None):
    return synth.staircase_native(nru or c["nru"], nrl or c["nrl"], ncr or c["ncr"], p or c["p"],
                                  dmin or c["dmin"], dmax or c["dmax"], seed=seed)


def _matrix(c, seed):
    if c["gen"] == "random":
        return synth.random_macaulay(c["nru"], c["nrl"], c["ncr"], c["p"], c["density"], seed=seed,
                                     dup_rows=c["nrl"] // 8)
    return _staircase(c, seed)


def _images(c, seed):
    q = 2 * c["bound"] + 1
    m = _staircase(c, seed, p=q)
    v = m.vals.astype(np.int64)
    m.vals = np.where(v > c["bound"], v - q, v).astype(np.int32)  # integers in [-bound, bound]
    return [synth.image_mod(m, p) for p in synth.largest_primes_below(1 << 31, c["n"])]


def _uneven(c, seed):
    rng = np.random.default_rng(seed)
    lo, hi = math.log(c["rows_min"]), math.log(c["rows_max"])
    out = []
    for i in range(c["n"]):
        # sizes and densities are the case's own, spread over its ranges; the seed draws the
        # structure of the rows and the entries
        rows = int(math.exp(lo + (hi - lo) * (i + 0.5) / c["n"]))
        nrl = rows // 5
        ncr = int(rows * (1.5 + 1.5 * ((i * 5) % c["n"]) / c["n"])) - (rows - nrl)
        d = c["dmin"] + (c["dmax"] - c["dmin"]) * ((i * 7 + 3) % c["n"]) / c["n"]
        out.append(synth.staircase_native(rows - nrl, nrl, ncr, c["p"], d, d,
                                          seed=int(rng.integers(1 << 30))))
    return out


def _basis_rows(c, seed):
    rng = np.random.default_rng(seed)
    leads = np.sort(rng.choice(c["nc"] - 1, size=c["nr"], replace=False))[::-1]
    cols, vals, ptr = [], [], [0]
    for lead in leads:
        k = min(int(c["row_len"]), c["nc"] - 1 - int(lead))
        rest = int(lead) + 1 + rng.choice(c["nc"] - 1 - int(lead), size=k, replace=False)
        cols.append(np.concatenate([[lead], rest]))
        vals.append(np.concatenate([[1], rng.integers(1, c["p"], size=k)]))
        ptr.append(ptr[-1] + k + 1)
    return ReducedRows(np.array(ptr), np.concatenate(cols), np.concatenate(vals))


def _uniform(p, shape, g):
    """Residues in [0, p) on the GPU (p < 2^31, so int32 holds them)."""
    return torch.randint(0, p, shape, device="cuda", dtype=torch.int64, generator=g).to(torch.int32)


def _gemm_operands(c, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return (_uniform(c["p"], (c["m"], c["k"]), g), _uniform(c["p"], (c["k"], c["n"]), g),
            _uniform(c["p"], (c["m"], c["n"]), g))


def _rref_block(c, seed):
    """m x n block of rank at most ``rank``: uniform rows and, for the rest, random
    combinations of two of them, in random order."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    m, n, r, p = c["m"], c["n"], min(c["rank"], c["m"]), c["p"]
    base = _uniform(p, (r, n), g)
    if r < m:
        pick = torch.randint(0, r, (2, m - r), device="cuda", generator=g)
        f = torch.randint(1, p, (2, m - r, 1), device="cuda", dtype=torch.int64, generator=g)
        more = (base[pick[0]].long() * f[0] % p + base[pick[1]].long() * f[1] % p) % p
        base = torch.cat([base, more.to(torch.int32)])
    return base[torch.randperm(m, device="cuda", generator=g)].contiguous()


def _caps(nrl, ncr):
    """Rows and entries an answer may have: np <= nrl rows with np unit columns hold at
    most np (ncr - np + 1) entries."""
    np_ = max(0, min(nrl, ncr, (ncr + 1) // 2))
    return max(0, min(nrl, ncr)) + 1, max(1, np_ * (ncr - np_ + 1))


def _value_bytes(p):
    return 1 if p < 1 << 8 else 2 if p < 1 << 16 else 4


class _Answer:
    """The program's own arrays for one answer, as large as it can get."""

    def __init__(self, nrl, ncr, vb=4, pinned=False):
        rows, cap = _caps(nrl, ncr)
        width = {1: torch.uint8, 2: torch.int16, 4: torch.int32}[vb]
        self.ptr = torch.zeros(rows, dtype=torch.int64, pin_memory=pinned)
        self.cols = torch.zeros(cap, dtype=torch.int32, pin_memory=pinned)
        self.vals = torch.zeros(cap, dtype=width, pin_memory=pinned)

    def take(self, rows):
        """Takes over the rows of a gbgpu_rows and gives that back."""
        C.memmove(self.ptr.data_ptr(), rows.row_ptr, 8 * (rows.np + 1))
        C.memmove(self.cols.data_ptr(), rows.cols, 4 * rows.nnz)
        C.memmove(self.vals.data_ptr(), rows.vals, 4 * rows.nnz)
        _lib.load().gbgpu_rows_free(C.byref(rows))
        return self.whole()

    def whole(self):
        return {"row_ptr": self.ptr, "cols": self.cols, "vals": self.vals}


def _csr(m):
    return _lib.Csr(m.p, m.laopt, m.nr, m.ncl, m.ncr, m.row_ptr.ctypes.data, m.cols.ctypes.data,
                    m.vals.ctypes.data)


def _answer_of(m, **kw):
    return _Answer(m.nr - m.ncl, m.ncr, **kw)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "reduce":
        m = _matrix(case, seed)
        return {"case": case, "mat": m, "csr": _csr(m), "out": _answer_of(m)}
    if kind == "plan":
        m = _staircase(case, seed)
        vb = _value_bytes(m.p)
        return {"case": case, "plan": la.Plan(m), "vb": vb,
                "out": _answer_of(m, vb=vb, pinned=True)}
    if kind in ("images", "batch"):
        ms = _images(case, seed) if kind == "images" else _uneven(case, seed)
        return {"case": case, "mats": ms, "csrs": (_lib.Csr * len(ms))(*[_csr(m) for m in ms]),
                "outs": [_answer_of(m) for m in ms]}
    if kind == "interreduce":
        return {"case": case, "rows": _basis_rows(case, seed),
                "out": _Answer(case["nr"], case["nc"])}
    if kind == "gemm":
        return {"case": case, "abd": _gemm_operands(case, seed)}
    return {"case": case, "block": _rref_block(case, seed),
            "work": torch.empty((case["m"], case["n"]), dtype=torch.int32, device="cuda"),
            "piv": torch.zeros(min(case["m"], case["n"]), dtype=torch.int32, device="cuda")}


def run(state):
    case, lib = state["case"], _lib.load()
    kind = case["kind"]
    host = _lib.Options(_lib.FORM_AUTO, 0, 1, 0, None)
    if kind == "reduce":
        rows = _lib.Rows()
        _lib.check(lib.gbgpu_reduce(C.byref(state["csr"]), C.byref(host), C.byref(rows)))
        return state["out"].take(rows)
    if kind == "plan":
        out, np_, nnz = state["out"], C.c_int32(), C.c_int64()
        _lib.check(lib.gbgpu_plan_run_into_v(
            state["plan"]._h, out.ptr.data_ptr(), out.cols.data_ptr(), out.vals.data_ptr(),
            state["vb"], out.ptr.numel(), out.cols.numel(), C.byref(np_), C.byref(nnz)))
        return {**out.whole(), "np": np_.value, "nnz": nnz.value}
    if kind in ("images", "batch"):
        n = len(state["mats"])
        rows, status = (_lib.Rows * n)(), (C.c_int32 * n)()
        _lib.check(lib.gbgpu_reduce_batch(n, state["csrs"], C.byref(host), rows,
                                          C.cast(status, C.POINTER(C.c_int32))))
        for st in status:
            _lib.check(st)
        return [o.take(r) for o, r in zip(state["outs"], rows)]
    if kind == "interreduce":
        r, rows = state["rows"], _lib.Rows()
        _lib.check(lib.gbgpu_interreduce(case["p"], r.np, case["nc"], r.row_ptr.ctypes.data,
                                         r.cols.ctypes.data, r.vals.ctypes.data, C.byref(host),
                                         C.byref(rows)))
        return state["out"].take(rows)
    opt = _lib.Options(_lib.FORM_AUTO, torch.cuda.current_device(), 1, 0,
                       torch.cuda.current_stream().cuda_stream)
    if kind == "gemm":
        A, B, D = state["abd"]
        _lib.check(lib.gbgpu_dense_submul(case["p"], case["m"], case["n"], case["k"], A.data_ptr(),
                                          case["k"], B.data_ptr(), case["n"], D.data_ptr(),
                                          case["n"], C.byref(opt)))
        return D
    # the program keeps its block and reduces a copy
    work, piv, rank = state["work"], state["piv"], C.c_int32()
    work.copy_(state["block"])
    _lib.check(lib.gbgpu_dense_rref(case["p"], case["m"], case["n"], work.data_ptr(), case["n"],
                                    C.byref(rank), piv.data_ptr(), C.byref(opt)))
    return {"rows": work, "piv": piv, "rank": rank.value}


# --------------------------------------------------------------------------
# what a pass cannot do without


def _reduction_work(nru, nrl, ncr, density, p, entry_bytes):
    """Input entries read and answer entries written once.  Modular multiply-adds
    (two operations each): every row to reduce takes one sparse pivot row per left
    column it has entries in or meets (a band of half its columns' share), then its
    dense right part is brought to reduced echelon form."""
    nc = nru + ncr
    nnz = (nru + nrl) * density * nc
    rank = min(nrl, ncr)
    out = rank * max(1, ncr - rank)
    schur = nrl * (nru / 2) * density * nc
    echelon = rank * rank * max(1, ncr - rank / 2)
    return {"bytes": entry_bytes * (nnz + out), "flops": 2.0 * (schur + echelon)}


def work(case):
    kind, p = case["kind"], case.get("p", P31)
    if kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 4.0 * (m * k + k * n + 2 * m * n), "flops": 2.0 * m * n * k}
    if kind == "rref":
        m, n, r = case["m"], case["n"], case["rank"]
        return {"bytes": 8.0 * m * n, "flops": 2.0 * r * m * (n - r / 2)}
    if kind == "interreduce":
        nnz = case["nr"] * case["row_len"]
        out = case["nr"] * max(1, case["nc"] - case["nr"])
        return {"bytes": 8.0 * (nnz + out), "flops": 2.0 * case["nr"] * nnz}
    if kind == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        for m in _uneven({**case, "dmin": 1e-9, "dmax": 1e-9}, 1):
            w = _reduction_work(m.ncl, m.nr - m.ncl, m.ncr, (case["dmin"] + case["dmax"]) / 2, p, 8)
            total = {k: total[k] + w[k] for k in total}
        return total
    density = case.get("density") or (case["dmin"] + case["dmax"]) / 2
    w = _reduction_work(case["nru"], case["nrl"], case["ncr"], density, p,
                        4 + _value_bytes(p) if kind == "plan" else 8)
    times = case["n"] if kind == "images" else 1
    return {k: v * times for k, v in w.items()}


# --------------------------------------------------------------------------
# the answers in plain 64-bit arithmetic


def _rref64(M, p):
    """Reduced row echelon form of an int64 matrix on the GPU (p < 2^31), with its
    pivot columns."""
    M = M.clone()
    rank, piv = 0, []
    for c in range(M.shape[1]):
        if rank == M.shape[0]:
            break
        nz = torch.nonzero(M[rank:, c])
        if nz.numel() == 0:
            continue
        i = rank + int(nz[0])
        if i != rank:
            M[[rank, i]] = M[[i, rank]]
        M[rank, c:] = M[rank, c:] * pow(int(M[rank, c]), p - 2, p) % p
        f = M[:, c].clone()
        f[rank] = 0
        M[:, c:] = (M[:, c:] - f[:, None] * M[rank, c:][None, :] % p) % p
        piv.append(c)
        rank += 1
    return M, piv


def _dense(row_ptr, cols, vals, nc):
    M = torch.zeros((len(row_ptr) - 1, nc), dtype=torch.int64)
    row = torch.from_numpy(np.repeat(np.arange(len(row_ptr) - 1), np.diff(row_ptr)))
    M[row, torch.from_numpy(cols.astype(np.int64))] = torch.from_numpy(vals.astype(np.int64))
    return M.cuda()


def _sparse_rows(M, nrl, ncr):
    nz = (M != 0).cpu().numpy()
    out = _Answer(nrl, ncr)
    ptr = np.concatenate([[0], np.cumsum(nz.sum(axis=1))])
    out.ptr[: len(ptr)] = torch.from_numpy(ptr)
    out.cols[: ptr[-1]] = torch.from_numpy(np.nonzero(nz)[1])
    out.vals[: ptr[-1]] = torch.from_numpy(M.cpu().numpy()[nz])
    return out.whole()


def _exact_reduce(m):
    M, piv = _rref64(_dense(m.row_ptr, m.cols, m.vals, m.nc), m.p)
    first = next((k for k, c in enumerate(piv) if c >= m.ncl), len(piv))
    return _sparse_rows(M[first: len(piv)].flip(0), m.nr - m.ncl, m.ncr)


def exact(case, seed):
    kind = case["kind"]
    if kind == "gemm":
        # 16-bit halves of A and of B: every sum of products is a whole number below 2^53
        p = case["p"]
        A, B, D = _gemm_operands(case, seed)
        A, B, D = A.long(), B.long(), D.long()
        out = D
        for i in (0, 16):
            for j in (0, 16):
                if (p - 1) >> i == 0 or (p - 1) >> j == 0:
                    continue
                S = ((A >> i) & 0xFFFF).double() @ ((B >> j) & 0xFFFF).double()
                out = (out - S.long() % p * pow(2, i + j, p)) % p
        return out.to(torch.int32)
    if kind == "reduce" and case["gen"] == "random":
        return _exact_reduce(_matrix(case, seed))
    if kind == "images":
        return [_exact_reduce(m) for m in _images(case, seed)]
    if kind == "interreduce":
        r = _basis_rows(case, seed)
        M, piv = _rref64(_dense(r.row_ptr, r.cols, r.vals, case["nc"]), case["p"])
        return _sparse_rows(M[: len(piv)], case["nr"], case["nc"])
    if kind == "rref" and case["m"] * case["n"] <= 2048 * 2048:
        M, piv = _rref64(_rref_block(case, seed).long(), case["p"])
        cols = torch.zeros(min(case["m"], case["n"]), dtype=torch.int32)
        cols[: len(piv)] = torch.tensor(piv, dtype=torch.int32)
        return {"rows": M.to(torch.int32), "piv": cols, "rank": len(piv)}
    return None
