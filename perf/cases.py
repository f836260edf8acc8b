"""What the framework's speed is measured on: calls that a program which uses it makes, through
``lela_b200.CudaModule``, at the sizes of the benchmark, the tests and the workloads they stand for.

``listed()`` names them; ``draw(rng)`` gives others of the same ranges.  Every input is drawn from
the seed on the GPU (or, for the sparse F4 matrices, by ``lela_b200.gen``); a program keeps one
module, its stream and its result buffers, and so do the states here.  The routines that work in
place get a fresh copy of their input in each pass, as a caller that still needs the input makes.
All outputs are residues, bits, ranks and determinants: whole numbers with one right value."""
import math
import types

import numpy as np
import torch

from lela_b200 import CudaModule, gen

P8, P16, P31 = 251, 65521, 2147483647  # one, two and four 8-bit limbs

_kept = {}


def _module():
    """The program's one module, on a stream of its own."""
    if not _kept:
        _kept["stream"] = torch.cuda.Stream()
        _kept["cm"] = CudaModule(0)
        _kept["cm"].set_stream(_kept["stream"])
    return _kept["cm"], _kept["stream"]


def listed():
    return [
        # one small product: the unit in which block algorithms call gemm; launches count
        dict(name="gemm_512", op="gemm", m=512, n=512, k=512, p=P16, b=0, elem="u32"),
        # the headline product, as a trailing update C <- C + A B
        dict(name="gemm_8192", op="gemm", m=8192, n=8192, k=8192, p=P16, b=1, elem="u32"),
        # the largest word-size modulus, as modular (multi-prime) methods use it
        dict(name="gemm_4096_p31", op="gemm", m=4096, n=4096, k=4096, p=P31, b=0, elem="u32"),
        # Modular<uint8> matrices of odd sizes
        dict(name="gemm_u8_odd", op="gemm", m=3001, n=2777, k=4099, p=P8, b=1, elem="u8"),
        # many right-hand sides against one triangular matrix
        dict(name="trsm_8192x4096", op="trsm", m=8192, n=4096, p=P16, upper=False, unit=True),
        # rank, row space and determinant of a dense matrix
        dict(name="echelon_4096", op="echelon", m=4096, n=4096, r=4096, p=P16, reduced=False),
        # a null space by the reduced form: ragged, rank-deficient, a word-size modulus
        dict(name="echelon_reduced_1500x2100", op="echelon", m=1500, n=2100, r=1207, p=P31, reduced=True),
        # one step of an F4 Groebner basis computation, matrix and result on the device
        dict(name="fl_20000", op="fl", m=20000, density=0.025, p=P16, host=False),
        # an early step of such a computation from a host program: CSR rows and result in host memory
        dict(name="fl_2000_host", op="fl", m=2000, density=0.03, p=P16, host=True),
        # GF(2): the product, and the form of a matrix of planted rank
        dict(name="gf2_gemm_16384", op="gf2_gemm", m=16384, n=16384, k=16384, b=1),
        dict(name="gf2_echelon_32768", op="gf2_echelon", m=32768, n=32768, r=30000),
        # many independent dense blocks of uneven sizes and moduli in one call
        dict(name="batch_48", op="batch", count=48, low=64, high=2048),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    op = rng.choice(["gemm", "gemm", "trsm", "echelon", "echelon", "fl", "gf2_gemm", "gf2_echelon", "batch"])
    p = rng.choice([P8, P16, P31])
    if op == "gemm":
        hi = 4096 if p == P31 else 8192
        elem = "u8" if p == P8 and rng.random() < 0.5 else "u32"
        return dict(op=op, m=_log(rng, 100, hi), n=_log(rng, 100, hi), k=_log(rng, 100, hi), p=p,
                    b=rng.choice([0, 1]), elem=elem)
    if op == "trsm":
        return dict(op=op, m=_log(rng, 200, 8192 if p != P31 else 4096), n=_log(rng, 100, 4096), p=p,
                    upper=rng.random() < 0.5, unit=rng.random() < 0.5)
    if op == "echelon":
        m, n = _log(rng, 200, 4096), _log(rng, 200, 4096)
        full = min(m, n)
        r = full if rng.random() < 0.5 else rng.randint(full // 2, full)
        return dict(op=op, m=m, n=n, r=r, p=p, reduced=rng.random() < 0.5)
    if op == "fl":
        host = rng.random() < 0.5
        return dict(op=op, m=_log(rng, 500, 4000 if host else 20000), density=round(rng.uniform(0.01, 0.03), 4),
                    p=rng.choice([P16, P16, P31]), host=host)
    if op == "gf2_gemm":
        return dict(op=op, m=_log(rng, 500, 16384), n=_log(rng, 500, 16384), k=_log(rng, 500, 16384),
                    b=rng.choice([0, 1]))
    if op == "gf2_echelon":
        m, n = _log(rng, 1000, 32768), _log(rng, 1000, 32768)
        return dict(op=op, m=m, n=n, r=rng.randint(min(m, n) // 2, min(m, n)))
    lo = _log(rng, 64, 256)
    return dict(op=op, count=rng.randint(8, 48), low=lo, high=_log(rng, 2 * lo, 2048))


# ------------------------------------------------------------------ inputs


def _uniform(g, m, n, p, dtype=torch.int32):
    return torch.randint(0, p, (m, n), generator=g, device="cuda", dtype=torch.int64).to(dtype)


def _matmul_mod(A, B, p):
    """A B mod p for integer matrices with entries in [0, p), exactly, in float64: 16-bit halves
    (8-bit where one product is already 32 bits wide) and at most 2^20 terms."""
    A, B = A.to(torch.int64), B.to(torch.int64)
    if p <= 1 << 16:
        return (A.double() @ B.double()).to(torch.int64) % p
    a1, a0, b1, b0 = ((x >> s & 65535).double() for x in (A, B) for s in (16, 0))
    hi = (a1 @ b1).to(torch.int64) % p
    mid = ((a1 @ b0).to(torch.int64) + (a0 @ b1).to(torch.int64)) % p
    lo = (a0 @ b0).to(torch.int64) % p
    return ((hi * 65536 % p + mid) % p * 65536 % p + lo) % p


def _planted(g, m, n, r, p):
    """m x n over Z/p, uniform, or of rank r as a product of two uniform factors."""
    if r >= min(m, n):
        return _uniform(g, m, n, p)
    return _matmul_mod(_uniform(g, m, r, p), _uniform(g, r, n, p), p).to(torch.int32)


def _pack(bits):
    """0/1 rows (uint8, m x n) as 64-bit words: bit j of word w is column 64 w + j."""
    m, n = bits.shape
    full = torch.zeros((m, -(-n // 64) * 64), dtype=torch.uint8, device="cuda")
    full[:, :n] = bits
    shift = torch.arange(8, dtype=torch.uint8, device="cuda")
    octets = (full.view(m, -1, 8) << shift).sum(2, dtype=torch.uint8)
    return octets.view(torch.int64)


def _unpack(words, n):
    shift = torch.arange(8, dtype=torch.uint8, device="cuda")
    return (words.contiguous().view(torch.uint8)[:, :, None] >> shift & 1).view(words.shape[0], -1)[:, :n]


def _bits(g, m, n):
    return torch.randint(0, 2, (m, n), generator=g, device="cuda", dtype=torch.uint8)


def _planted_bits(g, m, n, r):
    """Packed m x n bits of rank r (full: Bernoulli(1/2)), as a product of two random factors."""
    if r >= min(m, n):
        return _pack(_bits(g, m, n))
    up = lambda x: -(-x // 32) * 32  # noqa: E731
    F = torch.zeros((up(r), up(n)), dtype=torch.int8, device="cuda")
    F[:r, :n] = _bits(g, r, n)
    out = []
    for i in range(0, m, 8192):
        rows = min(8192, m - i)
        E = torch.zeros((max(32, up(rows)), up(r)), dtype=torch.int8, device="cuda")
        E[:rows, :r] = _bits(g, rows, r)
        out.append(_pack((torch._int_mm(E, F)[:rows, :n] & 1).to(torch.uint8)))
    return torch.cat(out)


def _blocks(case, seed):
    """(rows, columns, modulus) of the batch's blocks: the sizes are part of the workload, not of the seed."""
    r = np.random.Generator(np.random.PCG64(case["count"] * 7919 + case["low"]))
    size = np.exp(r.uniform(math.log(case["low"]), math.log(case["high"]), size=(case["count"], 2)))
    mod = r.integers(0, 3, size=case["count"])
    return [(int(a), int(b), (P8, P16, P31)[t]) for (a, b), t in zip(size, mod)]


def prepare(case, seed):
    cm, stream = _module()
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    s = types.SimpleNamespace(case=case, cm=cm, stream=stream, p=case.get("p"))
    op = case["op"]
    if op == "gemm":
        dtype = torch.uint8 if case["elem"] == "u8" else torch.int32
        m, n, k, p = case["m"], case["n"], case["k"], case["p"]
        s.A, s.B, s.C = _uniform(g, m, k, p, dtype), _uniform(g, k, n, p, dtype), _uniform(g, m, n, p, dtype)
        s.out = torch.empty_like(s.C)
    elif op == "trsm":
        m, p = case["m"], case["p"]
        A = _uniform(g, m, m, p)
        A = torch.triu(A, 1) if case["upper"] else torch.tril(A, -1)
        d = torch.ones(m, dtype=torch.int32, device="cuda") if case["unit"] else 1 + _uniform(g, 1, m, p - 1)[0]
        s.A = A + torch.diag(d)
        s.B = _uniform(g, m, case["n"], p)
        s.out = torch.empty_like(s.B)
    elif op == "echelon":
        s.A = _planted(g, case["m"], case["n"], case["r"], case["p"])
        s.out = torch.empty_like(s.A)
    elif op == "fl":
        s.X = gen.f4_matrix_fast(seed, case["m"], case["p"], density=case["density"])
        s.out = np.empty((s.X.m, s.X.n), dtype=np.uint32)
        if not case["host"]:
            X, dev = s.X, lambda a, t: torch.from_numpy(a.view(t)).cuda()  # noqa: E731
            s.X = types.SimpleNamespace(m=X.m, n=X.n, rowptr=dev(X.rowptr, np.int64),
                                        colidx=dev(X.colidx, np.int32), vals=dev(X.vals, np.int32))
            s.out = torch.empty((X.m, X.n), dtype=torch.int32, device="cuda")
    elif op == "gf2_gemm":
        m, n, k = case["m"], case["n"], case["k"]
        s.A, s.B, s.C = _pack(_bits(g, m, k)), _pack(_bits(g, k, n)), _pack(_bits(g, m, n))
        s.out = torch.empty_like(s.C)
    elif op == "gf2_echelon":
        s.A = _planted_bits(g, case["m"], case["n"], case["r"])
        s.out = torch.empty_like(s.A)
    else:
        shapes = _blocks(case, seed)
        s.ps = [p for _, _, p in shapes]
        s.A = torch.cat([_uniform(g, m, n, p).view(-1) for m, n, p in shapes])  # one copy a pass
        s.out = torch.empty_like(s.A)
        s.mats = [x.view(m, n) for x, (m, n, _) in zip(s.out.split([m * n for m, n, _ in shapes]), shapes)]
    torch.cuda.synchronize()
    return s


def run(s):
    op, case, cm, p = s.case["op"], s.case, s.cm, s.p
    if op == "fl":
        R, rank, det = cm.fl_echelonize(p, s.X, R=s.out)
        return [R, rank, det]
    with torch.cuda.stream(s.stream):
        if op in ("gemm", "gf2_gemm"):
            if case["b"]:
                s.out.copy_(s.C)
            if op == "gemm":
                return cm.gemm(p, 1, s.A, s.B, case["b"], s.out)
            return cm.gemm_gf2(s.A, s.B, s.out, case["n"], case["k"], 1, case["b"])
        s.out.copy_(s.B if op == "trsm" else s.A)
        if op == "trsm":
            return cm.trsm(p, 1, s.A, s.out, case["upper"], case["unit"])
        if op == "echelon":
            return list(cm.echelonize(p, s.out, reduced=case["reduced"]))
        if op == "gf2_echelon":
            return list(cm.echelonize_gf2(s.out, case["n"]))
        ranks, dets, status = cm.echelonize_batch(s.mats, s.ps)
        return [s.out, torch.tensor([ranks, dets, status])]


def _echelon_ops(m, n, r, reduced):
    """Multiply-adds of an elimination of rank r: each pivot updates the rows below (and above) it."""
    return sum((m - i - 1 + (i if reduced else 0)) * (n - i) for i in range(r))


def work(case):
    """Bytes: inputs once, outputs once.  Operations: multiply-adds of the 8-bit limb products (bits
    for GF(2)), two each, which is what the tensor cores can be asked for."""
    op = case["op"]
    limbs2 = lambda p: (1 if p <= 256 else 2 if p <= 65536 else 4) ** 2  # noqa: E731
    if op == "gemm":
        m, n, k, e = case["m"], case["n"], case["k"], 1 if case["elem"] == "u8" else 4
        return {"bytes": e * (m * k + k * n + (1 + 2 * case["b"]) * m * n),
                "flops": 2 * limbs2(case["p"]) * m * n * k}
    if op == "trsm":
        m, n = case["m"], case["n"]
        return {"bytes": 4 * (m * m // 2 + 2 * m * n), "flops": limbs2(case["p"]) * m * m * n}
    if op == "echelon":
        m, n = case["m"], case["n"]
        return {"bytes": 8 * m * n,
                "flops": 2 * limbs2(case["p"]) * _echelon_ops(m, n, case["r"], case["reduced"])}
    if op == "fl":
        m, n = case["m"], int(1.2 * case["m"])
        # the pivot block's solve and the Schur complement on the stored entries (three quarters of
        # the rows are pivots, the columns left over as many as n less those), D's form dense
        piv, rest, nnz = 3 * m // 4, n - 3 * m // 4, case["density"] * n * m
        d = m - piv
        return {"bytes": 8 * nnz + 4 * m * n,
                "flops": 2 * limbs2(case["p"]) * (nnz / 4 * rest + _echelon_ops(d, rest, d, True))}
    if op == "gf2_gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": (m * k + k * n + (1 + 2 * case["b"]) * m * n) // 8, "flops": 2 * m * n * k}
    if op == "gf2_echelon":
        m, n = case["m"], case["n"]
        return {"bytes": 2 * m * n // 8, "flops": 2 * _echelon_ops(m, n, case["r"], False)}
    b = _blocks(case, 0)
    return {"bytes": sum(8 * m * n for m, n, _ in b),
            "flops": sum(2 * limbs2(p) * _echelon_ops(m, n, min(m, n), False) for m, n, p in b)}


# ------------------------------------------------------------------- exact


def _eliminate(A, p, reduced=False, unit=False):
    """Row-echelon form of A (int64) mod the prime p by elementary row operations, the pivot being the
    first nonzero at or below the current row: (form, rank, product of the pivots)."""
    A, (m, n), i, det = A.clone(), A.shape, 0, 1
    for c in range(n):
        if i == m:
            break
        nz = torch.nonzero(A[i:, c])
        if not len(nz):
            continue
        q = i + int(nz[0])
        if q != i:
            A[[i, q]] = A[[q, i]]
        x = int(A[i, c])
        det = det * x % p
        inv = pow(x, -1, p)
        if unit:
            A[i] = A[i] * inv % p
            inv = 1
        f = A[:, c] * inv % p
        f[i] = 0
        if not reduced:
            f[:i] = 0
        A[:, c:] = (A[:, c:] + (p - f)[:, None] % p * A[i, c:] % p) % p
        i += 1
    return A, i, det % p


def exact(case, seed):
    op = case["op"]
    if op == "fl" and case["m"] > 2500 or op == "gf2_echelon" and min(case["m"], case["n"]) > 4096:
        return None
    if op == "echelon" and case["m"] * case["n"] * case["r"] > 3e10 or op == "batch" and case["high"] > 1000:
        return None
    s = prepare(case, seed)
    p = s.p
    if op == "gemm":
        out = _matmul_mod(s.A, s.B, p)
        return (out + case["b"] * s.C.to(torch.int64)) % p if case["b"] else out
    if op == "gf2_gemm":
        A, B = _unpack(s.A, case["k"]).double(), _unpack(s.B, case["n"]).double()
        out = torch.cat([(rows @ B).to(torch.int64) & 1 for rows in A.split(4096)]).to(torch.uint8)
        return _pack(out) ^ s.C if case["b"] else _pack(out)
    if op == "trsm":
        X, A = s.B.to(torch.int64), s.A.to(torch.int64)
        m, w = case["m"], 64
        starts = list(range(0, m, w))
        inv = [pow(int(d), -1, p) for d in torch.diagonal(A)]
        for a in reversed(starts) if case["upper"] else starts:
            z = min(m, a + w)
            rows = range(z - 1, a - 1, -1) if case["upper"] else range(a, z)
            done = slice(z, m) if case["upper"] else slice(0, a)
            X[a:z] = (X[a:z] + p - _matmul_mod(A[a:z, done], X[done], p)) % p if len(X[done]) else X[a:z]
            for i in rows:
                X[i] = X[i] * inv[i] % p
                rest = slice(a, i) if case["upper"] else slice(i + 1, z)
                X[rest] = (X[rest] + (p - A[rest, i])[:, None] % p * X[i] % p) % p
        return X
    if op == "echelon":
        return list(_eliminate(s.A.to(torch.int64), p, case["reduced"]))
    if op == "gf2_echelon":
        E, r, _ = _eliminate(_unpack(s.A, case["n"]).to(torch.int64), 2)
        return [_pack(E.to(torch.uint8)), r]
    if op == "batch":
        out = [_eliminate(x.to(torch.int64).view(m, n), q)
               for x, (m, n, q) in zip(s.A.split([m * n for m, n, _ in _blocks(case, seed)]), _blocks(case, seed))]
        return [torch.cat([E.view(-1) for E, _, _ in out]),
                torch.tensor([[r for _, r, _ in out], [d for _, _, d in out], [0] * len(out)])]
    X = s.X
    if case["host"]:
        D = torch.from_numpy(X.to_dense().astype(np.int64)).cuda()
    else:
        D = torch.zeros((X.m, X.n), dtype=torch.int64, device="cuda")
        rows = torch.repeat_interleave(torch.arange(X.m, device="cuda"), X.rowptr.diff())
        D[rows, X.colidx.long()] = X.vals.long()
    E, r, _ = _eliminate(D, p, True, True)
    return [E, r, None]
