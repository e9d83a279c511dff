"""Performance cases of the SPIKE-preconditioned Krylov solver: the work a
program using `saplibrary_b200` has it do, from the smallest call to the
largest, through the public classes (`Solver`, `BandedMatrix`, `CsrMatrix`,
`MVBanded`, `SpmvCusp`, `solve_batch`).

Kinds of case
* ``solve``:   `setup(A)` + `solve(spmv, b, x)` of a banded matrix; a new matrix
               every time, as in a time step with a new Jacobian.
* ``resolve``: `solve` alone with a solver that is already set up (many
               right-hand sides for one matrix).
* ``apply``:   one application of a set-up preconditioner (`precond`), for a
               program with a Krylov loop of its own.
* ``sparse``:  `setup` (DB, RCM, drop-off, second level) + `solve` of a CSR
               matrix whose rows come in a scrambled order.
* ``update``:  `update(entries)` + `solve`: the pattern kept, new values.
* ``batch``:   `solve_batch` of independent banded systems from host arrays.
* ``spmv``:    y = A x of a CSR matrix.

All right-hand sides are b = A x_true with a random x_true, formed in 64 bits,
so that x_true is the solution in 64 bits.  Bands: off-diagonals U[-1, 1]
(``dist`` 1) or N(0, 1) (``dist`` 2), diagonal ``d`` times the row sum of
their magnitudes.  Sparse: 5-point upwinded convection-diffusion stencil on a
w x len grid plus ``fill`` random entries per row within ``reach`` of the
diagonal, rows permuted at random.
"""
import math

import numpy as np
import torch

import saplibrary_b200 as sap

DEV = "cuda"


def listed():
    return [
        # the smallest call: a short narrow band, all latency and launches
        {"name": "tiny band fp64", "kind": "solve", "n": 2000, "k": 8, "parts": 4, "d": 1.0, "dist": 1,
         "prec": "double", "solver": "bicgstab2", "fact": "lu_ul", "precond": "spike"},
        # the reference's banded preset: 200,000 rows, half-bandwidth 50, plain FP64
        {"name": "preset band fp64", "kind": "solve", "n": 200000, "k": 50, "parts": 10, "d": 1.0, "dist": 1,
         "prec": "double", "solver": "bicgstab2", "fact": "lu_ul", "precond": "spike"},
        # the default factorisation method (LU only) and value type, odd sizes
        {"name": "odd band lu_only fp32", "kind": "solve", "n": 60013, "k": 37, "parts": 16, "d": 0.9, "dist": 1,
         "prec": "float", "solver": "fgmres", "fact": "lu_only", "precond": "spike"},
        # decoupled partitions (block Jacobi), many of them
        {"name": "decoupled band fp32", "kind": "solve", "n": 400000, "k": 20, "parts": 64, "d": 1.1, "dist": 1,
         "prec": "float", "solver": "fgmres", "fact": "lu_ul", "precond": "block"},
        # one matrix, right-hand side after right-hand side
        {"name": "resolve band fp64", "kind": "resolve", "n": 1000000, "k": 10, "parts": 32, "d": 1.0, "dist": 1,
         "prec": "double", "solver": "bicgstab2", "fact": "lu_ul", "precond": "spike"},
        # the preconditioner inside somebody else's Krylov loop
        {"name": "apply band fp32", "kind": "apply", "n": 200000, "k": 64, "parts": 32, "d": 1.0, "dist": 1,
         "prec": "float", "solver": "fgmres", "fact": "lu_ul", "precond": "spike"},
        # the mixed-precision wide band: 2,000,000 rows, half-bandwidth 200 (the largest)
        {"name": "wide band tf32", "kind": "solve", "n": 2000000, "k": 200, "parts": 32, "d": 0.8, "dist": 2,
         "prec": "tf32", "solver": "fgmres", "fact": "lu_ul", "precond": "spike"},
        # sparse with long-range fill: the band after reordering is thousands wide
        {"name": "sparse fill tf32_f16", "kind": "sparse", "w": 500, "len": 500, "fill": 2, "reach": 5000,
         "parts": 16, "drop": 1e-4, "prec": "tf32_f16", "solver": "fgmres"},
        # sparse on a long strip: the band after reordering is narrow, plain FP64
        {"name": "sparse strip fp64", "kind": "sparse", "w": 24, "len": 4000, "fill": 1, "reach": 30,
         "parts": 16, "drop": 0.0, "prec": "double", "solver": "bicgstab2"},
        # a nonlinear loop: the same pattern with new values, the default value type
        {"name": "sparse update fp32", "kind": "update", "w": 32, "len": 1500, "fill": 1, "reach": 40,
         "parts": 8, "drop": 0.0, "prec": "float", "solver": "fgmres"},
        # many independent systems of uneven size from host memory
        {"name": "ensemble fp32", "kind": "batch", "count": 24, "n_min": 2000, "n_max": 50000, "shape_seed": 3,
         "parts": 8, "prec": "float"},
        # the matrix-vector product of the 1,000,000-row sparse workload
        {"name": "spmv csr", "kind": "spmv", "w": 1000, "len": 1000, "fill": 2, "reach": 5000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "resolve", "apply", "sparse", "update", "batch", "spmv"])
    if kind in ("solve", "resolve", "apply"):
        prec = rng.choice(["float", "double", "float", "double", "tf32"])
        k = _log_int(rng, 4, 300 if prec == "tf32" else 150)
        n = max(_log_int(rng, 1000, 500000), 16 * k)
        n = min(n, 40000000 // (2 * k + 1))
        parts = rng.choice([2, 4, 7, 8, 10, 16, 32, 50, 64])
        # a partition keeps at most 30,000 rows: nobody leaves a long band to a few partitions
        parts = max(parts, -(-n // 30000))
        return {"kind": kind, "n": n, "k": k, "parts": parts, "d": round(rng.uniform(0.9, 1.3), 3),
                "dist": rng.choice([1, 2]), "prec": prec,
                "solver": "bicgstab2" if prec == "double" else "fgmres",
                "fact": rng.choice(["lu_ul", "lu_ul", "lu_only"]),
                "precond": rng.choice(["spike", "spike", "spike", "block"])}
    if kind in ("sparse", "update"):
        w = _log_int(rng, 10, 60)
        length = max(_log_int(rng, 200, 4000), 4 * w)
        prec = rng.choice(["float", "double"])
        return {"kind": kind, "w": w, "len": length, "fill": rng.choice([0, 1, 2]), "reach": w + rng.randrange(1, w),
                "parts": rng.choice([4, 8, 16]), "drop": 0.0, "prec": prec,
                "solver": "bicgstab2" if prec == "double" else "fgmres"}
    if kind == "batch":
        return {"kind": "batch", "count": rng.randrange(8, 33), "n_min": 1000, "n_max": _log_int(rng, 5000, 50000),
                "shape_seed": rng.randrange(1 << 20), "parts": rng.choice([4, 8, 16]), "prec": "float"}
    return {"kind": "spmv", "w": _log_int(rng, 100, 1000), "len": _log_int(rng, 100, 1000),
            "fill": rng.randrange(0, 8), "reach": rng.choice([200, 1000, 5000])}


# ---- inputs ---------------------------------------------------------------------
def _gen(seed, salt):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed * 1000003 + salt)
    return g


def _x_true(n, seed):
    return torch.randn(n, dtype=torch.float64, device=DEV, generator=_gen(seed, 1))


def _band(n, k, d, dist, seed):
    """Row-major band (n x (2k+1)) on the GPU."""
    A = torch.empty(n, 2 * k + 1, dtype=torch.float64, device=DEV)
    g = _gen(seed, 2)
    rows = max(1, (1 << 26) // (2 * k + 1))
    off = torch.arange(-k, k + 1, device=DEV)
    for a in range(0, n, rows):
        e = min(n, a + rows)
        B = A[a:e]
        if dist == 1:
            B.uniform_(-1.0, 1.0, generator=g)
        else:
            B.normal_(generator=g)
        c = torch.arange(a, e, device=DEV)[:, None] + off[None, :]
        B.masked_fill_((c < 0) | (c >= n), 0.0)
        B[:, k] = 0.0
        B[:, k] = d * B.abs().sum(dim=1)
    return A


def _band_mv(A, n, k, x):
    y = torch.empty_like(x)
    xp = torch.zeros(n + 2 * k, dtype=torch.float64, device=DEV)
    xp[k:k + n] = x
    rows = max(1, (1 << 26) // (2 * k + 1))
    for a in range(0, n, rows):
        e = min(n, a + rows)
        y[a:e] = (A[a:e] * xp[a:e + 2 * k].unfold(0, 2 * k + 1, 1)).sum(dim=1)
    return y


def _csr(case, seed):
    """(row offsets, columns, values) of the scrambled stencil + fill matrix, on the GPU."""
    w, length, fill, reach = case["w"], case["len"], case["fill"], case["reach"]
    n, conv = w * length, 0.3
    g = _gen(seed, 3)
    r = torch.arange(n, device=DEV)
    gi, gj = r // w, r % w
    rows, cols, vals = [r], [r], [torch.full((n,), 4.0 + 2.0 * conv, dtype=torch.float64, device=DEV)]
    for di, dj, v in ((0, -1, -1.0 - conv), (-1, 0, -1.0 - conv), (0, 1, -1.0), (1, 0, -1.0)):
        ok = (gi + di >= 0) & (gi + di < length) & (gj + dj >= 0) & (gj + dj < w)
        rows.append(r[ok])
        cols.append(r[ok] + di * w + dj)
        vals.append(torch.full((int(ok.sum()),), v, dtype=torch.float64, device=DEV))
    if fill:
        fr = r.repeat_interleave(fill)
        fc = fr + torch.randint(-reach, reach + 1, (n * fill,), device=DEV, generator=g)
        fv = torch.rand(n * fill, dtype=torch.float64, device=DEV, generator=g) * 0.2 - 0.1
        ok = (fc >= 0) & (fc < n)
        rows.append(fr[ok])
        cols.append(fc[ok])
        vals.append(fv[ok])
    perm = torch.randperm(n, device=DEV, generator=g)
    key = perm[torch.cat(rows)] * n + torch.cat(cols)
    val = torch.cat(vals)
    key, order = torch.sort(key, stable=True)
    first = torch.ones_like(key, dtype=torch.bool)
    first[1:] = key[1:] != key[:-1]  # of entries at one place the first stays
    key, val = key[first], val[order][first]
    rp = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    rp[1:] = torch.cumsum(torch.bincount(key // n, minlength=n), 0)
    return rp, key % n, val


def _csr_mv(rp, ci, v, x):
    """A x with each row's entries added in a fixed order (float64)."""
    n = rp.numel() - 1
    lens = rp[1:] - rp[:-1]
    y = torch.zeros(n, dtype=torch.float64, device=DEV)
    for t in range(int(lens.max())):
        rows = torch.nonzero(lens > t).flatten()
        e = rp[rows] + t
        y[rows] += v[e] * x[ci[e]]
    return y


def _csr_host(rp, ci, v):
    return rp.to(torch.int32).cpu().numpy(), ci.to(torch.int32).cpu().numpy(), v.cpu().numpy()


def _new_values(v, seed):
    return v * (1.0 + 0.02 * torch.rand(v.numel(), dtype=torch.float64, device=DEV, generator=_gen(seed, 4)))


def _batch_shapes(case):
    rng = np.random.default_rng(case["shape_seed"])
    out = []
    for _ in range(case["count"]):
        n = int(round(math.exp(rng.uniform(math.log(case["n_min"]), math.log(case["n_max"])))))
        out.append((n, int(rng.choice([8, 16, 32, 64])), float(rng.uniform(0.8, 1.2))))
    return out


_SOLVERS = {"bicgstab2": sap.BiCGStab2, "fgmres": sap.FGMRES}


def _options(case):
    sparse = case["kind"] in ("sparse", "update")
    return sap.Options(solverType=_SOLVERS[case.get("solver", "fgmres")], relTol=1e-10, maxNumIterations=400,
                       performReorder=sparse, variableBandwidth=sparse, applyScaling=sparse,
                       dropOffFraction=case.get("drop", 0.0), trackReordering=case["kind"] == "update",
                       factMethod=sap.LU_only if case.get("fact") == "lu_only" else sap.LU_UL,
                       precondType=sap.Block if case.get("precond") == "block" else sap.Spike)


def prepare(case, seed):
    kind, s = case["kind"], {"case": case}
    if kind in ("solve", "resolve", "apply"):
        n, k = case["n"], case["k"]
        band = _band(n, k, case["d"], case["dist"], seed)
        x = _x_true(n, seed)
        s["b"] = x if kind == "apply" else _band_mv(band, n, k, x)
        torch.cuda.synchronize()
        s["A"] = sap.BandedMatrix.from_array(band, n, k)
        s["spmv"] = sap.MVBanded(s["A"])
        del band
        torch.cuda.empty_cache()
    elif kind in ("sparse", "update", "spmv"):
        rp, ci, v = _csr(case, seed)
        n = rp.numel() - 1
        x = _x_true(n, seed)
        s["A"] = sap.CsrMatrix(*_csr_host(rp, ci, v))
        if kind == "spmv":
            s["b"] = x
        elif kind == "sparse":
            s["b"] = _csr_mv(rp, ci, v, x)
            s["spmv"] = sap.SpmvCusp(s["A"])
        else:
            s["entries"] = _new_values(v, seed)
            s["b"] = _csr_mv(rp, ci, s["entries"], x)
            s["spmv"] = sap.SpmvCusp(sap.CsrMatrix(*_csr_host(rp, ci, s["entries"])))
    else:
        s["bands"], s["ks"], s["bs"] = [], [], []
        for i, (n, k, d) in enumerate(_batch_shapes(case)):
            band = _band(n, k, d, 1, seed * 64 + i)
            s["bs"].append(_band_mv(band, n, k, _x_true(n, seed * 64 + i)).cpu().numpy())
            s["bands"].append(band.cpu().numpy())
            s["ks"].append(k)
        return s
    s["x"] = torch.zeros(n, dtype=torch.float64, device=DEV)
    torch.cuda.synchronize()
    if kind == "spmv":
        s["op"] = sap.SpmvCusp(s["A"])
        return s
    s["solver"] = sap.Solver(case["parts"], _options(case), prec=case["prec"])
    s["stream"] = torch.cuda.ExternalStream(s["solver"].stream())
    if kind in ("resolve", "apply", "update"):
        s["solver"].setup(s["A"])
    return s


def run(s):
    kind = s["case"]["kind"]
    if kind == "batch":
        return sap.solve_batch(s["bands"], s["ks"], s["bs"], s["case"]["parts"], _options(s["case"]),
                               prec=s["case"]["prec"])[0]
    if kind == "spmv":
        s["op"](s["b"], s["x"])
        return s["x"]
    solver = s["solver"]
    if kind == "apply":
        solver.precond(s["b"], s["x"])
        return s["x"]
    if kind in ("solve", "sparse"):
        solver.setup(s["A"])
    elif kind == "update":
        solver.update(s["entries"])
    with torch.cuda.stream(s["stream"]):  # x starts from zero, on the solver's own stream
        s["x"].zero_()
    solver.solve(s["spmv"], s["b"], s["x"])
    return s["x"]


# ---- what the path cannot do without ----------------------------------------------
def _band_work(n, k, setup, solve):
    entries = n * (2 * k + 1)
    return {"bytes": 8.0 * entries + 16.0 * n,
            "flops": (2.0 * n * k * (k + 1) if setup else 0.0) + (4.0 * n * k if solve else 0.0) + 2.0 * entries}


def work(case):
    kind = case["kind"]
    if kind in ("solve", "resolve", "apply"):
        w = _band_work(case["n"], case["k"], kind == "solve", True)
        if kind == "apply":  # the factors in the preconditioner's own type, the vectors in 64 bits
            size = 8.0 if case["prec"] == "double" else 4.0
            w["bytes"] = size * case["n"] * (2 * case["k"] + 1) + 16.0 * case["n"]
        return w
    if kind == "batch":
        ws = [_band_work(n, k, True, True) for n, k, _ in _batch_shapes(case)]
        return {"bytes": sum(w["bytes"] for w in ws), "flops": sum(w["flops"] for w in ws)}
    n = case["w"] * case["len"]
    nnz = n * (5 + case["fill"])
    w = {"bytes": 12.0 * nnz + 4.0 * n + 16.0 * n, "flops": 2.0 * nnz}
    if kind != "spmv":
        # LU of the band that any ordering leaves: the short side, or what the fill reaches
        k = max(case["w"], int(0.6 * case["reach"]) if case["fill"] else 0)
        w["flops"] += 2.0 * n * k * (k + 1) + 4.0 * n * k
    return w


def tolerance(case):
    kind = case["kind"]
    if kind == "spmv":
        return {"rel": 1e-14, "max": 1e-13}
    if kind == "apply":
        return {"rel": 1e-12} if case["prec"] == "double" else {"rel": 1e-2 if case["prec"] == "tf32" else 5e-6}
    # a solution with ||b - A x|| <= 1e-10 ||b|| (up to 2e-9 from x_true seen over drawn cases)
    return {"rel": 1e-8}


# ---- the same in 64 bits, in plain torch -------------------------------------------
def _partitions(n, k, parts):
    p = min(parts, max(1, n // max(k + 1, 2 * k)))
    q, r = divmod(n, p)
    starts = [i * q + min(i, r) for i in range(p)]
    return starts, [q + (1 if i < r else 0) for i in range(p)]


class _BlockTridiagonal:
    """The partitions' diagonal blocks of a band as block tridiagonal
    matrices (k x k blocks, identity padding), block LU kept."""

    def __init__(self, A, n, k, starts, sizes):
        self.k, self.nb = k, -(-max(sizes) // k)
        p, m = len(starts), self.nb * k
        st = torch.tensor(starts, device=DEV)[:, None]
        sz = torch.tensor(sizes, device=DEV)[:, None]
        loc = torch.arange(m, device=DEV)[None, :]
        self.rows = torch.where(loc < sz, st + loc, torch.full_like(loc, n))  # row n: padding
        self.p, self.n = p, n
        Ap = torch.cat([A, torch.zeros(1, 2 * k + 1, dtype=A.dtype, device=DEV)])
        c = torch.arange(k, device=DEV)
        self.inv, self.low, self.up = [], [], []
        prev = None
        for i in range(self.nb):
            R = Ap[self.rows[:, i * k:(i + 1) * k]]  # p x k x (2k+1)
            inside = loc[:, i * k:(i + 1) * k]

            def block(j):
                cl = j * k + c  # local columns
                off = cl[None, :] - (i * k + c)[:, None] + k
                ok = (off >= 0) & (off <= 2 * k)
                B = torch.gather(R, 2, off.clamp(0, 2 * k)[None].expand(p, k, k))
                keep = ok[None] & (inside < sz)[:, :, None] & (cl[None, :] < sz)[:, None, :]
                return torch.where(keep, B, torch.zeros_like(B))

            D = block(i)
            D = D + torch.diag_embed((inside >= sz).to(D.dtype))
            if i:
                F = block(i - 1)
                self.low.append(F @ self.inv[-1])
                D = D - self.low[-1] @ prev
            self.inv.append(torch.linalg.inv(D))
            prev = block(i + 1) if i + 1 < self.nb else None
            self.up.append(prev)

    def solve(self, f):
        """f: p x (nb k) x m."""
        k, y = self.k, []
        for i in range(self.nb):
            b = f[:, i * k:(i + 1) * k]
            y.append(b - self.low[i - 1] @ y[-1] if i else b)
        x = [None] * self.nb
        for i in reversed(range(self.nb)):
            b = y[i] - self.up[i] @ x[i + 1] if i + 1 < self.nb else y[i]
            x[i] = self.inv[i] @ b
        return torch.cat(x, dim=1)

    def to(self, v):
        return torch.cat([v, v.new_zeros(1)])[self.rows][:, :, None]

    def back(self, x):
        out = x.new_zeros(self.n + 1)
        out[self.rows] = x[:, :, 0]
        return out[:self.n]


def _apply_exact(case, seed):
    n, k = case["n"], case["k"]
    A = _band(n, k, case["d"], case["dist"], seed)
    f = _x_true(n, seed)
    starts, sizes = _partitions(n, k, case["parts"])
    T = _BlockTridiagonal(A, n, k, starts, sizes)
    g = T.back(T.solve(T.to(f)))
    if case["precond"] == "block" or len(starts) == 1:
        return g
    p = len(starts)
    rhs_v = torch.zeros(p, T.nb * k, k, dtype=torch.float64, device=DEV)
    rhs_w = torch.zeros_like(rhs_v)
    Bs, Cs = [], []
    r, c = torch.meshgrid(torch.arange(k, device=DEV), torch.arange(k, device=DEV), indexing="ij")
    for i in range(p - 1):
        s = starts[i + 1]
        off = (k + (k + c - r)).clamp(0, 2 * k)  # row s-k+r, column s+c
        B = torch.where(c <= r, A[s - k:s].gather(1, off), torch.zeros((), dtype=A.dtype, device=DEV))
        off = (k + (c - k - r)).clamp(0, 2 * k)  # row s+r, column s-k+c
        C = torch.where(c >= r, A[s:s + k].gather(1, off), torch.zeros((), dtype=A.dtype, device=DEV))
        Bs.append(B)
        Cs.append(C)
        rhs_v[i, sizes[i] - k:sizes[i]] = B
        rhs_w[i + 1, :k] = C
    V, W = T.solve(rhs_v), T.solve(rhs_w)
    f2 = f.clone()
    eye = torch.eye(k, dtype=torch.float64, device=DEV)
    for i in range(p - 1):
        s = starts[i + 1]
        v, w = V[i, sizes[i] - k:sizes[i]], W[i + 1, :k]
        z = torch.linalg.solve(eye - w @ v, g[s:s + k] - w @ g[s - k:s])
        x1 = g[s - k:s] - v @ z
        f2[s - k:s] -= Bs[i] @ z
        f2[s:s + k] -= Cs[i] @ x1
    return T.back(T.solve(T.to(f2)))


def exact(case, seed):
    kind = case["kind"]
    if kind == "apply":
        return _apply_exact(case, seed)
    if kind == "spmv":
        rp, ci, v = _csr(case, seed)
        return _csr_mv(rp, ci, v, _x_true(rp.numel() - 1, seed))
    if kind == "batch":
        return [_x_true(n, seed * 64 + i).cpu().numpy() for i, (n, _, _) in enumerate(_batch_shapes(case))]
    return _x_true(case["n"] if kind in ("solve", "resolve") else case["w"] * case["len"], seed)
