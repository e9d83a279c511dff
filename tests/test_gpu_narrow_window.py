"""The register-window kernels of the narrow path (narrow_sweeps.cuh) against
the oracle's apply at the widths where they can go wrong: half-bandwidths at
the edges of a lane's 32-row slots and of the packed rows' 16-byte padding,
the narrowest and widest of the path, partitions shorter than a window group,
ragged chunk lengths, LU_UL and LU_only tips, decoupled partitions (two chunks
per warp up to K = 16, an odd number of them included); two live solvers on the
same kernels; the kernels that read the factors in place.
Tolerances as in the other apply tests: 1e-10 (FP64), 2e-4 (FP32)."""
import numpy as np
import pytest

import oracle
import saplibrary_b200 as sap

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

TOL = {"double": 1e-10, "float": 2e-4}
SHAPES = [  # n, K, P
    (41, 1, 3), (1003, 2, 5), (2000, 8, 4), (6007, 31, 6), (6011, 32, 5), (9001, 33, 7), (12011, 64, 5),
    (12013, 65, 6), (15013, 96, 4), (16001, 97, 5), (18001, 107, 3), (150, 30, 2), (700, 5, 60),
    (18007, 108, 3),
]


@pytest.mark.parametrize("dtype", ["double", "float"])
@pytest.mark.parametrize("fact", [sap.LU_UL, sap.LU_only])
@pytest.mark.parametrize("n,K,P", SHAPES + [(20011, 121, 4), (20021, 155, 3)])
def test_window_apply_matches_oracle(n, K, P, fact, dtype):
    if dtype == "double" and K > 108:
        pytest.skip("FP64 bands this wide take the block path")
    band = sap.generate_band_host(n, K, 1.0, 1, seed=n + K)
    opts = sap.Options(performReorder=False, variableBandwidth=False, applyScaling=False, factMethod=fact)
    s = sap.Solver(P, opts, prec=dtype)
    s.setup(sap.BandedMatrix.from_array(band, n, K))
    assert s.blockLayout()[0] == 0
    o = oracle.Precond(P, fact=fact, dtype=dtype)
    assert o.setup_banded(band, n, K) == 0
    v = np.random.default_rng(K).standard_normal(n)
    z = torch.empty(n, dtype=torch.float64, device="cuda")
    s.precond(torch.tensor(v, device="cuda"), z)
    z, zo = z.cpu().numpy(), o.apply(v)
    assert np.linalg.norm(z - zo) / np.linalg.norm(zo) <= TOL[dtype]


@pytest.mark.parametrize("dtype", ["double", "float"])
@pytest.mark.parametrize("n,K,P", [(130, 1, 1), (97, 3, 1), (1009, 7, 3), (850, 16, 1), (5003, 16, 7), (5009, 17, 7), (9001, 33, 7),
                                   (16001, 97, 5), (18007, 108, 3)])
def test_decoupled_partitions_match_oracle(n, K, P, dtype):
    band = sap.generate_band_host(n, K, 1.0, 1, seed=n + K)
    s = sap.Solver(P, sap.Options(performReorder=False, variableBandwidth=False, applyScaling=False,
                                  precondType=sap.Block), prec=dtype)
    s.setup(sap.BandedMatrix.from_array(band, n, K))
    assert s.blockLayout()[0] == 0
    o = oracle.Precond(P, ptype=sap.Block, dtype=dtype)
    assert o.setup_banded(band, n, K) == 0
    v = np.random.default_rng(K).standard_normal(n)
    z, zo = band_apply(s, v), o.apply(v)
    assert np.linalg.norm(z - zo) / np.linalg.norm(zo) <= TOL[dtype]


def uneven_band(n, widths, seed):
    """Diagonally dominant CSR whose half-bandwidth changes along the matrix
    (sparse inside the band, its outermost diagonals kept)."""
    rng = np.random.default_rng(seed)
    rows, cols = [np.arange(n)], [np.arange(n)]
    for i, k in enumerate(widths):
        a, e = n * i // len(widths), n * (i + 1) // len(widths)
        for d in {1, k} | set(rng.integers(1, k + 1, 4).tolist()):
            r = np.arange(a, min(e, n - d))
            rows += [r, r + d]
            cols += [r + d, r]
    key = np.unique(np.concatenate(rows) * np.int64(n) + np.concatenate(cols))
    r, c = key // n, (key % n).astype(np.int32)
    v = rng.uniform(-1.0, 1.0, r.size)
    v[r == c] = 0.0
    v[r == c] = 1.5 * np.bincount(r, weights=np.abs(v), minlength=n)
    return np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]).astype(np.int32), c, v


@pytest.mark.parametrize("dtype", ["double", "float"])
@pytest.mark.parametrize("n,widths,P", [(8003, (3, 60, 9, 33), 8), (6001, (70, 2), 6), (5003, (12, 90, 5), 9)])
def test_partitions_of_uneven_width(n, widths, P, dtype):
    rp, ci, v = uneven_band(n, widths, n)
    s = sap.Solver(P, sap.Options(), prec=dtype)
    s.setup(sap.CsrMatrix(rp, ci, v))
    ks = s.getReorder("ks")
    assert ks.max() >= 2 * max(ks.min(), 1) and s.blockLayout()[0] == 0
    o = oracle.SparsePrecond(P, dtype=dtype)
    assert o.setup(rp, ci, v) == 0
    x = np.random.default_rng(1).standard_normal(n)
    z = torch.empty(n, dtype=torch.float64, device="cuda")
    s.precond(torch.tensor(x, device="cuda"), z)
    z, zo = z.cpu().numpy(), o.apply(x)
    assert np.linalg.norm(z - zo) / np.linalg.norm(zo) <= TOL[dtype]


def band_solver(n, K, P, dtype):
    band = sap.generate_band_host(n, K, 1.0, 1, seed=n + K)
    s = sap.Solver(P, sap.Options(performReorder=False, variableBandwidth=False, applyScaling=False,
                                  factMethod=sap.LU_UL), prec=dtype)
    s.setup(sap.BandedMatrix.from_array(band, n, K))
    return s


def band_apply(s, v):
    z = torch.empty(v.size, dtype=torch.float64, device="cuda")
    s.precond(torch.tensor(v, device="cuda"), z)
    return z.cpu().numpy()


# pairs that share a kernel and need different amounts of shared memory: the
# scan's width classes (9..16, 33..64, 65..128) and batch lengths, the reduced
# systems, the panel kernel's row counts
@pytest.mark.parametrize("dtype,one,two", [
    ("double", (200003, 16, 2), (20011, 10, 2)), ("double", (200003, 16, 2), (2003, 16, 2)),
    ("double", (90001, 60, 4), (9001, 40, 4)), ("double", (60013, 107, 3), (20011, 90, 3)),
    ("float", (60013, 120, 2), (20011, 70, 4)), ("float", (60013, 155, 3), (20021, 129, 3)),
])
def test_two_live_solvers(dtype, one, two):
    for first, second in ((one, two), (two, one)):
        n, K, P = first
        s1 = band_solver(n, K, P, dtype)
        v = np.random.default_rng(K).standard_normal(n)
        z = band_apply(s1, v)
        s2 = band_solver(*second, dtype)
        w = np.random.default_rng(second[1]).standard_normal(second[0])
        z2 = band_apply(s2, w)
        assert np.array_equal(band_apply(s1, v), z)
        assert np.array_equal(band_apply(s2, w), z2)
        o = oracle.Precond(P, fact=sap.LU_UL, dtype=dtype)
        assert o.setup_banded(sap.generate_band_host(n, K, 1.0, 1, seed=n + K), n, K) == 0
        zo = o.apply(v)
        assert np.linalg.norm(z - zo) / np.linalg.norm(zo) <= TOL[dtype]


@pytest.mark.parametrize("dtype", ["double", "float"])
@pytest.mark.parametrize("n,K,P", [(1003, 2, 5), (12011, 64, 5), (18001, 107, 3), (700, 5, 60)])
def test_factors_read_in_place(n, K, P, dtype, monkeypatch):
    # the kernels of bands without room for packed factors, first and after a
    # setup that packed them
    band = sap.generate_band_host(n, K, 1.0, 1, seed=n + K)
    A = sap.BandedMatrix.from_array(band, n, K)
    v = np.random.default_rng(K).standard_normal(n)
    for fact, kind in ((sap.LU_UL, sap.Spike), (sap.LU_only, sap.Spike), (sap.LU_UL, sap.Block)):
        o = oracle.Precond(P, fact=fact, ptype=kind, dtype=dtype)
        assert o.setup_banded(band, n, K) == 0
        zo = o.apply(v)
        s = sap.Solver(P, sap.Options(performReorder=False, variableBandwidth=False, applyScaling=False,
                                      factMethod=fact, precondType=kind), prec=dtype)
        for pack in ("0", "1", "0"):
            monkeypatch.setenv("SAPB_NARROW_PACK", pack)
            s.setup(A)
            assert np.linalg.norm(band_apply(s, v) - zo) / np.linalg.norm(zo) <= TOL[dtype]
    rp, ci, w = uneven_band(n, (K, max(1, K // 3)), n)
    s = sap.Solver(P, sap.Options(), prec=dtype)
    s.setup(sap.CsrMatrix(rp, ci, w))
    o = oracle.SparsePrecond(P, dtype=dtype)
    assert o.setup(rp, ci, w) == 0
    zo = o.apply(v)
    assert np.linalg.norm(band_apply(s, v) - zo) / np.linalg.norm(zo) <= TOL[dtype]


def test_band_that_leaves_no_room_for_packed_factors():
    n, K, P = 4_000_000, 60, 148
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    band = torch.empty(n, 2 * K + 1, dtype=torch.float64, device="cuda").uniform_(-1.0, 1.0, generator=g)
    band[:, K] = 2 * K + 1
    A = sap.BandedMatrix.from_array(band, n, K)  # 3.9 GB, as much as its factors
    del band
    v = torch.ones(n, dtype=torch.float64, device="cuda")
    opts = sap.Options(performReorder=False, variableBandwidth=False, applyScaling=False, precondType=sap.Block)

    def solve():
        s = sap.Solver(P, opts, prec="double")
        s.setup(A)
        z = torch.empty_like(v)
        s.precond(v, z)
        return z

    z = solve()
    sap.trim_memory()
    torch.cuda.empty_cache()
    torch.cuda.synchronize()
    rest = torch.empty(torch.cuda.mem_get_info()[0] - 6_500_000_000, dtype=torch.uint8, device="cuda")
    z2 = solve()
    del rest
    torch.cuda.empty_cache()
    assert float((z2 - z).norm() / z.norm()) <= 1e-10


def test_wide_setup_drops_the_packed_factors_of_a_narrow_one():
    n, K = 2_000_003, 60
    narrow = sap.BandedMatrix.from_array(sap.generate_band_host(n, K, 1.0, 1, seed=1), n, K)
    wide = sap.BandedMatrix.from_array(sap.generate_band_host(5003, 130, 1.0, 1, seed=2), 5003, 130)
    opts = sap.Options(performReorder=False, variableBandwidth=False, applyScaling=False, precondType=sap.Block)

    def free():
        sap.trim_memory()
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    s = sap.Solver(8, opts, prec="double")
    s.setup(narrow)
    held = free()
    s.setup(wide)
    assert s.blockLayout()[0] > 0
    # at least the packed factors (2 n K values) and the band (n (2 K + 1)) are gone
    assert free() - held >= 8 * n * (4 * K) - (1 << 29)
    z = band_apply(s, np.ones(5003))
    s2 = sap.Solver(8, opts, prec="double")
    s2.setup(wide)
    assert np.array_equal(band_apply(s2, np.ones(5003)), z)
    s.setup(narrow)
    z = band_apply(s, np.ones(n))
    s2.setup(narrow)
    assert np.array_equal(band_apply(s2, np.ones(n)), z)


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("variable", [False, True])
@pytest.mark.parametrize("dtype", ["double", "float"])
def test_partitions_shorter_than_two_couplings(dtype, variable, wide, monkeypatch):
    # a reordered matrix may be cut into partitions of K + 1 rows on, whose rows
    # then belong to both interfaces: both corrections arrive
    n, P = 700, 16
    rp, ci, v = uneven_band(n, (30,), 5)
    if wide:
        monkeypatch.setenv("SAPB_WIDE_MIN_K", "1")
    s = sap.Solver(P, sap.Options(performDB=False, applyScaling=False, variableBandwidth=variable), prec=dtype)
    s.setup(sap.CsrMatrix(rp, ci, v))
    assert (s.blockLayout()[0] > 0) == wide
    K = s.getStats().bandwidth
    q, r = divmod(n, P)
    assert s.getStats().numPartitions == P and K < q < 2 * K
    x = np.random.default_rng(1).standard_normal(n)
    z = [band_apply(s, x) for _ in range(20)]
    assert max(np.linalg.norm(a - z[0]) for a in z) <= 1e-2 * TOL[dtype] * np.linalg.norm(z[0])
    if variable:  # (the same matrix in another order inside the partitions)
        monkeypatch.delenv("SAPB_WIDE_MIN_K", raising=False)
        s = sap.Solver(P, sap.Options(performDB=False, applyScaling=False, variableBandwidth=False), prec=dtype)
        s.setup(sap.CsrMatrix(rp, ci, v))
    row, col = s.getReorder("finalPerm"), np.argsort(s.getReorder("finalReordering"))
    A = np.zeros((n, n))
    A[row[np.repeat(np.arange(n), np.diff(rp))], col[ci]] = v
    ends = np.concatenate([[0], np.cumsum([q + (i < r) for i in range(P)])])
    D = [A[a:e, a:e] for a, e in zip(ends[:-1], ends[1:])]
    f = np.empty(n)
    f[row] = x
    solve = lambda f: np.concatenate([np.linalg.solve(d, f[a:a + len(d)]) for d, a in zip(D, ends)])
    g, f2 = solve(f), f.copy()
    for i, e in enumerate(ends[1:-1]):
        b, t = slice(e - K, e), slice(e, e + K)
        V = np.linalg.solve(D[i], np.concatenate([np.zeros((len(D[i]) - K, K)), A[b, t]]))[-K:]
        W = np.linalg.solve(D[i + 1], np.concatenate([A[t, b], np.zeros((len(D[i + 1]) - K, K))]))[:K]
        z2 = np.linalg.solve(np.eye(K) - W @ V, g[t] - W @ g[b])
        f2[b] -= A[b, t] @ z2
        f2[t] -= A[t, b] @ (g[b] - V @ z2)
    ref = solve(f2)[col]
    assert np.linalg.norm(z[0] - ref) / np.linalg.norm(ref) <= TOL[dtype]
