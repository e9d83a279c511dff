"""Wide bands on the block path at the sizes where its kernels change: block
sizes around the leaf (32 .. 128 rows, FP64 96), recursion levels with uneven
halves, the widest blocks of the cluster sweep and the first beyond it, corners
narrower than the block (TF32 blocks of 448 rows), few and many partitions
(clusters of 8 and of 4 CTAs), ragged last blocks.  Applies against the oracle
with the tolerances of the other apply tests (1e-10 FP64, 2e-4 FP32); the TF32
forms solve to 1e-10 with flexible GMRES.  And the banded product at the edges
of its lanes-per-row choice, with NaN outside the matrix."""
import numpy as np
import pytest

import oracle
import saplibrary_b200 as sap

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

TOL = {"double": 1e-10, "float": 2e-4}


def setup(n, K, P, prec, band, **kw):
    s = sap.Solver(P, sap.Options(performReorder=False, variableBandwidth=False, applyScaling=False,
                                  factMethod=sap.LU_UL, **kw), prec=prec)
    A = sap.BandedMatrix.from_array(band, n, K)
    s.setup(A)
    assert s.blockLayout()[0] >= K
    return A, s


@pytest.mark.parametrize("prec,n,K,P", [
    ("double", 3001, 109, 3), ("double", 4003, 128, 4), ("double", 5003, 129, 2), ("double", 7001, 200, 20),
    ("double", 6001, 320, 4), ("double", 6005, 321, 3), ("float", 4001, 157, 5), ("float", 9001, 192, 40),
    ("float", 5007, 225, 1), ("float", 8009, 448, 3), ("float", 8011, 449, 2)])
def test_block_path_apply_matches_oracle(prec, n, K, P):
    band = sap.generate_band_host(n, K, 1.0, 1, seed=n + K)
    _, s = setup(n, K, P, prec, band)
    o = oracle.Precond(P, fact=sap.LU_UL, dtype=prec)
    assert o.setup_banded(band, n, K) == 0
    v = np.random.default_rng(K).standard_normal(n)
    z = torch.empty(n, dtype=torch.float64, device="cuda")
    for _ in range(3):  # direct, captured and replayed factorisations apply alike
        s.precond(torch.tensor(v, device="cuda"), z)
        zo = o.apply(v)
        assert np.linalg.norm(z.cpu().numpy() - zo) / np.linalg.norm(zo) <= TOL[prec]
        s.setup(sap.BandedMatrix.from_array(band, n, K))


@pytest.mark.parametrize("prec,n,K,P", [("double", 9001, 20, 3), ("double", 20011, 50, 4), ("double", 24001, 96, 40),
                                        ("float", 9001, 32, 2), ("float", 20011, 70, 40), ("float", 30011, 128, 3)])
def test_blocks_of_one_leaf(prec, n, K, P, monkeypatch):
    # many block rows whose factorisation is one leaf, without a recursion whose
    # joins would order the copies of one row's corners before the next row's
    # products: direct, captured and replayed factorisations give the same bits
    monkeypatch.setenv("SAPB_WIDE_MIN_K", "16")
    band = sap.generate_band_host(n, K, 1.0, 1, seed=n + K)
    A, s = setup(n, K, P, prec, band)
    bs, nb, _ = s.blockLayout()
    assert bs <= (96 if prec == "double" else 128) and nb > 5
    o = oracle.Precond(P, fact=sap.LU_UL, dtype=prec)
    assert o.setup_banded(band, n, K) == 0
    v = np.random.default_rng(K).standard_normal(n)
    z = torch.empty(n, dtype=torch.float64, device="cuda")
    zo, first = o.apply(v), None
    for _ in range(8):
        s.precond(torch.tensor(v, device="cuda"), z)
        first = z.cpu().numpy() if first is None else first
        assert np.linalg.norm(first - zo) / np.linalg.norm(zo) <= TOL[prec]
        assert np.array_equal(z.cpu().numpy(), first)
        s.setup(A)
    # and without the second workspaces (a captured factorisation is replaced)
    monkeypatch.setenv("SAPB_FACTOR_AHEAD", "0")
    for _ in range(3):
        s.setup(A)
        s.precond(torch.tensor(v, device="cuda"), z)
        assert np.array_equal(z.cpu().numpy(), first)


@pytest.mark.parametrize("prec,n,K,P", [("double", 9001, 130, 4), ("float", 9001, 300, 3), ("tf32", 20011, 200, 19)])
def test_second_workspaces_change_no_bit(prec, n, K, P, monkeypatch):
    band = sap.generate_band_host(n, K, 1.0, 1, seed=n + K)
    A, s = setup(n, K, P, prec, band)
    assert s.blockLayout()[1] > 1
    v = torch.tensor(np.random.default_rng(K).standard_normal(n), device="cuda")
    out = []
    for ahead in ("1", "0", "0", "0", "1", "1", "1"):  # direct, captured, replayed in turn
        monkeypatch.setenv("SAPB_FACTOR_AHEAD", ahead)
        s.setup(A)
        out.append(torch.empty_like(v))
        s.precond(v, out[-1])
    assert all(torch.equal(z, out[0]) for z in out)


@pytest.mark.parametrize("prec,K", [("float", 157), ("double", 109)])
def test_cluster_sweep_of_single_block_rows(prec, K, monkeypatch):
    # one block per partition: the first exchange between the CTAs of a cluster
    # comes right after the launch, and more clusters than the chip holds start
    # in waves; every application gives the same bits
    bs = {"float": 448, "double": 320}[prec]
    P = 120
    n = P * bs - 7
    monkeypatch.setenv("SAPB_BLOCK_SIZE", str(bs))
    band = sap.generate_band_host(n, K, 1.0, 1, seed=K)
    _, s = setup(n, K, P, prec, band)
    assert s.blockLayout()[:2] == (bs, 1)
    o = oracle.Precond(P, fact=sap.LU_UL, dtype=prec)
    assert o.setup_banded(band, n, K) == 0
    v = np.random.default_rng(K).standard_normal(n)
    vd, z = torch.tensor(v, device="cuda"), torch.empty(n, dtype=torch.float64, device="cuda")
    s.precond(vd, z)
    first, zo = z.cpu().numpy(), o.apply(v)
    assert np.linalg.norm(first - zo) / np.linalg.norm(zo) <= TOL[prec]
    for _ in range(50):
        s.precond(vd, z)
        assert np.array_equal(z.cpu().numpy(), first)


@pytest.mark.parametrize("prec", ["tf32", "tf32_f16"])
@pytest.mark.parametrize("n,K,P", [(5003, 160, 2), (20011, 200, 19), (9001, 300, 3), (9007, 447, 2), (12011, 460, 3)])
def test_tf32_blocks_solve(prec, n, K, P):
    band = sap.generate_band_host(n, K, 1.0, 2, seed=n)
    A, s = setup(n, K, P, prec, band, solverType=sap.FGMRES, relTol=1e-10, maxNumIterations=100)
    xt = np.random.default_rng(1).standard_normal(n)
    x = np.zeros(n)
    assert s.solve(sap.MVBanded(A), oracle.spmv_banded(band, n, K, xt), x)
    assert np.linalg.norm(x - xt) / np.linalg.norm(xt) <= 1e-9
    assert s.getStats().numIterations <= 6


@pytest.mark.parametrize("n,K", [(1, 0), (5, 2), (300, 7), (257, 8), (1000, 15), (1001, 16), (999, 31), (130, 32),
                                 (4097, 63), (700, 64), (513, 127), (600, 128), (50, 49)])
def test_banded_product_edges(n, K):
    rng = np.random.default_rng(n + K)
    band = rng.standard_normal((n, 2 * K + 1))
    c = np.arange(n)[:, None] + np.arange(-K, K + 1)[None, :]
    inside = (c >= 0) & (c < n)
    x = rng.standard_normal(n)
    terms = np.where(inside, band * x[np.clip(c, 0, n - 1)], 0.0)
    A = sap.BandedMatrix.from_array(np.where(inside, band, np.nan).ravel(), n, K)
    y = torch.empty(n, dtype=torch.float64, device="cuda")
    sap.MVBanded(A)(torch.tensor(x, device="cuda"), y)
    bound = (2 * K + 2) * 2.0 ** -53 * np.abs(terms).sum(axis=1)  # of any order of 2K+1 products
    assert np.all(np.abs(y.cpu().numpy() - terms.sum(axis=1)) <= 2 * bound)
