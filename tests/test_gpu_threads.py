"""Solvers of several host threads and the memory kept between them: one thread
makes, sets up and destroys solvers while another has a graph capture open, or
repeats setups that capture their factorisation; the kept memory is returned on
request."""
import threading

import numpy as np
import pytest

import oracle
import saplibrary_b200 as sap

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def options(**kw):
    return sap.Options(performReorder=False, variableBandwidth=False, applyScaling=False, factMethod=sap.LU_UL, **kw)


def in_thread(f):
    errors = []

    def run():
        try:
            f()
        except Exception as e:  # shown by the caller
            errors.append(e)

    t = threading.Thread(target=run)
    t.start()
    return t, errors


def test_solvers_come_and_go_beside_an_open_capture():
    n, K = 2000, 8
    A = sap.BandedMatrix.from_array(sap.generate_band_host(n, K, 1.0, 1, seed=3), n, K)
    x = torch.ones(1 << 16, device="cuda")
    y = torch.zeros_like(x)

    def rounds(k):
        for _ in range(k):
            s = sap.Solver(4, options(), prec="double")
            s.setup(A)
            del s

    rounds(1)  # kernels loaded
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, capture_error_mode="thread_local"):
        y.copy_(x)
        t, errors = in_thread(lambda: rounds(3))
        t.join()
        y.mul_(3.0)
    assert not errors, errors
    g.replay()
    torch.cuda.synchronize()
    assert bool((y == 3.0).all())
    rounds(1)


@pytest.mark.parametrize("prec", ["double", "tf32"])
def test_captured_setups_beside_other_solvers(prec):
    n, K = 30011, 150
    band = sap.generate_band_host(n, K, 1.0, 1, seed=n)
    A = sap.BandedMatrix.from_array(band, n, K)
    n2, K2 = 2000, 8
    A2 = sap.BandedMatrix.from_array(sap.generate_band_host(n2, K2, 1.0, 1, seed=3), n2, K2)
    stop = threading.Event()

    def narrow():
        while not stop.is_set():
            s = sap.Solver(4, options(), prec="double")
            s.setup(A2)
            del s

    v = np.random.default_rng(1).standard_normal(n)
    vd, z = torch.tensor(v, device="cuda"), torch.empty(n, dtype=torch.float64, device="cuda")
    t, errors = in_thread(narrow)
    try:
        for P in (4, 5, 6, 7):
            s = sap.Solver(P, options(), prec=prec)
            out = []
            for _ in range(4):  # direct, captured, replayed
                s.setup(A)
                s.precond(vd, z)
                out.append(z.cpu().numpy())
            assert all(np.array_equal(o, out[0]) for o in out)
            if prec == "double":
                o = oracle.Precond(P, fact=sap.LU_UL, dtype=prec)
                assert o.setup_banded(band, n, K) == 0
                zo = o.apply(v)
                assert np.linalg.norm(out[0] - zo) / np.linalg.norm(zo) <= 1e-10
    finally:
        stop.set()
        t.join()
    assert not errors, errors


def test_threads_choose_their_sweep_schedules_side_by_side():
    # blocks above 448 rows, a layout of its own for each solver: every first
    # application times the schedules and enters the choice
    jobs = [(6011 + 97 * i, 449 + 32 * (i % 3), 2 + i % 4) for i in range(8)]
    bands = [sap.generate_band_host(n, K, 1.0, 1, seed=n) for n, K, _ in jobs]
    As = [sap.BandedMatrix.from_array(b, n, K) for b, (n, K, _) in zip(bands, jobs)]

    def apply(i, rounds, out):
        n, K, P = jobs[i]
        s = sap.Solver(P, options(), prec="tf32")
        s.setup(As[i])
        v = torch.ones(n, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        for _ in range(rounds):
            z = torch.zeros_like(v)
            torch.cuda.synchronize()
            s.precond(v, z)
            out.append(z)

    outs = [[] for _ in jobs]
    ts = [in_thread(lambda i=i: apply(i, 3, outs[i])) for i in range(len(jobs))]
    for t, errors in ts:
        t.join()
        assert not errors, errors
    for i, (n, K, P) in enumerate(jobs):
        alone = []
        apply(i, 1, alone)
        for z in outs[i]:
            assert float((z - alone[0]).norm() / alone[0].norm()) <= 1e-5


def test_kept_memory_is_returned_on_request():
    n, K = 400003, 50
    A = sap.BandedMatrix.from_array(sap.generate_band_host(n, K, 1.0, 1, seed=3), n, K)

    def use():
        s = sap.Solver(8, options(), prec="double")
        s.setup(A)

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    use()  # kernels loaded
    sap.trim_memory()
    before = free()
    use()
    assert free() < before - (64 << 20)
    sap.trim_memory()
    assert free() >= before - (32 << 20)


def test_kept_memory_is_bounded():
    ns = (300_007, 500_009, 700_001, 900_001, 1_100_009)
    As = [sap.BandedMatrix.from_array(sap.generate_band_host(n, 30, 1.0, 1, seed=n), n, 30) for n in ns]

    def use(A):
        s = sap.Solver(16, options(), prec="double")
        s.setup(A)

    use(As[0])
    sap.trim_memory()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    for A in As + As[:1]:  # 4 GB of buffers in blocks of many sizes
        use(A)
        torch.cuda.synchronize()
        assert torch.cuda.mem_get_info()[0] >= before - (2 << 30) - (64 << 20)
    sap.trim_memory()
