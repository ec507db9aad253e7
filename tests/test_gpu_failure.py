"""Failure paths without a GPU fault: device-memory exhaustion is injected on
the host (sl1x1_debug_fail_alloc) at each growth of a library-owned buffer in
turn, after sl1x1_finalize has dropped them all. Every call must either
complete with a correct solution (the sliced-product scratch and the solve's
block inverses are optional: the FP64 DMMA update and the substitution solves
take over) or return INFO = -10002 (-10000 - cudaErrorMemoryAllocation); the
next call, with the hook off, must be correct again. No kernel is launched on
a missing buffer, so nothing here can fault the device.
"""
import numpy as np
import pytest

from lu_helpers import RESID_THRESH, system

pytestmark = pytest.mark.gpu
ENOMEM_INFO = -10002


@pytest.fixture(scope="module")
def ctx(sl, gpu_required):
    assert sl.lib().sl1x1_device_ok() == 1
    return sl.blacs_gridinit(1, 1)


def _pdgesv(sl, ctx, A0, B0, nb):
    n, nrhs = A0.shape[0], B0.shape[1]
    A = np.asfortranarray(A0.copy())
    X = np.asfortranarray(B0.copy())
    desca = np.array([1, ctx, n, n, nb, nb, 0, 0, n], np.int32)
    descb = np.array([1, ctx, n, nrhs, nb, nb, 0, 0, n], np.int32)
    ipiv = np.zeros(n + nb, np.int32)
    return sl.pdgesv(n, nrhs, A, 1, 1, desca, ipiv, X, 1, 1, descb), X


def test_pdgesv_exhaustion_at_each_growth(sl, orc, ctx):
    n, nrhs, nb = 600, 3, 64
    A0, B0 = system(orc, n, nrhs)
    L = sl.lib()
    failed = fell_back = 0
    try:
        for k in range(64):
            L.sl1x1_finalize()
            L.sl1x1_debug_fail_alloc(k)
            info, X = _pdgesv(sl, ctx, A0, B0, nb)
            fired = L.sl1x1_debug_fail_alloc(-1) < 0
            if not fired:
                assert info == 0
                break  # k is past the last growth of the call
            if info == 0:
                fell_back += 1
                assert orc.sresid(A0, B0, X) < RESID_THRESH
            else:
                assert info == ENOMEM_INFO
                failed += 1
            info, X = _pdgesv(sl, ctx, A0, B0, nb)
            assert info == 0
            assert orc.sresid(A0, B0, X) < RESID_THRESH
        else:
            pytest.fail("the hook still fired after 64 growths")
    finally:
        L.sl1x1_debug_fail_alloc(-1)
    assert failed >= 3 and fell_back >= 1, (failed, fell_back)


def test_mixed_exhaustion_at_each_growth(sl, orc, ctx):
    import torch

    n, nrhs = 1024, 1
    A0, B0 = system(orc, n, nrhs)
    L = sl.lib()
    dev = torch.device("cuda", 0)

    def run():
        dA = torch.from_numpy(np.ascontiguousarray(A0.T)).to(dev)
        dB = torch.from_numpy(np.ascontiguousarray(B0.T)).to(dev)
        dX = torch.zeros_like(dB)
        piv = torch.zeros(n, dtype=torch.int32, device=dev)
        info, _, _ = sl.dgesv_ir_dev(n, nrhs, dA.data_ptr(), n, piv.data_ptr(), dB.data_ptr(), n,
                                     dX.data_ptr(), n, fmt="bf16x3", nb=256)
        torch.cuda.synchronize()
        return info, np.asfortranarray(dX.cpu().numpy().T)

    failed = 0
    try:
        for k in range(64):
            L.sl1x1_finalize()
            L.sl1x1_debug_fail_alloc(k)
            info, X = run()
            fired = L.sl1x1_debug_fail_alloc(-1) < 0
            if not fired:
                assert info == 0
                break
            if info == 0:
                assert orc.sresid(A0, B0, X) < RESID_THRESH
            else:
                assert info == ENOMEM_INFO
                failed += 1
            info, X = run()
            assert info == 0
            assert orc.sresid(A0, B0, X) < RESID_THRESH
        else:
            pytest.fail("the hook still fired after 64 growths")
    finally:
        L.sl1x1_debug_fail_alloc(-1)
    assert failed >= 10, failed


@pytest.mark.parametrize("polls", [0, 1])
def test_panel_wait_runs_out_and_library_recovers(sl, orc, ctx, polls):
    """A device wait that gives up: with the panel's poll limit at 0 or 1, the
    cooperative panel's waits for the other CTAs' pivot candidates run out
    (no trap, no fault: each CTA records the timeout and returns, block 0
    writes identity pivots so the interchanges after it stay in range). The
    call returns INFO = -20002 (-20000 - kFlagTimeout); with the default
    limit restored the next call matches the oracle."""
    from lu_helpers import compare_ipiv

    n, nrhs, nb = 700, 2, 128  # 700 rows: six panel CTAs exchange candidates
    A0, B0 = system(orc, n, nrhs)
    L = sl.lib()
    try:
        L.sl1x1_debug_set_spin_limit(polls)
        info, X = _pdgesv(sl, ctx, A0, B0, nb)
        if polls == 0:
            assert info == -20002
        else:
            assert info in (-20002, 0)
    finally:
        L.sl1x1_debug_set_spin_limit(-1)
    A = np.asfortranarray(A0.copy())
    X = np.asfortranarray(B0.copy())
    desca = np.array([1, ctx, n, n, nb, nb, 0, 0, n], np.int32)
    descb = np.array([1, ctx, n, nrhs, nb, nb, 0, 0, n], np.int32)
    ipiv = np.zeros(n + nb, np.int32)
    assert sl.pdgesv(n, nrhs, A, 1, 1, desca, ipiv, X, 1, 1, descb) == 0
    bad, _ = compare_ipiv(orc, A0, ipiv[:n], nb)
    assert bad == 0
    assert orc.sresid(A0, B0, X) < RESID_THRESH


def _recovers(sl, orc, ctx, n, nrhs, nb, polls, repeats):
    """Calls with a poll limit of `polls` return INFO 0 or -20002 (always the latter
    with none allowed), and the next call with the default limit is right."""
    from lu_helpers import compare_ipiv, run_pdgesv

    A0, B0 = system(orc, n, nrhs)
    L = sl.lib()
    try:
        L.sl1x1_debug_set_spin_limit(polls)
        for _ in range(repeats):
            info, _ = _pdgesv(sl, ctx, A0, B0, nb)
            assert info == -20002 if polls == 0 else info in (-20002, 0)
    finally:
        L.sl1x1_debug_set_spin_limit(-1)
    info, _, ipiv, X = run_pdgesv(sl, ctx, A0, B0, nb)
    assert info == 0
    bad, _ = compare_ipiv(orc, A0, ipiv, nb)
    assert bad == 0
    assert orc.sresid(A0, B0, X) < RESID_THRESH


@pytest.mark.parametrize("polls", [0, 1, 2, 4, 16])
@pytest.mark.parametrize("n", [33, 40, 520, 1500])
def test_cluster_panel_gives_up_whole(sl, orc, ctx, n, polls):
    """Panels of 2, 4 and 16 CTAs of one cluster whose waits run out, at different
    warps and columns: every CTA stops as a whole and the cluster ends."""
    _recovers(sl, orc, ctx, n, 1, 64, polls, 8)


@pytest.mark.parametrize("polls", [0, 1, 8, 64])
def test_products_beside_a_panel_that_gives_up(sl, orc, ctx, polls):
    """With the look-ahead the products on the other stream meet the status word while
    it changes: blocks of both product kernels leave as a whole. At 2600 rows the first
    panels exchange through L2 (panel_kernel), the later ones within a cluster."""
    _recovers(sl, orc, ctx, 2600, 1, 256, polls, 4)


@pytest.mark.parametrize("n,polls", [(700, 0), (700, 2), (3000, 0), (3000, 2), (9000, 0)])
def test_mixed_panel_gives_up(sl, orc, ctx, n, polls):
    """The FP32 panel's waits (a cluster up to 8192 rows, through L2 beyond), and
    those of the FP64 factorization that it falls back to."""
    import torch

    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.rand((n, n), dtype=torch.float64, device="cuda", generator=g).sub_(0.5)
    B = torch.rand((1, n), dtype=torch.float64, device="cuda", generator=g).sub_(0.5)
    X = torch.zeros_like(B)
    piv = torch.zeros(n, dtype=torch.int32, device="cuda")

    def run():
        torch.cuda.synchronize()
        return sl.dgesv_ir_dev(n, 1, A.data_ptr(), n, piv.data_ptr(), B.data_ptr(), n, X.data_ptr(), n,
                               fmt="bf16x3", nb=256, keep_a=True)[0]

    try:
        sl.lib().sl1x1_debug_set_spin_limit(polls)
        info = run()
        assert info == -20002 if polls == 0 else info in (-20002, 0)
    finally:
        sl.lib().sl1x1_debug_set_spin_limit(-1)
    assert run() == 0
    r = (B - X @ A).abs().max()
    assert r / (A.abs().sum(0).max() * X.abs().max() * n * 2.0**-53) < RESID_THRESH


@pytest.mark.parametrize("trans", ["N", "T"])
@pytest.mark.parametrize("polls,nrhs", [(0, 1), (0, 7), (1, 1), (3, 16), (20, 3)])
def test_chained_solve_gives_up(sl, orc, ctx, trans, polls, nrhs):
    """The chained solve's waits for the blocks before (four blocks of 64 rows and a
    partial one) run out: INFO = -20002, and the next solve is right."""
    import torch

    n = 300
    g = torch.Generator(device="cuda").manual_seed(nrhs)
    A0 = torch.rand((n, n), dtype=torch.float64, device="cuda", generator=g).sub_(0.5)
    B0 = torch.rand((nrhs, n), dtype=torch.float64, device="cuda", generator=g).sub_(0.5)
    A = A0.clone()
    piv = torch.zeros(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert sl.dgetrf_dev(n, n, A.data_ptr(), n, piv.data_ptr()) == 0

    def solve():
        X = B0.clone()
        torch.cuda.synchronize()
        return sl.dgetrs_dev(trans, n, nrhs, A.data_ptr(), n, piv.data_ptr(), X.data_ptr(), n), X

    try:
        sl.lib().sl1x1_debug_set_spin_limit(polls)
        for _ in range(4):
            info, _ = solve()
            assert info == -20002 if polls == 0 else info in (-20002, 0)
    finally:
        sl.lib().sl1x1_debug_set_spin_limit(-1)
    info, X = solve()
    assert info == 0
    M = A0 if trans == "T" else A0.T  # (a torch tensor holds the transpose)
    r = (B0.T - M @ X.T).abs().max()
    assert r / (M.abs().sum(1).max() * X.abs().max() * n * 2.0**-53) < RESID_THRESH


def test_solve_that_gives_up_is_reported_by_every_caller(sl, orc, ctx):
    """PDGETRI, PDGERFS and PDGESVX make several solves in one call: a wait that gives
    up in any of them is INFO = -20002, and nothing of it is left for the next call."""
    import torch

    n, nrhs = 120, 2
    A0, B0 = system(orc, n, nrhs)
    d = np.array([1, ctx, n, n, 32, 32, 0, 0, n], np.int32)
    db = np.array([1, ctx, n, nrhs, 32, 32, 0, 0, n], np.int32)
    LU = np.asfortranarray(A0.copy())
    ipiv = np.zeros(n + 32, np.int32)
    assert sl.pdgetrf(n, n, LU, 1, 1, d, ipiv) == 0
    dev = {k: torch.from_numpy(np.ascontiguousarray(v.T)).cuda() for k, v in (("A", A0), ("LU", LU), ("B", B0))}
    piv = torch.from_numpy(ipiv[:n].copy()).cuda()
    X = {t: np.linalg.solve(A0.T if t == "T" else A0, B0) for t in "NT"}

    def getri():
        inv = np.asfortranarray(LU.copy())
        r = sl.pdgetri(n, inv, 1, 1, d, ipiv.copy())[0]
        return r, abs(inv @ A0 - np.eye(n)).max()

    def getri_dev():
        inv = dev["LU"].clone()
        torch.cuda.synchronize()
        r = sl.lib().sl1x1_dgetri_dev(n, inv.data_ptr(), n, piv.data_ptr(), None)
        return r, abs(inv.cpu().numpy().T @ A0 - np.eye(n)).max()

    def gerfs(t):
        x = torch.from_numpy(np.ascontiguousarray(X[t].T) * (1 + 1e-9)).cuda()
        torch.cuda.synchronize()
        r = sl.dgerfs_dev(t, n, nrhs, dev["A"].data_ptr(), n, dev["LU"].data_ptr(), n, piv.data_ptr(),
                          dev["B"].data_ptr(), n, x.data_ptr(), n)
        return r[0], abs(x.cpu().numpy().T - X[t]).max()

    def gesvx(t):
        a, af, b, x = (np.asfortranarray(v.copy()) for v in (A0, LU, B0, 0 * B0))
        r = sl.pdgesvx("F", t, n, nrhs, a, 1, 1, d, af, 1, 1, d, ipiv.copy(), "N", np.ones(n), np.ones(n), b, 1, 1,
                       db, x, 1, 1, db, np.zeros(nrhs), np.zeros(nrhs))
        return r["info"], abs(x - X[t]).max()

    calls = [getri, getri_dev] + [(lambda f=f, t=t: f(t)) for f in (gerfs, gesvx) for t in "NT"]
    for call in calls:
        try:
            sl.lib().sl1x1_debug_set_spin_limit(0)
            assert call()[0] == -20002
        finally:
            sl.lib().sl1x1_debug_set_spin_limit(-1)
        info, err = call()
        assert info == 0 and err < 1e-9


@pytest.mark.parametrize("polls", [0, 1, 8])
def test_grid_panel_gives_up(sl, orc, ctx, polls):
    """The panel that exchanges through L2, asked for by a row-slice setting at an order
    whose panels are one cluster otherwise."""
    sl.lib().sl1x1_set_panel_rows(64)
    try:
        _recovers(sl, orc, ctx, 700, 1, 64, polls, 4)
    finally:
        sl.lib().sl1x1_set_panel_rows(0)
