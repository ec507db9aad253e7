"""GPU parity tests of the plain FP64 path through the C ABI (pdgesv_,
pdgetrf_, pdgetrs_ and the device entry points) against the CPU oracle.

Bar: IPIV identical to the oracle's except in logged near-tie columns (top-2
candidates within 1e-10 relative); scaled residuals ||A-PLU||/(||A|| max(M,N)
eps) and ||Ax-b||/(||A|| ||x|| N eps) below 16 (LIN/pdlafchk.f,
LIN/pdlaschk.f); exact INFO; untouched guard zones around every array.
"""
import json
import os

import numpy as np
import pytest

from lu_helpers import PADVAL, RESID_THRESH, compare_ipiv, guards_intact, padded, run_pdgesv, system

pytestmark = pytest.mark.gpu
GOLD = os.path.join(os.path.dirname(__file__), "golden")
@pytest.fixture(scope="module")
def ctx(sl, gpu_required):
    assert sl.lib().sl1x1_device_ok() == 1
    return sl.blacs_gridinit(1, 1)


# NB 320 exceeds the composite row-interchange table (256 pivots) and takes the
# sequential interchange kernel for the outer swaps.
SMALL = [(1, 1), (2, 1), (3, 2), (31, 4), (64, 64), (65, 64), (257, 64), (257, 256), (1000, 64),
         (1000, 256), (513, 1), (100, 2), (700, 320)]


@pytest.mark.parametrize("n,nb", SMALL)
def test_pdgesv_small_parity(sl, orc, ctx, n, nb):
    A0, B0 = system(orc, n, 3)
    info, LU, rel, X = run_pdgesv(sl, ctx, A0, B0, nb)
    assert info == 0
    bad, ties = compare_ipiv(orc, A0, rel, nb)
    assert bad == 0, f"IPIV differs outside near-ties (ties logged: {ties})"
    assert orc.fresid(LU, rel, A0) < RESID_THRESH
    assert orc.sresid(A0, B0, X) < RESID_THRESH


def test_example_known_answer_gpu(sl, orc, ctx):
    d = json.load(open(os.path.join(GOLD, "dscaex.json")))
    n = d["n"]
    A0 = np.array(d["a_colmajor"]).reshape((n, n), order="F")
    B0 = np.array(d["b"]).reshape((n, 1), order="F")
    info, LU, rel, X = run_pdgesv(sl, ctx, A0, B0, d["nb"])
    assert info == 0
    np.testing.assert_allclose(X[:, 0], d["x_exact"], rtol=1e-13)
    assert orc.sresid(A0, B0, X) < d["threshold"]


@pytest.mark.parametrize("m,n", [(4, 4), (10, 12), (17, 13), (13, 13), (23, 23), (31, 31),
                                 (57, 50)])
@pytest.mark.parametrize("nb", [2, 3, 4, 5])
def test_pdgetrf_lu_dat_shapes(sl, orc, ctx, m, n, nb):
    # LU.dat sizes with the tester's own (-1,1] generator, factor only (M != N allowed)
    A0 = orc.matgen(m, n, 100, kind=0)
    Ab = padded(A0)
    desc = np.array([1, ctx, Ab.shape[0], Ab.shape[1], nb, nb, 0, 0, Ab.shape[0]], np.int32)
    ipiv = np.zeros(Ab.shape[0] + nb, dtype=np.int32)
    info = sl.pdgetrf(m, n, Ab, 1, 1, desc, ipiv)
    assert info == 0
    assert guards_intact(Ab, 1, 1, m, n)
    mn = min(m, n)
    LU = np.asfortranarray(Ab[:m, :n])
    bad, _ = compare_ipiv(orc, A0, ipiv[:mn], nb)
    assert bad == 0
    assert orc.fresid(LU, ipiv[:mn], A0) < 1.0  # LU.dat THRESH


def test_submatrix_offsets(sl, orc, ctx):
    nb, ia, ja, n = 8, 9, 17, 40
    A0, B0 = system(orc, n, 2)
    info, LU, rel, X = run_pdgesv(sl, ctx, A0, B0, nb, ia=ia, ja=ja)
    assert info == 0
    bad, _ = compare_ipiv(orc, A0, rel, nb)
    assert bad == 0
    assert orc.sresid(A0, B0, X) < RESID_THRESH


def test_singular_info_and_no_solve(sl, orc, ctx):
    n, nb = 80, 16
    A0, B0 = system(orc, n, 1)
    A0[:, 37] = 0.0
    info, LU, rel, X = run_pdgesv(sl, ctx, A0, B0, nb)
    _, _, infol = orc.lapack_dgetrf(A0)
    assert info == infol == 38
    np.testing.assert_array_equal(X, B0)  # PDGETRS skipped (pdgesv.f:231)
    bad, _ = compare_ipiv(orc, A0, rel, nb)
    assert bad == 0


def test_zero_matrix_info_one(sl, orc, ctx):
    n, nb = 10, 4
    A0 = np.zeros((n, n), order="F")
    Ab = padded(A0)
    desc = np.array([1, ctx, Ab.shape[0], Ab.shape[1], nb, nb, 0, 0, Ab.shape[0]], np.int32)
    ipiv = np.zeros(Ab.shape[0] + nb, dtype=np.int32)
    assert sl.pdgetrf(n, n, Ab, 1, 1, desc, ipiv) == 1
    np.testing.assert_array_equal(ipiv[:n], np.arange(1, n + 1))  # AMAX == 0 keeps the row


@pytest.mark.parametrize("trans", ["N", "T", "C"])
def test_pdgetrs_trans(sl, orc, ctx, trans):
    n, nb, nrhs = 300, 32, 5
    A0, B0 = system(orc, n, nrhs)
    A = np.asfortranarray(A0.copy())
    desc = np.array([1, ctx, n, n, nb, nb, 0, 0, n], np.int32)
    ipiv = np.zeros(n + nb, dtype=np.int32)
    assert sl.pdgetrf(n, n, A, 1, 1, desc, ipiv) == 0
    X = np.asfortranarray(B0.copy())
    descb = np.array([1, ctx, n, nrhs, nb, nb, 0, 0, n], np.int32)
    assert sl.pdgetrs(trans, n, nrhs, A, 1, 1, desc, ipiv, X, 1, 1, descb) == 0
    Aop = A0 if trans == "N" else np.asfortranarray(A0.T)
    assert orc.sresid(Aop, B0, X) < RESID_THRESH


def test_device_entry_points(sl, orc, ctx):
    import torch

    n, nrhs, nb = 777, 4, 64
    A0, B0 = system(orc, n, nrhs)
    ldda = 800
    dA = torch.zeros((n, ldda), dtype=torch.float64, device="cuda")  # column-major via transpose
    dA[:, :n] = torch.from_numpy(np.ascontiguousarray(A0.T)).cuda()
    dB = torch.from_numpy(np.ascontiguousarray(B0.T)).cuda()
    dpiv = torch.zeros(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    info = sl.dgesv_dev(n, nrhs, dA.data_ptr(), ldda, dpiv.data_ptr(), dB.data_ptr(), n, nb)
    assert info == 0
    X = np.asfortranarray(dB.cpu().numpy().T)
    rel = dpiv.cpu().numpy()
    bad, _ = compare_ipiv(orc, A0, rel, nb)
    assert bad == 0
    assert orc.sresid(A0, B0, X) < RESID_THRESH


def test_config_n2048_nb64(sl, orc, ctx):
    # Plain FP64 PDGESV, N=2048, NB=64, NRHS=1, U[-0.5,0.5] from the seeded LCG
    n, nb = 2048, 64
    A0, B0 = system(orc, n, 1)
    info, LU, rel, X = run_pdgesv(sl, ctx, A0, B0, nb)
    assert info == 0
    bad, ties = compare_ipiv(orc, A0, rel, nb)
    assert bad == 0, ties
    assert orc.fresid(LU, rel, A0) < RESID_THRESH
    assert orc.sresid(A0, B0, X) < RESID_THRESH


@pytest.mark.parametrize("m,n,nb", [(2048, 2048, 64), (1000, 1000, 64), (3000, 3000, 256),
                                    (1500, 900, 64), (700, 1300, 64), (600, 600, 256)])
def test_host_path_chunked_copy_matches_device_path(sl, orc, ctx, m, n, nb):
    # pdgetrf_ / pdgesv_ copy A to the GPU in column chunks and run step 0 of
    # the factorization chunk by chunk as they land; the device entry points
    # get A whole. The interchanges and the trailing update are per column;
    # the U12 solve's first product balances its slices by the row maxima of
    # the columns it is given, so step 0's U12 rows agree to rounding rather
    # than bitwise. Pivots must be identical, factors and solution equal to
    # rounding.
    import torch

    rng = np.random.default_rng(m * 7 + n + nb)
    A0 = np.asfortranarray(rng.uniform(-0.5, 0.5, (m, n)))
    dA = torch.from_numpy(np.ascontiguousarray(A0.T)).cuda()
    mn = min(m, n)
    dpiv = torch.zeros(mn, dtype=torch.int32, device="cuda")
    assert sl.dgetrf_dev(m, n, dA.data_ptr(), m, dpiv.data_ptr(), nb) == 0
    LU_dev = np.asfortranarray(dA.cpu().numpy().T)
    piv_dev = dpiv.cpu().numpy()  # 1-based, as LAPACK's
    LU = np.asfortranarray(A0.copy())
    desca = np.array([1, ctx, m, n, nb, nb, 0, 0, m], np.int32)
    ipiv = np.zeros(m + nb, np.int32)
    assert sl.pdgetrf(m, n, LU, 1, 1, desca, ipiv) == 0
    np.testing.assert_array_equal(ipiv[:mn], piv_dev)
    scale = np.max(np.abs(LU_dev), axis=1, keepdims=True)
    assert np.max(np.abs(LU - LU_dev) / scale) < 1e-10
    if m == n:
        B0 = np.asfortranarray(rng.uniform(-0.5, 0.5, (n, 3)))
        dA = torch.from_numpy(np.ascontiguousarray(A0.T)).cuda()
        dB = torch.from_numpy(np.ascontiguousarray(B0.T)).cuda()
        assert sl.dgesv_dev(n, 3, dA.data_ptr(), n, dpiv.data_ptr(), dB.data_ptr(), n, nb) == 0
        X_dev = np.asfortranarray(dB.cpu().numpy().T)
        LU2, X = np.asfortranarray(A0.copy()), np.asfortranarray(B0.copy())
        descb = np.array([1, ctx, n, 3, nb, nb, 0, 0, n], np.int32)
        assert sl.pdgesv(n, 3, LU2, 1, 1, desca, ipiv, X, 1, 1, descb) == 0
        assert np.max(np.abs(LU2 - LU_dev) / scale) < 1e-10
        assert np.max(np.abs(X - X_dev)) <= 1e-10 * np.max(np.abs(X_dev))
        assert orc.sresid(A0, B0, X) < RESID_THRESH


@pytest.mark.parametrize("n,nb", [(3000, 256), (4096, 128)])
def test_update_sm_reserve_changes_no_bit(sl, orc, ctx, n, nb):
    # The look-ahead trailing update leaves SMs to the panel's stream by
    # capping its grid; each tile's product is the same whichever CTA computes
    # it, so the factors and pivots are bitwise those of the uncapped update.
    import torch

    L = sl.lib()
    rng = np.random.default_rng(n + nb)
    A0 = np.asfortranarray(rng.uniform(-0.5, 0.5, (n, n)))
    outs = []
    try:
        for lo, hi in ((0, 0), (24, 88), (120, 120), (8, 8)):
            L.sl1x1_set_update_reserve(lo, hi)
            dA = torch.from_numpy(np.ascontiguousarray(A0.T)).cuda()
            dpiv = torch.zeros(n, dtype=torch.int32, device="cuda")
            assert sl.dgetrf_dev(n, n, dA.data_ptr(), n, dpiv.data_ptr(), nb) == 0
            outs.append((dA.cpu().numpy(), dpiv.cpu().numpy()))
    finally:
        L.sl1x1_set_update_reserve(24, 88)
    for LU_t, piv in outs[1:]:
        np.testing.assert_array_equal(piv, outs[0][1])
        np.testing.assert_array_equal(LU_t, outs[0][0])
    assert orc.fresid(np.asfortranarray(outs[0][0].T), outs[0][1], A0) < RESID_THRESH


def test_config_n16384_nb256_full_size(sl, orc, ctx):
    # The headline case at full size: plain FP64 PDGESV, N=16384, NB=256,
    # NRHS=16, U[-0.5,0.5] from the tester's seeded generator. IPIV against
    # the oracle's pdgetrf (all host cores), then both scaled residuals.
    n, nb, nrhs = 16384, 256, 16
    orc.set_threads(os.cpu_count() or 1)
    A0, B0 = system(orc, n, nrhs)
    info, LU, rel, X = run_pdgesv(sl, ctx, A0, B0, nb)
    assert info == 0
    bad, ties = compare_ipiv(orc, A0, rel, nb)
    print(f"N={n}: {bad} pivot mismatches outside near ties; logged tie columns {ties}")
    assert bad == 0, ties
    assert orc.sresid(A0, B0, X) < RESID_THRESH
    assert orc.fresid(LU, rel, A0) < RESID_THRESH


@pytest.mark.parametrize("norm", ["M", "1", "O", "I", "F", "E"])
def test_pdlange_norms(sl, orc, ctx, norm):
    m, n = 300, 170
    A = orc.matgen(m, n, 100)
    Ab = padded(A, ia=5, ja=3)
    d = np.array([1, ctx, Ab.shape[0], Ab.shape[1], 4, 4, 0, 0, Ab.shape[0]], np.int32)
    v = sl.pdlange(norm, m, n, Ab, 5, 3, d)
    ref = {"M": np.abs(A).max(), "1": np.abs(A).sum(0).max(), "O": np.abs(A).sum(0).max(),
           "I": np.abs(A).sum(1).max(), "F": np.linalg.norm(A), "E": np.linalg.norm(A)}[norm]
    assert abs(v - ref) <= 1e-13 * ref


@pytest.mark.parametrize("norm", ["1", "I"])
@pytest.mark.parametrize("n", [2, 77, 600])
def test_pdgecon_brackets_true_rcond(sl, orc, ctx, norm, n):
    A0, _ = system(orc, n, 1)
    A = np.asfortranarray(A0.copy())
    nb = 32
    d = np.array([1, ctx, n, n, nb, nb, 0, 0, n], np.int32)
    ipiv = np.zeros(n + nb, dtype=np.int32)
    anorm = sl.pdlange(norm, n, n, A, 1, 1, d)
    assert sl.pdgetrf(n, n, A, 1, 1, d, ipiv) == 0
    rc, info, _, _ = sl.pdgecon(norm, n, A, 1, 1, d, anorm)
    assert info == 0
    inv = np.linalg.inv(A0)
    true = 1.0 / (anorm * (np.abs(inv).sum(0).max() if norm == "1" else np.abs(inv).sum(1).max()))
    # the estimate of ||inv(A)|| never exceeds the true norm, and is rarely far below it
    assert true * (1 - 1e-10) <= rc <= 10.0 * true, (rc, true)


@pytest.mark.parametrize("n,nb", [(1, 1), (5, 2), (200, 32), (1000, 64)])
def test_pdgetri_inverse(sl, orc, ctx, n, nb):
    A0, _ = system(orc, n, 1)
    A = np.asfortranarray(A0.copy())
    d = np.array([1, ctx, n, n, nb, nb, 0, 0, n], np.int32)
    ipiv = np.zeros(n + nb, dtype=np.int32)
    assert sl.pdgetrf(n, n, A, 1, 1, d, ipiv) == 0
    LU = np.asfortranarray(A.copy())
    info, _, _ = sl.pdgetri(n, A, 1, 1, d, ipiv)
    assert info == 0
    R = A0 @ A - np.eye(n)
    eps = 2.0 ** -53
    assert np.abs(R).sum(1).max() / (np.abs(A0).sum(1).max() * np.abs(A).sum(1).max() * n * eps) < 16
    # the oracle's restatement of the reference's algorithm on the same factors
    info_o, Xo = orc.pdgetri(LU, ipiv[:n] - 1, nb)
    assert info_o == 0
    assert np.abs(A - Xo).max() <= 1e-8 * np.abs(Xo).max()


def test_pdgetri_singular_info(sl, orc, ctx):
    n, nb = 50, 8
    A0, _ = system(orc, n, 1)
    A0[:, 20] = 0.0
    A = np.asfortranarray(A0.copy())
    d = np.array([1, ctx, n, n, nb, nb, 0, 0, n], np.int32)
    ipiv = np.zeros(n + nb, dtype=np.int32)
    k = sl.pdgetrf(n, n, A, 1, 1, d, ipiv)
    assert k == 21
    before = A.copy()
    info, _, _ = sl.pdgetri(n, A, 1, 1, d, ipiv)
    assert info == 21
    np.testing.assert_array_equal(A, before)  # inverse not computed


def test_tall_matrix_beyond_shared_memory_panel(sl, orc, ctx):
    """M = 200,000 > 152 SMs x 768 rows: the panel's rows no longer fit the
    SMs' shared memory, and each CTA keeps its rows in a library-owned global
    buffer instead. pdgetrf_ on a 200000 x 512 matrix (0.8 GB): IPIV identical
    to the oracle's, the tester's factor residual below 16."""
    m, n, nb = 200000, 512, 256
    assert m > 152 * 768
    A0 = orc.matgen(m, n, 100, kind=1)
    A = np.asfortranarray(A0.copy())
    desc = np.array([1, ctx, m, n, nb, nb, 0, 0, m], np.int32)
    ipiv = np.zeros(m + nb, np.int32)
    assert sl.pdgetrf(m, n, A, 1, 1, desc, ipiv) == 0
    bad, ties = compare_ipiv(orc, A0, ipiv[:n], nb)
    assert bad == 0, ties
    assert orc.fresid(A, ipiv[:n], A0) < RESID_THRESH


@pytest.mark.parametrize("n,nb", [(200, 32), (1000, 64)])
def test_scratch_on_reused_dirty_memory(sl, orc, ctx, n, nb):
    # The sliced products keep epoch-tagged balancing words at the start of
    # their scratch buffers; a buffer allocated over memory that held other
    # data (here: all bits set, freed back to the driver) must start clean,
    # or the words of later products would never replace the stale ones.
    import torch

    L = sl.lib()
    L.sl1x1_finalize()
    junk = torch.full((1 << 27,), -1, dtype=torch.int64, device="cuda")  # 1 GiB of 0xff
    torch.cuda.synchronize()
    del junk
    torch.cuda.empty_cache()
    rng = np.random.default_rng(n + 3)
    A0 = np.asfortranarray(rng.uniform(-1, 1, (n, n)))
    dA = torch.from_numpy(np.ascontiguousarray(A0.T)).cuda()
    dpiv = torch.zeros(n, dtype=torch.int32, device="cuda")
    assert sl.dgetrf_dev(n, n, dA.data_ptr(), n, dpiv.data_ptr(), nb) == 0
    LU = np.asfortranarray(dA.cpu().numpy().T)
    assert orc.fresid(LU, dpiv.cpu().numpy(), A0) < RESID_THRESH


@pytest.mark.parametrize("trans", ["N", "T"])
@pytest.mark.parametrize("n,nrhs", [(1, 1), (63, 2), (64, 1), (65, 16), (129, 3), (200, 17), (1300, 16), (2500, 5)])
def test_chained_solve_edges(sl, gpu_required, n, nrhs, trans):
    """PDGETRS over the edges of the chained solve: blocks of 64 rows, one
    to many CTAs per SM (1300 x 16, 2500 x 5); padded leading dimensions,
    untouched padding."""
    import torch

    rng = np.random.default_rng(n + nrhs)
    A = rng.uniform(-0.5, 0.5, (n, n))
    B = rng.uniform(-0.5, 0.5, (n, nrhs))
    lda, ldb = n + 3, n + 1
    dA = torch.full((n, lda), -9923.0, dtype=torch.float64, device="cuda")
    dB = torch.full((nrhs, ldb), -9923.0, dtype=torch.float64, device="cuda")
    dA[:, :n] = torch.from_numpy(A.T.copy())
    dB[:, :n] = torch.from_numpy(B.T.copy())
    ip = torch.zeros(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert sl.dgetrf_dev(n, n, dA.data_ptr(), lda, ip.data_ptr(), 64) == 0
    assert sl.dgetrs_dev(trans, n, nrhs, dA.data_ptr(), lda, ip.data_ptr(), dB.data_ptr(), ldb) == 0
    X = dB[:, :n].T.cpu().numpy()
    assert (dB[:, n:] == -9923.0).all()
    op = A if trans == "N" else A.T
    res = np.abs(B - op @ X).max(axis=0)
    scale = np.abs(op).sum(axis=1).max() * np.abs(X).max(axis=0) * n * 2.0**-53
    assert (res / scale < 16.0).all()  # the tester's bound


def _triangle(kind, n, seed):
    """Triangles with large inverses that are their own LU factors."""
    r = np.random.default_rng(seed)
    if kind == "uniform":
        return np.triu(r.uniform(-0.5, 0.5, (n, n)))
    if kind == "normal":
        return np.triu(r.standard_normal((n, n)))
    if kind == "lower":  # inv(L) doubles with every row
        return np.tril(-np.ones((n, n)), -1) + np.eye(n)
    # rows of very different size: 1/u_ii and u_ij/u_ii leave the range of a double
    a = np.triu(r.uniform(-0.5, 0.5, (n, n))) + np.eye(n)
    a[0, 0] *= 1e-200
    a[0, 1:] *= 1e110
    a[n // 2, n // 2] *= 2.0**-1030
    a[n // 2, n // 2 + 1:] *= 2.0**-1030
    a[:n // 2, n // 2] *= 2.0**-1030
    return a


@pytest.mark.parametrize("trans", ["N", "T"])
@pytest.mark.parametrize("nrhs", [1, 16, 128, 129, 300])
@pytest.mark.parametrize("kind,n,seed", [("uniform", 32, 0), ("uniform", 32, 1), ("normal", 32, 2), ("uniform", 64, 0),
                                         ("uniform", 100, 3), ("uniform", 300, 4), ("lower", 60, 0), ("lower", 200, 0)])
def test_solve_with_ill_conditioned_triangles(sl, gpu_required, kind, n, seed, nrhs, trans):
    """Diagonal blocks whose inverses are large are solved as accurately as by substitution:
    the tester's bound, which their inverses miss by up to 12 orders of magnitude."""
    import torch

    A = _triangle(kind, n, seed)
    op = A if trans == "N" else A.T
    B = op @ np.random.default_rng(seed).uniform(-1, 1, (n, nrhs))
    dA, dB = torch.from_numpy(A.T.copy()).cuda(), torch.from_numpy(B.T.copy()).cuda()
    ip = torch.zeros(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert sl.dgetrf_dev(n, n, dA.data_ptr(), n, ip.data_ptr()) == 0
    assert torch.equal(dA.cpu(), torch.from_numpy(A.T.copy()))
    assert sl.dgetrs_dev(trans, n, nrhs, dA.data_ptr(), n, ip.data_ptr(), dB.data_ptr(), n) == 0
    X = dB.T.cpu().numpy()
    res = np.abs(B - op @ X).max(axis=0) / (np.abs(op).sum(axis=1).max() * np.abs(X).max(axis=0) * n * 2.0**-53)
    assert (res < RESID_THRESH).all(), res.max()


@pytest.mark.parametrize("kind,n,seed", [("uniform", 64, 0), ("uniform", 300, 4), ("lower", 200, 0), ("lower", 400, 0)])
def test_inverse_of_ill_conditioned_triangles(sl, gpu_required, kind, n, seed):
    """PDGETRI through the same block steps, below and above 256 (inv(L) as a triangle):
    each column of the inverse solves its system within the tester's bound."""
    import torch

    A = _triangle(kind, n, seed)
    dA = torch.from_numpy(A.T.copy()).cuda()
    ip = torch.arange(1, n + 1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert sl.lib().sl1x1_dgetri_dev(n, dA.data_ptr(), n, ip.data_ptr(), None) == 0
    X = dA.T.cpu().numpy()
    res = np.abs(np.eye(n) - A @ X).max(axis=0) / (np.abs(A).sum(axis=1).max() * np.abs(X).max(axis=0) * n * 2.0**-53)
    assert (res < RESID_THRESH).all(), res.max()


@pytest.mark.parametrize("trans", ["N", "T"])
@pytest.mark.parametrize("nrhs", [1, 129, 300])
@pytest.mark.parametrize("n", [20, 90])
def test_solve_with_rows_of_extreme_size(sl, gpu_required, n, nrhs, trans):
    """A subnormal diagonal entry, and a row whose quotients by its own leave the range: no
    overflow that a substitution does not have."""
    import torch

    A = _triangle("extreme", n, 5)
    x0 = np.random.default_rng(n).uniform(0.5, 1, (n, nrhs))
    x0[0] = 1e-120  # (T: u_0j x_0 far below the others)
    B = (A if trans == "N" else A.T) @ x0
    dA, dB = torch.from_numpy(A.T.copy()).cuda(), torch.from_numpy(B.T.copy()).cuda()
    ip = torch.arange(1, n + 1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert sl.dgetrs_dev(trans, n, nrhs, dA.data_ptr(), n, ip.data_ptr(), dB.data_ptr(), n) == 0
    X = dB.T.cpu().numpy()
    assert np.isfinite(X).all()
    op = np.abs(A if trans == "N" else A.T)
    # componentwise: |b - op x| <= n eps |op| |x| for either order of the sums (Higham, 8.5)
    r = np.abs(B - (A if trans == "N" else A.T) @ X)
    assert (r <= 4 * n * 2.0**-53 * (op @ np.abs(X)) + 2.0**-1040).all()


def test_chained_solve_on_reused_dirty_memory(sl, gpu_required):
    """The chained solve's words start cleared in every buffer they grow into, also
    when it stands at the old one's address among memory that holds the epochs
    of the calls to come."""
    import torch

    L = sl.lib()
    L.sl1x1_finalize()
    rng = np.random.default_rng(2)
    epoch = 0
    for n in (40, 64, 90, 200, 333, 700, 1000, 1500):
        dirty = [torch.full((1 << 24,), epoch + e, dtype=torch.int64, device="cuda") for e in (1, 2, 1, 2)]
        dirty += [torch.full((4096,), epoch + 1 + i % 2, dtype=torch.int64, device="cuda") for i in range(64)]
        torch.cuda.synchronize()
        del dirty
        torch.cuda.empty_cache()
        A = rng.uniform(-0.5, 0.5, (n, n))
        B = rng.uniform(-0.5, 0.5, (n, 3))
        dA, dB = torch.from_numpy(A.T.copy()).cuda(), torch.from_numpy(B.T.copy()).cuda()
        ip = torch.zeros(n, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        assert sl.dgesv_dev(n, 3, dA.data_ptr(), n, ip.data_ptr(), dB.data_ptr(), n) == 0
        epoch += 2
        X = dB.T.cpu().numpy()
        res = np.abs(B - A @ X).max(axis=0) / (np.abs(A).sum(axis=1).max() * np.abs(X).max(axis=0) * n * 2.0**-53)
        assert (res < 16.0).all(), n


@pytest.mark.parametrize("kind", ["random", "ties", "zero column", "nan"])
@pytest.mark.parametrize("m", [1, 5, 31, 33, 64, 65, 128, 129, 513, 1024, 1025, 2047, 2048, 2049])
def test_cluster_panel_equals_grid_panel(sl, gpu_required, m, kind):
    """The one-cluster panel (up to 2048 rows) and the one that exchanges through L2
    (asked for by a row-slice setting) give the same factors and pivots, bit for
    bit: cluster sizes 1 to 16, partial rows and widths, ties, zero pivots, NaN in
    and off the diagonal."""
    import torch

    n = 70
    rng = np.random.default_rng(m)
    A = rng.uniform(-0.5, 0.5, (m, n))
    if kind == "ties":
        A = rng.integers(-2, 3, (m, n)).astype(float)
    elif kind == "zero column":
        A[:, min(m, n) // 2] = 0.0
    elif kind == "nan":
        A[rng.integers(0, m), min(3, m - 1)] = np.nan
        A[min(40, m - 1), min(40, m - 1)] = np.nan
    L = sl.lib()
    got = []
    try:
        for rows in (0, 256):
            L.sl1x1_set_panel_rows(rows)
            dA = torch.from_numpy(A.T.copy()).cuda()
            ip = torch.zeros(min(m, n), dtype=torch.int32, device="cuda")
            torch.cuda.synchronize()
            info = sl.dgetrf_dev(m, n, dA.data_ptr(), m, ip.data_ptr(), 64)
            got.append((info, ip.cpu().numpy(), dA.cpu().numpy()))
    finally:
        L.sl1x1_set_panel_rows(0)
    assert got[0][0] == got[1][0]
    np.testing.assert_array_equal(got[0][1], got[1][1])
    np.testing.assert_array_equal(got[0][2], got[1][2])


@pytest.mark.parametrize("ib", [1, 2, 3])
@pytest.mark.parametrize("m,n", [(33, 33), (64, 70), (95, 97), (130, 40), (40, 130), (300, 257), (700, 321)])
def test_in_panel_steps(sl, orc, gpu_required, m, n, ib):
    """The in-panel step (interchanges, solve and product keys in one launch) for one
    and two sub-panels per block, the unfused one beyond; partial sub-panels, wide
    and tall matrices: pivots of the oracle's, and P A = L U to the tester's bound."""
    import torch

    rng = np.random.default_rng(m * n)
    A = np.asfortranarray(rng.uniform(-0.5, 0.5, (m, n)))
    dA = torch.from_numpy(A.T.copy()).cuda()
    ip = torch.zeros(min(m, n), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    L = sl.lib()
    try:
        L.sl1x1_set_panel_ib(ib)
        assert sl.dgetrf_dev(m, n, dA.data_ptr(), m, ip.data_ptr(), 256) == 0
    finally:
        L.sl1x1_set_panel_ib(0)
    F, piv = dA.T.cpu().numpy(), ip.cpu().numpy() - 1
    PA = A.copy()
    for k, p in enumerate(piv):
        PA[[k, p]] = PA[[p, k]]
    k = min(m, n)
    low, up = np.tril(F[:, :k], -1) + np.eye(m, k), np.triu(F[:k])
    assert np.abs(low).max() <= 1.0 + 1e-15  # partial pivoting
    assert np.abs(PA - low @ up).max() < 16.0 * max(m, n) * 2.0**-53 * np.abs(A).sum(axis=1).max()


@pytest.mark.parametrize("kind", ["random", "ties", "singular", "nan"])
@pytest.mark.parametrize("n,nrhs", [(1, 1), (2, 3), (4, 4), (5, 1), (16, 16), (17, 15), (17, 16), (31, 1), (32, 1), (32, 16), (32, 17)])
def test_small_gesv_equals_two_calls(sl, gpu_required, n, nrhs, kind):
    """PDGESV of up to 32 rows and 16 right-hand sides is one launch: pivots, INFO and
    factors bit for bit those of PDGETRF, X within the tester's bound, B untouched
    when singular; NaN and ties as IDAMAX takes them; padded arrays."""
    import torch

    rng = np.random.default_rng(n * 40 + nrhs)
    A = rng.uniform(-0.5, 0.5, (n, n))
    if kind == "ties":
        A = rng.integers(-2, 3, (n, n)).astype(float)
    elif kind == "singular":
        A[:, n // 2] = 0.0
    elif kind == "nan":
        A[n // 3, n // 2] = np.nan
    B = rng.uniform(-0.5, 0.5, (n, nrhs))
    lda, ldb = n + 2, n + 1
    dA = torch.full((n, lda), -9923.0, dtype=torch.float64, device="cuda")
    dA[:, :n] = torch.from_numpy(A.T.copy())
    dB = torch.full((nrhs, ldb), -9923.0, dtype=torch.float64, device="cuda")
    dB[:, :n] = torch.from_numpy(B.T.copy())
    dF = dA.clone()
    ip, ip2 = (torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    info = sl.dgesv_dev(n, nrhs, dA.data_ptr(), lda, ip.data_ptr(), dB.data_ptr(), ldb)
    info2 = sl.dgetrf_dev(n, n, dF.data_ptr(), lda, ip2.data_ptr())
    assert info == info2 and (kind != "singular" or info > 0)
    np.testing.assert_array_equal(ip.cpu().numpy(), ip2.cpu().numpy())
    np.testing.assert_array_equal(dA.cpu().numpy(), dF.cpu().numpy())
    assert (dB[:, n:] == -9923.0).all()
    X = dB[:, :n].T.cpu().numpy()
    if info > 0:
        np.testing.assert_array_equal(X, B)
    elif kind in ("random", "ties"):
        res = np.abs(B - A @ X).max(axis=0) / (np.abs(A).sum(axis=1).max() * np.abs(X).max(axis=0) * n * 2.0**-53)
        assert (res < 16.0).all()


@pytest.mark.parametrize("n", [255, 256, 257, 383, 640, 1000])
def test_inverse_by_triangles(sl, gpu_required, n):
    """PDGETRI on both sides of the order from which inv(L) is formed as a triangle
    and the interchanges become a column permutation; partial last blocks."""
    import torch

    rng = np.random.default_rng(n)
    A = rng.uniform(-0.5, 0.5, (n, n))
    dA = torch.full((n, n + 3), -9923.0, dtype=torch.float64, device="cuda")
    dA[:, :n] = torch.from_numpy(A.T.copy())
    ip = torch.zeros(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert sl.dgetrf_dev(n, n, dA.data_ptr(), n + 3, ip.data_ptr()) == 0
    assert sl.lib().sl1x1_dgetri_dev(n, dA.data_ptr(), n + 3, ip.data_ptr(), None) == 0
    assert (dA[:, n:] == -9923.0).all()
    V = dA[:, :n].T.cpu().numpy()
    res = np.abs(A @ V - np.eye(n)).sum(axis=1).max()
    assert res / (np.abs(A).sum(axis=1).max() * np.abs(V).sum(axis=1).max() * n * 2.0**-53) < 16.0  # the tester's bound


@pytest.mark.parametrize("m", [1, 2, 31, 32, 33, 64, 65, 127, 129, 224, 255, 256])
def test_u12_through_inverse_edges(sl, gpu_required, m):
    """One panel of m columns and a block row of 200: U12 = inv(L11) A12 with the
    inverse's last block partial, its middle column alone (odd m) or everything one
    block. P A = L U to the tester's bound."""
    import torch

    n = m + 200
    rng = np.random.default_rng(m)
    A = np.asfortranarray(rng.uniform(-0.5, 0.5, (m, n)))
    dA = torch.from_numpy(A.T.copy()).cuda()
    ip = torch.zeros(m, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert sl.dgetrf_dev(m, n, dA.data_ptr(), m, ip.data_ptr(), 256) == 0
    F, piv = dA.T.cpu().numpy(), ip.cpu().numpy() - 1
    PA = A.copy()
    for k, p in enumerate(piv):
        PA[[k, p]] = PA[[p, k]]
    low, up = np.tril(F[:, :m], -1) + np.eye(m), np.triu(F)
    assert np.abs(PA - low @ up).max() < 16.0 * n * 2.0**-53 * np.abs(A).sum(axis=1).max()


@pytest.mark.parametrize("m,n", [(1024, 1024), (1025, 1025), (1536, 1536), (1537, 1537), (2432, 1024), (2433, 1024), (257, 256), (40, 257), (600, 601)])
def test_one_panel_rule_edges(sl, orc, gpu_required, m, n):
    """Both sides of the sizes up to which a matrix is one panel (width, tiles of its
    in-panel products, wide matrices never): P A = L U to the tester's bound, and the
    caller's block size changes nothing."""
    import torch

    rng = np.random.default_rng(m + n)
    A = np.asfortranarray(rng.uniform(-0.5, 0.5, (m, n)))
    k, got = min(m, n), []
    for nb in (64, 1024):
        dA = torch.from_numpy(A.T.copy()).cuda()
        ip = torch.zeros(k, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        assert sl.dgetrf_dev(m, n, dA.data_ptr(), m, ip.data_ptr(), nb) == 0
        got.append((dA.T.cpu().numpy(), ip.cpu().numpy() - 1))
    F, piv = got[0]
    np.testing.assert_array_equal(F, got[1][0])
    np.testing.assert_array_equal(piv, got[1][1])
    PA = A.copy()
    for q, p in enumerate(piv):
        PA[[q, p]] = PA[[p, q]]
    low, up = np.tril(F[:, :k], -1) + np.eye(m, k), np.triu(F[:k])
    assert np.abs(low).max() <= 1.0 + 1e-15  # partial pivoting
    assert np.abs(PA - low @ up).max() < 16.0 * max(m, n) * 2.0**-53 * np.abs(A).sum(axis=1).max()


@pytest.mark.parametrize("trans", ["N", "T"])
@pytest.mark.parametrize("n,nrhs", [(1000, 128), (1000, 129), (2048, 128), (2049, 128), (4097, 64)])
def test_solve_dispatch_edges(sl, gpu_required, n, nrhs, trans):
    """Both sides of the number of right-hand sides up to which the solves are chained:
    the tester's scaled residual of every column below 16."""
    import torch

    rng = np.random.default_rng(n + nrhs)
    A, B = rng.uniform(-0.5, 0.5, (n, n)), rng.uniform(-0.5, 0.5, (n, nrhs))
    dA, dB = torch.from_numpy(A.T.copy()).cuda(), torch.from_numpy(B.T.copy()).cuda()
    ip = torch.zeros(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert sl.dgetrf_dev(n, n, dA.data_ptr(), n, ip.data_ptr()) == 0
    assert sl.dgetrs_dev(trans, n, nrhs, dA.data_ptr(), n, ip.data_ptr(), dB.data_ptr(), n) == 0
    X, op = dB.T.cpu().numpy(), A if trans == "N" else A.T
    res = np.abs(op @ X - B).max(axis=0) / (np.abs(op).sum(axis=1).max() * np.abs(X).max(axis=0) * n * 2.0**-53)
    assert (res < 16.0).all()


@pytest.mark.parametrize("m,n", [(1792, 1792), (1793, 1793), (2000, 1700), (5120, 5120), (5121, 5121)])
def test_tail_as_one_panel_edges(sl, gpu_required, m, n):
    """The last columns as one panel that also interchanges the rows of the columns
    before it: widths and left parts on both sides of its limits. P A = L U to the
    tester's bound over every column."""
    import torch

    g = torch.Generator(device="cuda").manual_seed(m + n)
    A = torch.rand((n, m), dtype=torch.float64, device="cuda", generator=g) - 0.5  # column-major m x n
    dA, ip = A.clone(), torch.zeros(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert sl.dgetrf_dev(m, n, dA.data_ptr(), m, ip.data_ptr()) == 0
    perm = np.arange(m)
    for k, p in enumerate(ip.cpu().numpy() - 1):
        perm[[k, p]] = perm[[p, k]]
    low = torch.tril(dA.T, -1)
    assert low.abs().max().item() <= 1.0 + 1e-15  # partial pivoting
    low.diagonal().fill_(1.0)
    res = A.T[torch.from_numpy(perm).cuda()] - low @ torch.triu(dA.T[:n])
    assert res.abs().max().item() < 16.0 * m * 2.0**-53 * A.T.abs().sum(dim=1).max().item()


@pytest.mark.parametrize("zero", [100, 300, 700, 1650])
def test_singular_info_in_blocks(sl, orc, ctx, zero):
    """A zero column in the first, second and third block of 256 and in the last panel."""
    n, nb = 1700, 64
    A0, B0 = system(orc, n, 1)
    A0[:, zero] = 0.0
    info, LU, rel, X = run_pdgesv(sl, ctx, A0, B0, nb)
    assert info == zero + 1
    np.testing.assert_array_equal(X, B0)
    bad, _ = compare_ipiv(orc, A0, rel, nb)
    assert bad == 0
    assert orc.fresid(LU, rel, A0) < RESID_THRESH


@pytest.mark.parametrize("col", [400, 1650])
def test_nan_in_blocks(sl, orc, ctx, col):
    """A NaN in one column of a matrix factored in blocks leaves the columns before it
    as they are, pivots and factors, and reaches the columns behind it."""
    n, nb = 1700, 64
    A0, B0 = system(orc, n, 1)
    _, LU0, rel0, _ = run_pdgesv(sl, ctx, A0, B0, nb)
    A1 = np.asfortranarray(A0.copy())
    A1[1000, col] = np.nan
    _, LU1, rel1, X = run_pdgesv(sl, ctx, A1, B0, nb)
    np.testing.assert_array_equal(rel1[:col], rel0[:col])
    # (columns of L, in the rows' order at that point: the later pivots permute them)
    np.testing.assert_allclose(LU1[:col, :col], LU0[:col, :col], rtol=0, atol=1e-9)
    assert np.isnan(LU1[:, col]).any() and np.isnan(LU1[-1, -1]) and np.isnan(X).any()
