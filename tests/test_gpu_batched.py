"""GPU tests of the batched solver (plan -> CUDA-graph execution) through the
C ABI: every system's solution is checked against the CPU oracle's FP64 solve
with the tester's scaled residual, INFO is exact, inputs are untouched and a
second execution of the graph gives identical results."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def make_batch(rng, count, nmin=16, nmax=512, rmax=8, singular=None):
    systems = []
    for i in range(count):
        n = int(rng.integers(nmin, nmax + 1))
        r = int(rng.integers(1, rmax + 1))
        A = np.asfortranarray(rng.uniform(-0.5, 0.5, size=(n, n)))
        if i % 2 == 0:
            A[np.diag_indices(n)] += n / 4.0  # diagonal shift on half the batch
        B = np.asfortranarray(rng.uniform(-0.5, 0.5, size=(n, r)))
        if singular is not None and i == singular:
            A[:, n // 3] = 0.0
        systems.append((A, B))
    return systems


class Plan:
    def __init__(self, sl, torch, systems, mode, autotune=1, tol=1.0):
        self.sl, self.torch = sl, torch
        self.dA = [torch.from_numpy(np.ascontiguousarray(A.T)).cuda() for A, _ in systems]
        self.dB = [torch.from_numpy(np.ascontiguousarray(B.T)).cuda() for _, B in systems]
        self.dX = [torch.zeros_like(b) for b in self.dB]
        k = len(systems)
        I = C.c_int * k
        P = C.c_void_p * k
        n = I(*[A.shape[0] for A, _ in systems])
        r = I(*[B.shape[1] for _, B in systems])
        self.batch = k
        self.plan = C.c_void_p()
        L = sl.lib()
        L.sl1x1_batch_plan_create.argtypes = [C.POINTER(C.c_void_p), C.c_int, C.c_void_p, C.c_void_p,
                                              C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p,
                                              C.c_void_p, C.c_void_p, C.c_int, C.c_double, C.c_int,
                                              C.c_void_p]
        L.sl1x1_batch_plan_create.restype = C.c_int
        L.sl1x1_batch_plan_execute.argtypes = [C.c_void_p, C.c_void_p]
        L.sl1x1_batch_plan_results.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p,
                                               C.c_void_p]
        L.sl1x1_batch_plan_shape.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p]
        L.sl1x1_batch_plan_destroy.argtypes = [C.c_void_p]
        torch.cuda.synchronize()
        info = L.sl1x1_batch_plan_create(
            C.byref(self.plan), k, n, r, P(*[t.data_ptr() for t in self.dA]), n,
            P(*[t.data_ptr() for t in self.dB]), n, P(*[t.data_ptr() for t in self.dX]), n, mode,
            tol, autotune, None)
        assert info == 0, info
        self.L = L

    def run(self):
        assert self.L.sl1x1_batch_plan_execute(self.plan, None) == 0
        info = (C.c_int * self.batch)()
        its = (C.c_int * self.batch)()
        sr = (C.c_double * self.batch)()
        assert self.L.sl1x1_batch_plan_results(self.plan, info, its, sr, None) == 0
        X = [np.asfortranarray(t.cpu().numpy().T) for t in self.dX]
        return list(info), list(its), list(sr), X

    def shape(self):
        t, c, s = C.c_int(), C.c_int(), C.c_int()
        self.L.sl1x1_batch_plan_shape(self.plan, C.byref(t), C.byref(c), C.byref(s))
        return t.value, c.value, s.value

    def close(self):
        self.L.sl1x1_batch_plan_destroy(self.plan)


@pytest.mark.parametrize("mode", [0, 1])
def test_batched_matches_oracle(sl, orc, gpu_required, mode):
    import torch

    rng = np.random.default_rng(100 + mode)
    systems = make_batch(rng, 48)
    plan = Plan(sl, torch, systems, mode)
    info, its, sr, X = plan.run()
    assert plan.shape()[0] in (128, 256, 512)
    for i, (A, B) in enumerate(systems):
        assert info[i] == 0
        r = orc.sresid(A, B, X[i])
        assert r < 16.0, (i, A.shape, r)
        # the kernel's own residual is at the same rounding-noise level (different summation order)
        assert sr[i] < 16.0 and sr[i] <= 10.0 * r + 0.1 and r <= 10.0 * sr[i] + 0.1, (sr[i], r)
        if mode == 1:
            assert its[i] >= 1 or its[i] == -1
    # inputs untouched
    for (A, B), dA, dB in zip(systems, plan.dA, plan.dB):
        np.testing.assert_array_equal(dA.cpu().numpy().T, A)
        np.testing.assert_array_equal(dB.cpu().numpy().T, B)
    # replaying the graph gives identical results
    info2, its2, sr2, X2 = plan.run()
    assert info2 == info and its2 == its
    for a, b in zip(X, X2):
        np.testing.assert_array_equal(a, b)
    plan.close()


@pytest.mark.parametrize("mode", [0, 1])
def test_batched_singular_and_edges(sl, orc, gpu_required, mode):
    import torch

    rng = np.random.default_rng(7)
    systems = make_batch(rng, 9, nmin=1, nmax=70, rmax=8, singular=4)
    systems.append((np.asfortranarray(np.array([[2.0]])), np.asfortranarray(np.array([[3.0]]))))
    plan = Plan(sl, torch, systems, mode, autotune=0)
    info, its, sr, X = plan.run()
    A4 = systems[4][0]
    _, _, info_l = orc.lapack_dgetrf(A4)
    assert info[4] == info_l > 0
    for i, (A, B) in enumerate(systems):
        if i == 4:
            continue
        assert info[i] == 0
        assert orc.sresid(A, B, X[i]) < 16.0
    np.testing.assert_allclose(X[-1], [[1.5]])
    plan.close()


def test_batched_plan_rejects_bad_sizes(sl):
    L = sl.lib()
    saved = L.sl1x1_batch_plan_create.argtypes
    L.sl1x1_batch_plan_create.argtypes = None
    try:
        k = 1
        n = (C.c_int * k)(600)
        r = (C.c_int * k)(1)
        p = C.c_void_p()
        P = (C.c_void_p * k)(None)
        assert L.sl1x1_batch_plan_create(C.byref(p), k, n, r, P, n, P, n, P, n, 0, C.c_double(1.0),
                                         0, None) == -3
    finally:
        L.sl1x1_batch_plan_create.argtypes = saved


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("orders", [(1, 2, 15, 16, 17), (31, 32, 33, 127, 128, 129), (255, 257, 496, 511, 512)])
def test_batched_panel_edges(sl, orc, gpu_required, mode, orders):
    """Orders around the panel width (16), the chunk widths, the threads per CTA
    and the largest order, with 1 and 8 right-hand sides and a permuted matrix
    whose columns interchange rows of every part of the panel."""
    import torch

    rng = np.random.default_rng(sum(orders) + mode)
    systems = []
    for n in orders:
        for r in (1, 8):
            A = rng.uniform(-0.5, 0.5, (n, n))
            A[rng.permutation(n), np.arange(n)] += 0.5 * np.sqrt(n)
            systems.append((np.asfortranarray(A), np.asfortranarray(rng.uniform(-0.5, 0.5, (n, r)))))
    plan = Plan(sl, torch, systems, mode, autotune=0)
    info, its, sr, X = plan.run()
    for i, (A, B) in enumerate(systems):
        assert info[i] == 0
        assert orc.sresid(A, B, X[i]) < 16.0  # the tester's bound
    plan.close()


def test_one_by_one_systems_divide(sl, gpu_required):
    """The backward substitution's quotient from the diagonal's reciprocal: the rounded one
    over random and special significands (all ones, powers of two, neighbours of 1), and
    within one unit in the last place where remainders or reciprocals are subnormal. As
    one-by-one systems of a plan and of PDGESV."""
    import torch

    rng = np.random.default_rng(11)
    a = rng.uniform(1, 2, 512) * np.exp2(rng.integers(-300, 301, 512))
    a[:6] = [1.0, 2.0 - 2.0**-52, 1.0 + 2.0**-52, 0.5, 3.0, 1.0 - 2.0**-53]
    b = rng.uniform(1, 2, (512, 8)) * np.exp2(rng.integers(-300, 301, (512, 8)))
    b[:6] = rng.uniform(1, 2, (6, 8))
    b[:, 0] = a
    a[::3] *= -1
    edge_a = np.array([2.0**1023, 1.7e308, 2.0**-1022, 5e-324 * 12345, 1.0, 3.0, 2.0**1000, 2.0**-500])
    edge_b = np.array([[1.0, 1.5e308, 2.0**-1000 * 1.7, 3e-310, 1.1e-300, 2.0**-1022, 1.2e-308, 7.0 * 5e-324]]).repeat(8, 0)
    for A, B, ulps in ((a, b, 0), (edge_a, edge_b, 1)):
        with np.errstate(over="ignore", under="ignore"):
            want = B / A[:, None]
        ok = np.isfinite(want)
        systems = [(np.full((1, 1), v, order="F"), np.asfortranarray(w[None, :])) for v, w in zip(A, B)]
        p = Plan(sl, torch, systems, mode=0, autotune=0)
        p.run()
        torch.cuda.synchronize()
        got = np.array([x.cpu().numpy().reshape(-1) for x in p.dX])
        p.close()
        assert (np.abs(got[ok] - want[ok]) <= ulps * np.spacing(np.abs(want[ok]))).all()
        assert np.array_equal(np.isfinite(got), ok)
        dA, dB = torch.from_numpy(A.copy()).cuda(), torch.from_numpy(B.copy()).cuda()
        ip = torch.zeros(1, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        for i in range(0, len(A), 1 if ulps else 16):
            assert sl.dgesv_dev(1, 8, dA.data_ptr() + 8 * i, 1, ip.data_ptr(), dB.data_ptr() + 64 * i, 1) == 0
            x = dB[i].cpu().numpy()
            x, w = x[ok[i]], want[i][ok[i]]
            assert (np.abs(x - w) <= ulps * np.spacing(np.abs(w))).all()


@pytest.mark.parametrize("mode", [0, 1])
def test_zero_right_hand_sides(sl, orc, gpu_required, mode):
    """Zero columns first, in the middle, last and throughout: zero solutions, finite
    residuals of the others, and no system sent to the FP64 pass for them."""
    import torch

    rng = np.random.default_rng(21)
    systems = make_batch(rng, 8, nmin=20, nmax=150, rmax=1)
    zeros = [[0], [2], [4], [0, 4], [1, 2, 3], [0, 1, 2, 3, 4], [0, 1, 2, 3], []]
    systems = [(A + np.eye(len(A)) * 4, np.asfortranarray(rng.uniform(-0.5, 0.5, (len(A), 5)))) for A, _ in systems]
    for (_, B), z in zip(systems, zeros):
        B[:, z] = 0.0
    systems = [(np.asfortranarray(A), B) for A, B in systems]
    plan = Plan(sl, torch, systems, mode)
    info, its, sr, X = plan.run()
    plan.close()
    for i, ((A, B), z) in enumerate(zip(systems, zeros)):
        assert info[i] == 0 and np.isfinite(sr[i]) and sr[i] < 16.0
        assert its[i] >= 1 if mode == 1 else its[i] == 0
        assert (X[i][:, z] == 0.0).all()
        keep = [c for c in range(5) if c not in z]
        if keep:
            assert orc.sresid(A, np.asfortranarray(B[:, keep]), np.asfortranarray(X[i][:, keep])) < 16.0
