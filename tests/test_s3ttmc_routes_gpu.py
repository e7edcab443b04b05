"""S3TTMc forms that the automatic schedule takes and the other tests do not reach:
row bands of every kernel, the FP64 tensor-core form of the order-5 CTA kernel at
its group and prefix counts and with infinities and NaN, order 4 at R <= 8 in FP32
with the same, and the order-5 call without memory for the group kernel's owners."""
import itertools

import numpy as np
import pytest

import oracle_lib as orc
from symprop_b200 import synth
from test_memory_gpu import refuse

pytestmark = pytest.mark.gpu


def rows_differ(a, b):
    norm = np.linalg.norm(b, axis=1)
    return float(np.max(np.linalg.norm(a - b, axis=1) / np.where(norm == 0, 1.0, norm)))


@pytest.mark.parametrize("bands", [1, 2, 5, 64])
@pytest.mark.parametrize("order,n,nnz,R", [(6, 400, 900, 8), (6, 400, 900, 3), (6, 300, 900, 10), (5, 200, 4000, 8),
                                           (5, 900, 3000, 16), (4, 300, 6000, 8), (4, 300, 6000, 11)])
def test_row_bands_match_the_device_call(gpu, monkeypatch, order, n, nnz, R, bands):
    """Order 6 at R <= 8 forks in every band: rows of at most 8 owners and others."""
    import torch
    monkeypatch.setenv("SPB_HOST_BANDS", str(bands))
    t = synth.zipf_tuples(order, n, nnz, 1.1, order + R)
    v = synth.uniform_values(t.shape[0], 3)
    X = gpu.SpSymtensor(n, order, t, v)
    U = np.random.default_rng(R).standard_normal((n, R))
    for prec, dt in ((gpu.FP64, torch.float64), (gpu.FP32, torch.float32)):
        Uc = U.astype(np.float64 if prec == gpu.FP64 else np.float32)
        Yh = X.S3TTMc(Uc, R, True, precision=prec)
        dU = torch.from_numpy(Uc).cuda()
        dY = torch.full(Yh.shape, float("nan"), dtype=dt, device="cuda")
        torch.cuda.synchronize()
        X.s3ttmc_device(dU.data_ptr(), R, dY.data_ptr(), True, prec)
        torch.cuda.synchronize()
        np.testing.assert_array_equal(Yh, dY.cpu().numpy())
    Yo = orc.s3ttmc(order, n, t, v, U, R, True)
    assert np.linalg.norm(X.S3TTMc(U, R, True) - Yo) <= 1e-12 * np.linalg.norm(Yo)


def grouped_tensor():
    """Order 5, over 64 owners a node on average (the rule of the tensor-core form).
    Hubs 0..29 are dense; row 30 + i has 1 + i groups (first pivots), of 1 to 7 prefixes
    each by i % 7; nodes 130.. appear in one tuple each."""
    rng = np.random.default_rng(7)
    t = [tuple(x) for x in synth.zipf_tuples(5, 30, 6000, 0.3, 5).astype(np.int64) - 1]
    nxt = 130
    for i in range(28):
        for g in range(1 + i):
            for h in range(1 + i % 7):
                t.append((g, 29 - h, 30 + i, 60 + (i + 3 * g + h) % 60, 60 + (5 * i + g + 7 * h) % 60))
    for k in range(20):
        t.append((k, k + 1, 30 + k, 60 + k, nxt))
        nxt += 1
    t = np.unique(np.sort(np.array(t, np.int64) + 1, axis=1), axis=0).astype(np.uint32)
    return nxt, t, rng.uniform(0.1, 1.0, t.shape[0])


@pytest.mark.parametrize("R", [13, 14, 16])
def test_order5_tensor_core_form(gpu, R):
    n, t, v = grouped_tensor()
    assert t.shape[0] * 5 >= 64 * n
    U = np.random.default_rng(R).uniform(0.5, 1.5, (n, R))  # no cancellation: the bar holds row by row
    X = gpu.SpSymtensor(n, 5, t, v)
    Y = X.S3TTMc(U, R, True)
    assert rows_differ(Y, orc.s3ttmc(5, n, t, v, U, R, True)) < 1e-12
    assert np.array_equal(Y, X.S3TTMc(U, R, True))


def check_nonfinite(gpu, n, order, t, v, R, node, bad, prec):
    U = np.random.default_rng(2).uniform(0.5, 1.0, (n, R))
    U[node] = bad
    U = U.astype(np.float32) if prec == gpu.FP32 else U
    Y = gpu.SpSymtensor(n, order, t, v).S3TTMc(U, R, True, precision=prec)
    has = np.sum(t == node + 1, axis=1)
    uses = {int(i) - 1 for k, row in enumerate(t) for i in row if has[k] > (i == node + 1)}
    assert 0 < len(uses) < n
    assert {i for i in range(n) if not np.isfinite(Y[i]).any()} == uses
    assert {i for i in range(n) if not np.isfinite(Y[i]).all()} == uses


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("node", [131, 149, 70, 57])
def test_order5_tensor_core_form_nonfinite(gpu, node, bad):
    n, t, v = grouped_tensor()
    check_nonfinite(gpu, n, 5, t, v, 16, node, bad, gpu.FP64)


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("R,prec", [(8, "f32"), (5, "f32"), (3, "f64")])
def test_order4_small_rank_nonfinite(gpu, R, prec, bad):
    """Rows of the warp kernel (over 16 owners) as well as light ones use the bad row of U."""
    rng = np.random.default_rng(3)
    t = [tuple(x) for x in synth.zipf_tuples(4, 40, 3000, 0.5, 5).astype(np.int64) - 1]
    t += [(a, b, 41 + (a + b) % 5, 50) for a, b in itertools.combinations(range(0, 12), 2)]  # row 50: one item
    t += [(50, 51, 52 + k, 60) for k in range(4)]
    t = np.unique(np.sort(np.array(t, np.int64) + 1, axis=1), axis=0).astype(np.uint32)
    v = rng.uniform(0.1, 1.0, t.shape[0])
    for node in (3, 41, 50, 60):
        check_nonfinite(gpu, 62, 4, t, v, R, node, bad, gpu.FP32 if prec == "f32" else gpu.FP64)


@pytest.mark.parametrize("R,prec,tol", [(8, "f32", 5e-6), (12, "f64", 1e-12), (16, "f32", 5e-6)])
def test_order5_without_memory_for_the_groups(gpu, R, prec, tol):
    """The copy of the owners (16 + 8 bytes each) is refused: the CTA kernel runs, and goes on
    doing so on this tensor."""
    n, nnz = 300, 40000
    t = synth.zipf_tuples(5, n, nnz, 0.8, 9)
    v = synth.uniform_values(t.shape[0], 9) + 0.1
    U = np.random.default_rng(R).uniform(0.5, 1.5, (n, R))
    p = gpu.FP32 if prec == "f32" else gpu.FP64
    Uc = U.astype(np.float32) if prec == "f32" else U
    Yo = orc.s3ttmc(5, n, t, v, Uc.astype(np.float64), R, True)
    X = gpu.SpSymtensor(n, 5, t, v)
    X.S3TTMc(np.ones((n, 16)), 16, True)  # FP64 at R = 16: the CTA kernel, its data and the transfer buffers
    with refuse(gpu, 1000, 8 * t.shape[0] * 5):
        Y = X.S3TTMc(Uc, R, True, precision=p)
    assert rows_differ(Y.astype(np.float64), Yo) < tol
    assert np.array_equal(Y, X.S3TTMc(Uc, R, True, precision=p))
    fresh = gpu.SpSymtensor(n, 5, t, v).S3TTMc(Uc, R, True, precision=p)
    assert rows_differ(fresh.astype(np.float64), Yo) < tol
