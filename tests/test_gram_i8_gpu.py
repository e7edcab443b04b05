"""FP64 Gram on the integer tensor cores: sizes at the edges of its tiles
(256 columns), k blocks (128 rows) and chunks, against extended precision.

Bound per entry: every column is rounded at 2^-53 of its largest magnitude in
a chunk (half a unit each), so |C - A^T A|_ij <= 2^-53 sum_k (max_i |a_kj| +
max_j |a_ki|) + 2^-52 |C_ij| per chunk sum and addition (8 of them allowed),
and the scaling doubles the rounding of the result once more."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def gram(gpu, A, sd=None):
    import torch
    n, m = A.shape
    Y = torch.from_numpy(np.ascontiguousarray(A)).cuda()
    s = torch.ones(m, dtype=torch.float64, device="cuda") if sd is None else torch.from_numpy(sd).cuda()
    G = torch.empty((m, m), dtype=torch.float64, device="cuda")
    gpu.gram_device(Y.data_ptr(), n, m, s.data_ptr(), G.data_ptr(), gpu.FP64)
    return G.cpu().numpy()


def check(A, G, cols):
    B = A[:, cols].astype(np.longdouble)
    E = (B.T @ B).astype(np.longdouble)
    mx, s1 = np.abs(A[:, cols]).max(axis=0), np.abs(A[:, cols]).sum(axis=0)
    bound = 2.0**-53 * (mx[:, None] * s1[None, :] + s1[:, None] * mx[None, :]) + 10 * 2.0**-52 * np.abs(E).astype(np.float64)
    d = np.abs(G[np.ix_(cols, cols)].astype(np.longdouble) - E).astype(np.float64)
    assert np.all(d <= bound), (d / np.maximum(bound, 1e-300)).max()


@pytest.mark.parametrize("n,m", [(1536, 320), (1537, 321), (1663, 512), (2048, 514), (40007, 770), (131200, 320)])
def test_sizes(gpu, n, m):
    rng = np.random.default_rng(n + m)
    A = rng.standard_normal((n, m)) * rng.uniform(0.01, 10.0, (n, 1)) ** 2 + rng.standard_normal((1, m))
    G = gram(gpu, A)
    assert np.array_equal(G, G.T)
    cols = np.unique(np.r_[0:16, m - 16:m, rng.integers(0, m, 24)])
    check(A, G, cols)
    sd = rng.uniform(1.0, 5.0, m)
    assert np.array_equal(gram(gpu, A, sd), G * (sd[:, None] * sd[None, :]))


def test_column_scales_zeros_and_extremes(gpu):
    rng = np.random.default_rng(5)
    n, m = 2000, 330
    A = rng.standard_normal((n, m)) * 10.0 ** rng.integers(-150, 150, (1, m))
    A[:, 3] = 0.0
    A[:, 7] *= 10.0 ** rng.uniform(-12, 0, n)
    A[:, 11] = 5e-324 * rng.integers(0, 1000, n)     # subnormal
    A[:, 12] = np.where(rng.random(n) < 0.5, -1, 1) * 1.7e150
    A[0, 13] = 2.0**52 - 0.5                          # halves round to even
    G = gram(gpu, A)
    check(A, G, np.arange(0, 40))
    assert not G[3].any()


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_input_gives_the_floating_point_result(gpu, bad):
    rng = np.random.default_rng(1)
    A = rng.standard_normal((1600, 340))
    A[700, 5] = bad
    G = gram(gpu, A)
    assert np.isnan(G[5]).all() if np.isnan(bad) else np.isinf(G[5, 5])
    keep = np.r_[0:5, 6:340]
    assert np.isfinite(G[np.ix_(keep, keep)]).all()


def test_expired_wait_is_an_error_and_the_next_call_works(gpu):
    A = np.random.default_rng(2).standard_normal((4096, 512))
    good = gram(gpu, A)
    gpu.lib().symprop_debug_set_tc_wait_ns(1)
    try:
        with pytest.raises(gpu.SympropError) as e:
            gram(gpu, A)
        assert e.value.status == gpu.ERR_TIMEOUT
    finally:
        gpu.lib().symprop_debug_set_tc_wait_ns(0)
    assert np.array_equal(gram(gpu, A), good)
