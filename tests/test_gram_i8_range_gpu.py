"""FP64 column Grams of columns with a wide range, through gram_device: every entry
has the rounding bound of a sum of n products in FP64,
    |C_ij - sum_k a_ki a_kj| <= n 2^-53 sum_k |a_ki| |a_kj| + 4 2^-53 |C_ij|
(the last term: chunk sums added, the scaling by 1), whichever kernel forms it.
Sums in extended precision."""
import numpy as np
import pytest

from test_gram_i8_gpu import gram

pytestmark = pytest.mark.gpu


def check(A, G, cols):
    B = A[:, cols].astype(np.longdouble)
    E, T = B.T @ B, np.abs(B).T @ np.abs(B)
    bound = A.shape[0] * 2.0**-53 * T + 4 * 2.0**-53 * np.abs(E)
    d = np.abs(G[np.ix_(cols, cols)].astype(np.longdouble) - E)
    assert np.all(d <= bound), float((d / np.maximum(bound, 1e-4900)).max())


@pytest.mark.parametrize("n,m", [(1536, 320), (2000, 330), (40007, 515)])
def test_large_entries_in_different_rows(gpu, n, m):
    """Few odd columns among ordinary ones: one entry far above the others, in a row
    where other columns are zero or small."""
    rng = np.random.default_rng(n)
    A = rng.standard_normal((n, m))
    A[0, 5], A[0, 6] = 1e17, 0.0
    A[:, 7], A[:, 8] = 1e-17, 1.0
    A[0, 7], A[0, 8] = 1.0, 0.0
    A[n - 1, m - 1], A[n - 1, 9] = 3e20, 1e-30
    A[:, 10] *= 10.0 ** rng.uniform(-16, 0, n)
    G = gram(gpu, A)
    assert np.array_equal(G, G.T)
    check(A, G, np.r_[0:16, 254:258, m - 8:m])


def test_every_entry_of_its_own_scale(gpu):
    """Magnitudes spread over 16 decades independently: many entries to be summed in FP64."""
    rng = np.random.default_rng(3)
    A = rng.standard_normal((3001, 322)) * 10.0 ** rng.uniform(-16, 0, (3001, 322))
    A[:, ::3] = 0.0
    A[rng.integers(0, 3001, 108), np.arange(0, 322, 3)] = 1e9
    check(A, gram(gpu, A), np.r_[0:40, 300:322])


def test_columns_without_common_rows(gpu):
    """Blocks of columns with entries in disjoint rows, and noise far below elsewhere."""
    rng = np.random.default_rng(4)
    n, m = 4096, 384
    A = 1e-14 * rng.standard_normal((n, m))
    for b in range(4):
        A[b * 1024:(b + 1) * 1024, b * 96:(b + 1) * 96] = rng.standard_normal((1024, 96))
    check(A, gram(gpu, A), np.arange(0, m, 6))


def test_wide_range_in_the_last_rows_only(gpu):
    """Three chunks of rows: only the last one has a column that needs the FP64 sums."""
    rng = np.random.default_rng(5)
    n, m = 131200, 320
    A = rng.standard_normal((n, m))
    A[n - 1, 3], A[n - 1, 4] = 1e18, 0.0
    G = gram(gpu, A)
    check(A, G, np.r_[0:8, 316:320])
