"""Split-leaf S3TTMc schedule (order 6, rank <= 10): every rank it covers, rows
whose owner counts sit at the edges of its stages (16 owners) and work items,
against the C oracle and the level-recursion kernels.  The bars are those of
the other schedules: the sums are the oracle's, associated differently."""
import numpy as np
import pytest

import oracle_lib as orc
from symprop_b200 import synth

pytestmark = pytest.mark.gpu


def rel(a, b):
    return np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b)


def edge_tensor(seed):
    """Rows of 0, 1, 3, 4, 5, 15, 16, 17, 33 and (row 0) several hundred owners,
    tuples with repeated ids among them."""
    rng = np.random.default_rng(seed)
    tuples, nxt = [], 20
    for row, k in enumerate([1, 3, 4, 5, 15, 16, 17, 33], start=1):
        for _ in range(k):  # the row, the hub, one filler node per tuple, small ids repeated
            tuples.append([0, row, nxt, nxt, 10 + rng.integers(0, 3), 13 + rng.integers(0, 4)])
            nxt += 1
    for _ in range(400):
        tuples.append([0, 0, 10 + rng.integers(0, 3), 13 + rng.integers(0, 4), nxt, nxt + 1])
        nxt += 1
    t = np.sort(np.array(tuples, np.uint32) + 1, axis=1)
    return nxt + 6, t, rng.uniform(-1.0, 1.0, t.shape[0])  # the last rows have no owner


@pytest.mark.parametrize("R", range(1, 11))
def test_edge_rows_against_oracle(gpu, R):
    n, t, v = edge_tensor(R)
    U = np.random.default_rng(R).standard_normal((n, R))
    X = gpu.SpSymtensor(n, 6, t, v)
    Yo = orc.s3ttmc(6, n, t, v, U, R, True)
    Y = X.S3TTMc(U, R, True)
    assert rel(Y, Yo) < 1e-12
    assert np.all(Y[-4:] == 0.0)
    for i in range(12):  # short rows by themselves: the hub's norm hides them
        assert np.linalg.norm(Y[i] - Yo[i]) <= 1e-12 * max(np.linalg.norm(Yo[i]), 1e-300), i
    U32 = U.astype(np.float32)
    Y32 = X.S3TTMc(U32, R, True, precision=gpu.FP32)
    # FP64 sums of the FP32 factor, rounded once
    assert rel(Y32, orc.s3ttmc(6, n, t, v, U32.astype(np.float64), R, True)) < 1e-7
    assert np.array_equal(Y, X.S3TTMc(U, R, True))


def test_more_items_than_ctas_and_full_rows(gpu):
    n, R = 1200, 7
    t = synth.zipf_tuples(6, n, 9000, 1.1, 3)
    v = synth.uniform_values(t.shape[0], 3)
    U = np.random.default_rng(0).standard_normal((n, R))
    X = gpu.SpSymtensor(n, 6, t, v)
    assert rel(X.S3TTMc(U, R, True), orc.s3ttmc(6, n, t, v, U, R, True)) < 1e-12
    full = X.S3TTMc(U, R, False)
    gpu.lib().symprop_s3ttmc_schedule(1)
    try:
        rows = X.S3TTMc(U, R, False)
    finally:
        gpu.lib().symprop_s3ttmc_schedule(0)
    assert rel(full, rows) < 1e-12


def test_nan_factor_row_stays_in_the_rows_that_use_it(gpu):
    n, t, v = edge_tensor(1)
    R, bad = 10, 25  # a filler node: row 2 (and the hub) use it
    v[3] = 0.0
    U = np.random.default_rng(2).standard_normal((n, R))
    U[bad] = np.nan
    X = gpu.SpSymtensor(n, 6, t, v)
    Y = X.S3TTMc(U, R, True)
    uses = {int(i) - 1 for row in t for i in row if bad + 1 in row and (i - 1 != bad or np.sum(row == bad + 1) > 1)}
    assert {i for i in range(n) if np.isnan(Y[i]).any()} == uses
