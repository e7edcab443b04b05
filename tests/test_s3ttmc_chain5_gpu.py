"""Order-5 S3TTMc by groups of the first pivot: rows whose owners and groups sit at
the edges of its sub-groups (16 owners), stages (8 sub-groups) and items (256
owners), against the C oracle.  FP64: the oracle's sums associated differently.
FP32: sums of FP32 products over sub-groups of 16, the bar of the FP32 schedules."""
import numpy as np
import pytest

import oracle_lib as orc
from symprop_b200 import synth

pytestmark = pytest.mark.gpu


def edge_tensor(seed):
    """Rows 20.. of 1 to 600 owners: in one group, each owner a group, and in
    groups of 1 to 12 owners; a row of no owner and repeated ids among them."""
    rng = np.random.default_rng(seed)
    tuples, nxt, row = [], 400, 20
    for owners in (1, 3, 4, 5, 7, 8, 9, 15, 16, 17, 64, 129, 255, 256, 257, 600):
        for shape in range(3):
            for k in range(owners):
                a, b = 100 + k % 37, 140 + (k // 37) % 40
                if shape == 0:
                    tuples.append((0, row, a, b, nxt + k // 100))
                elif shape == 1:
                    tuples.append((row, a, 180 + k % 200, nxt + k, nxt + k))
                else:
                    tuples.append((k % 12, row, a, b, nxt + k // 300))
            nxt += owners + 1 if shape == 1 else 8
            row += 1
    tuples += [(99, 99, 99, 0, 1), (98, 98, 98, 98, nxt)]
    t = np.unique(np.sort(np.array(tuples, np.uint32) + 1, axis=1), axis=0)
    return nxt + 6, t, rng.uniform(-1.0, 1.0, t.shape[0])


def dense_tensor(seed):
    t = synth.zipf_tuples(5, 60, 4000, 1.05, seed)  # over 64 owners a node: FP32 at every rank
    return 60, t, synth.uniform_values(t.shape[0], seed)


def rows_differ(a, b):
    norm = np.linalg.norm(b, axis=1)
    return float(np.max(np.linalg.norm(a - b, axis=1) / np.where(norm == 0, 1.0, norm)))


@pytest.mark.parametrize("make", [edge_tensor, dense_tensor])
@pytest.mark.parametrize("R", [1, 2, 5, 7, 8, 9, 11, 12, 13, 16])
def test_rows_against_oracle(gpu, make, R):
    n, t, v = make(R)
    U = np.random.default_rng(R).uniform(0.5, 1.5, (n, R))
    v = np.abs(v) + 0.1  # no cancellation: the bars hold row by row
    X = gpu.SpSymtensor(n, 5, t, v)
    Y = X.S3TTMc(U, R, True)
    assert rows_differ(Y, orc.s3ttmc(5, n, t, v, U, R, True)) < 1e-12
    assert np.array_equal(Y, X.S3TTMc(U, R, True))
    U32 = U.astype(np.float32)
    Y32 = X.S3TTMc(U32, R, True, precision=gpu.FP32).astype(np.float64)
    assert rows_differ(Y32, orc.s3ttmc(5, n, t, v, U32.astype(np.float64), R, True)) < 5e-6
    full = X.S3TTMc(U, R, False)
    assert np.linalg.norm(full) > 0 and np.isfinite(full).all()


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("node", [0, 30, 101, 141])
def test_nonfinite_factor_row_stays_in_the_rows_that_use_it(gpu, node, bad):
    n, t, v = edge_tensor(1)
    for R, kw in ((12, {}), (8, {"precision": gpu.FP32})):
        U = np.random.default_rng(2).uniform(0.5, 1.0, (n, R))
        U[node] = bad
        U = U.astype(np.float32) if kw else U
        Y = gpu.SpSymtensor(n, 5, t, np.abs(v) + 0.1).S3TTMc(U, R, True, **kw)
        has = np.sum(t == node + 1, axis=1)
        uses = {int(i) - 1 for k, row in enumerate(t) for i in row if has[k] > (i == node + 1)}
        assert {i for i in range(n) if not np.isfinite(Y[i]).any()} == uses
        assert {i for i in range(n) if not np.isfinite(Y[i]).all()} == uses
