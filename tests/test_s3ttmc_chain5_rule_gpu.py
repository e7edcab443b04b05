"""Order-5 S3TTMc in FP32 at R > 12, on either side of the line between the group kernel
(at least one group of owners with the same first pivot to 10 owners) and the CTA kernel,
against the C oracle; both also after the other kernel's ranks ran on the tensor."""
import numpy as np
import pytest

import oracle_lib as orc
from symprop_b200 import synth

pytestmark = pytest.mark.gpu


def groups_per_owner(n, t):
    deg = np.bincount(t.ravel(), minlength=n + 1)
    rank = np.empty(n + 1, np.int64)
    rank[np.argsort(-deg, kind="stable")] = np.arange(n + 1)  # ties by id
    r = np.sort(rank[t.astype(np.int64)], axis=1)
    owners, groups = 0, set()
    for k in range(5):
        own = np.ones(len(t), bool) if k == 0 else r[:, k] != r[:, k - 1]
        rest = np.delete(r, k, axis=1)[own]
        owners += len(rest)
        groups |= set(zip(r[own, k].tolist(), rest[:, 0].tolist()))
    assert owners >= 64 * n
    return len(groups) / owners


@pytest.mark.parametrize("R", [13, 16])
@pytest.mark.parametrize("s,nnz,low,high", [(0.0, 3000, 0.15, 1.0), (0.4, 3000, 0.1, 0.13), (0.4, 4000, 0.09, 0.1),
                                             (1.05, 6000, 0.0, 0.05)])
def test_rows_on_both_sides_of_the_line(gpu, s, nnz, low, high, R):
    n = 60
    t = synth.zipf_tuples(5, n, nnz, s, 3)
    assert low <= groups_per_owner(n, t) <= high
    v = synth.uniform_values(t.shape[0], 1) + 0.1
    U = np.random.default_rng(R).uniform(0.5, 1.5, (n, R)).astype(np.float32)
    Yo = orc.s3ttmc(5, n, t, v, U.astype(np.float64), R, True)
    X = gpu.SpSymtensor(n, 5, t, v)
    first = X.S3TTMc(U, R, True, precision=gpu.FP32)
    for other in (8, 12):
        X.S3TTMc(np.ascontiguousarray(U[:, :other]), other, True, precision=gpu.FP32)
    norm = np.linalg.norm(Yo, axis=1)
    for Y in (first, X.S3TTMc(U, R, True, precision=gpu.FP32)):
        assert float(np.max(np.linalg.norm(Y - Yo, axis=1) / np.where(norm == 0, 1.0, norm))) < 5e-6
