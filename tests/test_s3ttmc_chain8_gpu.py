"""Order-4 pivot-chain S3TTMc at rank <= 8 (one warp per work item): rows whose
owners, prefixes and groups sit at the edges of its batches (32 owners), tiles
(8 prefixes, 4 groups) and items, against the C oracle.  FP64: the oracle's sums
associated differently; FP32: FP64 sums of the FP32 factor rounded once, 2^-24."""
import numpy as np
import pytest

import oracle_lib as orc

pytestmark = pytest.mark.gpu

HUBS = 12


def edge_tensor(seed):
    """Rows 20.. of 17 to 1,100 owners: all in one prefix, each owner a prefix of
    one group, each owner a group, and groups of 1 to 9 prefixes; rows of 0 and 1
    owners and repeated ids among them."""
    rng = np.random.default_rng(seed)
    tuples, heavy, nxt, row = [], [], 400, 20
    for owners in (17, 31, 32, 33, 63, 64, 65, 96, 300, 1100):
        for shape in range(4):
            for k in range(owners):
                fresh = nxt + k  # one new node per owner
                if shape == 0:
                    t = (0, 1, row, fresh)
                elif shape == 1:
                    t = (0, row, 60 + k % 340, fresh)
                elif shape == 2:
                    t = (row, 60 + k % 340, fresh, fresh)
                else:
                    h = k % HUBS
                    t = (h, row, 60 + (k // HUBS) % (1 + h), fresh)
                tuples.append(t)
            heavy.append(row)
            nxt += 1100 if shape == 3 else 0
            row += 1
    tuples += [(row, row, row, nxt), (59, 59, 0, 1)]
    t = np.unique(np.sort(np.array(tuples, np.uint32) + 1, axis=1), axis=0)
    return nxt + 6, t, rng.uniform(-1.0, 1.0, t.shape[0]), heavy


@pytest.fixture
def chain_only(gpu):
    gpu.lib().symprop_s3ttmc_schedule(4)
    yield gpu
    gpu.lib().symprop_s3ttmc_schedule(0)


@pytest.mark.parametrize("R", range(1, 10))
def test_edge_rows_against_oracle(chain_only, R):
    sp = chain_only
    n, t, v, heavy = edge_tensor(R)
    U = np.random.default_rng(R).standard_normal((n, R))
    X = sp.SpSymtensor(n, 4, t, v)
    Y, Yo = X.S3TTMc(U, R, True), orc.s3ttmc(4, n, t, v, U, R, True)
    assert np.all(Y[-4:] == 0.0)
    for i in range(n):
        assert np.linalg.norm(Y[i] - Yo[i]) <= 1e-12 * np.linalg.norm(Yo[i]), i
    if R <= 8:
        U32 = U.astype(np.float32)
        Y32 = X.S3TTMc(U32, R, True, precision=sp.FP32).astype(np.float64)
        Yo = orc.s3ttmc(4, n, t, v, U32.astype(np.float64), R, True)
        for i in heavy:  # coefficients rounded to FP32 as well: 2^-24 of each owner's product
            assert np.linalg.norm(Y32[i] - Yo[i]) <= 1e-6 * np.linalg.norm(Yo[i]), i
    assert np.array_equal(Y, X.S3TTMc(U, R, True))


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("node", [0, 30, 61, 402])  # s_1, the row itself, s_2, s_3
def test_nonfinite_factor_row_stays_in_the_rows_that_use_it(chain_only, node, bad):
    sp = chain_only
    n, t, v, _ = edge_tensor(1)
    U = np.random.default_rng(2).uniform(0.5, 1.0, (n, 8))
    U[node] = bad
    Y = sp.SpSymtensor(n, 4, t, np.abs(v) + 0.1).S3TTMc(U, 8, True)
    has = np.sum(t == node + 1, axis=1)
    uses = {int(i) - 1 for k, row in enumerate(t) for i in row if has[k] > (i == node + 1)}
    assert {i for i in range(n) if not np.isfinite(Y[i]).any()} == uses
    assert {i for i in range(n) if not np.isfinite(Y[i]).all()} == uses
