"""Order-5 S3TTMc in FP32 (group kernel): the four terms of an entry are added in FP64.
With integer U whose products and sums are exact in FP32 up to those terms, every
entry must be the exact value rounded once."""
import itertools

import numpy as np
import pytest

import oracle_lib as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("R", [4, 7, 8])
def test_terms_are_rounded_once(gpu, R):
    rng = np.random.default_rng(R)
    n = 5
    t = np.arange(1, n + 1, dtype=np.uint32)[None, :]
    # row 5: leaf {1, 2, 3, 4}, pivot 1 (equal degrees: by id).  |U| <= 127 keeps
    # the sums over the orderings of {2, 3, 4} below 2^24, powers of two keep
    # their products with U[1] exact; the entries need up to 36 bits.
    U = rng.integers(-127, 128, (n, R)).astype(np.float64)
    U[0] = 2.0 ** rng.integers(0, 12, R)
    q = np.array(list(itertools.combinations_with_replacement(range(R), 4)))
    E = np.zeros(len(q))
    for p in itertools.permutations(range(4)):
        E += np.prod([U[p[k]][q[:, k]] for k in range(4)], axis=0)  # exact: below 2^53
    X = gpu.SpSymtensor(n, 5, t, np.ones(1))
    Yo = orc.s3ttmc(5, n, t, np.ones(1), U, R, True)
    np.testing.assert_array_equal(Yo[4], E)
    Y = X.S3TTMc(U.astype(np.float32), R, True, precision=gpu.FP32)
    np.testing.assert_array_equal(Y[4], E.astype(np.float32))
