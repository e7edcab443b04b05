"""FP64 column Grams on either side of the line between the FP64 kernels and the integer
tensor cores.  Where the FP64 kernels are faster (odd widths of few rows, some even ones)
the call gives what it gives when the integer kernel's operands are refused; every
entry has the rounding bound of a sum of n products in FP64,
    |C_ij - sum_k a_ki a_kj| <= n 2^-53 sum_k |a_ki| |a_kj| + 4 2^-53 |C_ij|."""
import numpy as np
import pytest

from test_memory_gpu import column_errors, diagonal_error, gram, refuse

pytestmark = pytest.mark.gpu


def rows(n, m):
    import torch
    return torch.randn(n, m, generator=torch.Generator().manual_seed(n + m), dtype=torch.float64).cuda()


@pytest.mark.parametrize("n,m", [(1536, 321), (1537, 333), (2000, 495), (3001, 455), (4000, 321)])
def test_fp64_kernel_where_it_is_faster(gpu, n, m):
    import torch
    Y = rows(n, m)
    G = gram(gpu, Y, gpu.FP64)
    if m < 400:  # (wider: the FP64 kernel's own partial sums are the larger ones)
        with refuse(gpu, 1000, 12 << 20):  # the integer kernel's operands of 1,024 rows
            assert torch.equal(G, gram(gpu, Y, gpu.FP64))
    assert torch.equal(G, G.T)
    assert column_errors(Y, G, [0, 63, 64, m // 2, m - 1]) <= 1.0


@pytest.mark.parametrize("n,m", [(1536, 320), (2000, 330), (8001, 455), (3001, 816), (1600, 2002)])
def test_integer_kernel_where_it_is_faster(gpu, n, m):
    """(diagonal entries within a few units: one rounding a chunk)"""
    Y = rows(n, m)
    G = gram(gpu, Y, gpu.FP64)
    assert column_errors(Y, G, [0, 255, 256, m // 2, m - 1]) <= 1.0
    assert diagonal_error(Y, G, np.arange(0, m, 7)) <= 4.0
