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


@pytest.mark.parametrize("odd", [False, True])
def test_check_before_the_sums(gpu, odd):
    """A width at which the check runs first, over the blocks with the largest rows: rows
    with scales of a power law; columns whose large entry meets a zero, in a row of a
    block that is not among them, go to the FP64 sums."""
    import torch
    n, m = 20011, 2002
    Y = rows(n, m)
    Y *= ((torch.randperm(n, generator=torch.Generator().manual_seed(1)) + 1).double() / n).pow(-0.45).cuda()[:, None]
    if odd:
        low = int(Y.abs().sum(1).view(-1)[: n // 128 * 128].view(-1, 128).sum(1).argmin()) * 128
        Y[low + 3, 4], Y[low + 3, 5] = 1e17, 0.0
        Y[n - 1, m - 1], Y[n - 1, 300] = 1e18, 0.0
    G = gram(gpu, Y, gpu.FP64)
    assert torch.equal(G, G.T)
    assert column_errors(Y, G, [0, 4, 5, 300, m - 1]) <= 1.0
