"""Device memory: an allocation that the device refuses once is tried again after the
library's pool has given its unused memory back.  The refusals are
injected on the host."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
COUNT, BYTES, GRAM_CHUNKS = 1, 2, 3  # SYMPROP_DEBUG_REFUSE_*, SYMPROP_DEBUG_GRAM_CHUNKS


class refuse:
    def __init__(self, gpu, count, least):
        self.set, self.count, self.least = gpu.lib().symprop_debug_set, count, least

    def __enter__(self):
        assert self.set(COUNT, self.count) == 0 and self.set(BYTES, self.least) == 0

    def __exit__(self, *a):
        self.set(BYTES, 0)
        self.set(COUNT, 0)


def gram(gpu, Y, prec):
    import torch
    n, m = Y.shape
    sd = torch.ones(m, dtype=Y.dtype, device="cuda")
    G = torch.empty(m, m, dtype=torch.float64, device="cuda")
    gpu.gram_device(Y.data_ptr(), n, m, sd.data_ptr(), G.data_ptr(), prec)
    return G


@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_one_refusal_changes_nothing(gpu, prec):
    """An FP32 Gram whose workspace is refused once, while the pool holds what earlier
    calls left there (it gives it back: the pool is empty after the retry)."""
    import torch
    Y = torch.randn(20000, 1000, generator=torch.Generator().manual_seed(1), dtype=torch.float64).cuda()
    Y = Y.float() if prec == "f32" else Y
    p = gpu.FP32 if prec == "f32" else gpu.FP64
    good = gram(gpu, Y, p)
    gpu.trim_memory()
    big = torch.randn(8000, 3000, dtype=torch.float64, device="cuda")
    gram(gpu, big, gpu.FP64)  # leaves hundreds of MB in the pool
    del big
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    with refuse(gpu, 1, 8 << 20):
        assert torch.equal(gram(gpu, Y, p), good)
    assert torch.cuda.mem_get_info()[0] - before > (64 << 20)


def column_errors(Y, G, cols):
    """Entries of the columns against extended precision, in units of the FP64 bound."""
    A = Y.cpu().numpy().astype(np.longdouble)
    B = A[:, cols]
    E, T = A.T @ B, np.abs(A).T @ np.abs(B)
    d = np.abs(G[:, torch_index(cols)].cpu().numpy().astype(np.longdouble) - E)
    return float((d / (Y.shape[0] * 2.0**-53 * T + 4 * 2.0**-53 * np.abs(E))).max())


def torch_index(cols):
    import torch
    return torch.as_tensor(cols, device="cuda")


def diagonal_error(Y, G, cols):
    """Median relative error of diagonal entries in units of 2^-53: the integer product
    rounds a chunk's sum once and adds at most some tens of chunks (about 1); an FP64 sum
    of thousands of squares is off by 10 and more (0.4 sqrt(n / 3))."""
    A = Y[:, torch_index(cols)].cpu().numpy().astype(np.longdouble)
    E = (A * A).sum(axis=0)
    d = np.abs(G.diagonal()[torch_index(cols)].cpu().numpy().astype(np.longdouble) - E)
    return float(np.median(d / E) * 2.0**53)


def test_integer_gram_with_little_memory(gpu):
    """Refused operands: smaller launches, in the end the FP64 kernel."""
    import torch
    Y = torch.randn(100000, 330, generator=torch.Generator().manual_seed(2), dtype=torch.float64).cuda()
    for least in (400 << 20, 100 << 20, 16 << 20, 9 << 20):  # the FP64 kernel's own sums take 7 MB
        with refuse(gpu, 1000, least):
            G = gram(gpu, Y, gpu.FP64)
        assert column_errors(Y, G, [0, 200, 329]) <= 1.0, least
        if least >= 16 << 20:  # operands of 1,024 rows: 10 MB
            assert diagonal_error(Y, G, np.arange(0, 330, 3)) <= 4.0, least


@pytest.mark.parametrize("n,m,chunks", [(40007, 770, 5), (131200, 320, 3)])
def test_integer_gram_in_several_launches(gpu, n, m, chunks):
    """The same chunks of rows, one and two to a launch: the same bits."""
    import torch
    Y = torch.randn(n, m, generator=torch.Generator().manual_seed(n), dtype=torch.float64).cuda()
    Y[n - 1, 3], Y[n - 1, 4], Y[0, 5] = 1e18, 0.0, 1e17  # entries for the FP64 sums
    one = gram(gpu, Y, gpu.FP64)
    try:
        for k in range(1, chunks):
            assert gpu.lib().symprop_debug_set(GRAM_CHUNKS, k) == 0
            assert torch.equal(gram(gpu, Y, gpu.FP64), one), k
    finally:
        gpu.lib().symprop_debug_set(GRAM_CHUNKS, 0)
    assert column_errors(Y, one, [0, 3, 4, 5, m - 1]) <= 1.0


def test_operands_of_a_wide_gram_are_bounded(gpu):
    """15,504 columns: the integer product in launches of at most 4.5 GB, of which the
    pool keeps one buffer (and the small ones: column scales, norms, odd entries)."""
    import torch
    n, m = 16384, 15504
    Y = torch.randn(n, m, dtype=torch.float64, device="cuda")
    sd = torch.ones(m, dtype=torch.float64, device="cuda")
    G = torch.empty(m, m, dtype=torch.float64, device="cuda")
    gpu.trim_memory()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    with refuse(gpu, 1000, (9 << 29) + 1):
        gpu.gram_device(Y.data_ptr(), n, m, sd.data_ptr(), G.data_ptr(), gpu.FP64)
    kept = before - torch.cuda.mem_get_info()[0]
    gpu.trim_memory()
    assert kept <= (9 << 29) + (256 << 20), kept
    cols = np.r_[0:20, 7000:7020, m - 20:m]
    assert diagonal_error(Y, G, cols) <= 4.0
    j = torch_index(cols[::8])
    T = Y.abs().T @ Y[:, j].abs()  # the product compared with has the same bound
    assert bool(((G[:, j] - Y.T @ Y[:, j]).abs() <= 2 * (n + 4) * 2.0**-53 * T).all())
