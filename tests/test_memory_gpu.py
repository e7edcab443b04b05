"""Device memory: an allocation that the device refuses once is tried again after the
library's pool has given its unused memory back.  The refusals are
injected on the host."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
COUNT, BYTES = 1, 2  # SYMPROP_DEBUG_REFUSE_*


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
