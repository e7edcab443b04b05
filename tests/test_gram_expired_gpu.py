"""A tensor-core Gram in which the wait of one warp for its sums runs out, whichever
warp it is, ends with a status: the rows it did not store are never taken for
results.  The wait is declared expired by the failure-injection hook; the sums
are in fact complete, so nothing is left in flight."""
import pytest

pytestmark = pytest.mark.gpu
KEY = 0  # SYMPROP_DEBUG_TC_EXPIRED_WARP


@pytest.mark.parametrize("prec,warps", [("f64", 8), ("f32", 4)])
def test_each_warp(gpu, prec, warps):
    import torch
    n, m = 2048, 330
    dt = torch.float64 if prec == "f64" else torch.float32
    Y = torch.randn(n, m, generator=torch.Generator().manual_seed(3), dtype=dt).cuda()
    sd = torch.ones(m, dtype=dt, device="cuda")
    G = torch.empty(m, m, dtype=torch.float64, device="cuda")

    def run():
        gpu.gram_device(Y.data_ptr(), n, m, sd.data_ptr(), G.data_ptr(), gpu.FP64 if prec == "f64" else gpu.FP32)
        return G.clone()

    good = run()
    try:
        for w in range(warps):
            assert gpu.lib().symprop_debug_set(KEY, w + 1) == 0
            with pytest.raises(gpu.SympropError) as e:
                run()
            assert e.value.status == gpu.ERR_TIMEOUT, w
    finally:
        gpu.lib().symprop_debug_set(KEY, 0)
    assert torch.equal(run(), good)
    assert gpu.lib().symprop_debug_set(99, 1) == gpu.ERR_INVALID
