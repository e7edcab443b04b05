"""S3TTMc calls captured into a CUDA graph, when an earlier call on the tensor had
another precision or rank: nothing may be allocated or waited for during the capture,
and later calls must leave the buffers that a graph holds where they are."""
import numpy as np
import pytest

import oracle_lib as orc
from symprop_b200 import synth

pytestmark = pytest.mark.gpu
TOL = {"f64": 1e-12, "f32": 1e-5}


class Call:
    def __init__(self, gpu, X, R, prec, seed=0, packed=True):
        import torch
        self.gpu, self.X, self.R, self.prec, self.packed = gpu, X, R, prec, packed
        self.U = np.random.default_rng(seed).standard_normal((X.dim(), R))
        dt = torch.float64 if prec == "f64" else torch.float32
        self.dU = torch.from_numpy(self.U).to(dt).cuda()
        self.Y = torch.full((X.dim(), X.ncols(R, packed)), float("nan"), dtype=dt, device="cuda")
        torch.cuda.synchronize()

    def run(self, stream=0):
        p = self.gpu.FP64 if self.prec == "f64" else self.gpu.FP32
        self.X.s3ttmc_device(self.dU.data_ptr(), self.R, self.Y.data_ptr(), self.packed, p, stream)

    def eager(self):
        import torch
        self.run()
        torch.cuda.synchronize()
        return self

    def capture(self):
        import torch
        g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        with torch.cuda.graph(g, stream=s):
            self.run(s.cuda_stream)
        return g

    def check(self, t, v):
        import torch
        torch.cuda.synchronize()
        Yo = orc.s3ttmc(self.X.order(), self.X.dim(), t, v, self.U, self.R, self.packed)
        Y = self.Y.double().cpu().numpy().reshape(Yo.shape)
        assert np.linalg.norm(Y - Yo) <= TOL[self.prec] * np.linalg.norm(Yo)


def tensor(gpu, order, n, nnz, s=1.1, seed=1):
    t = synth.zipf_tuples(order, n, nnz, s, seed)
    v = synth.uniform_values(t.shape[0], seed)
    return gpu.SpSymtensor(n, order, t, v), t, v


@pytest.mark.parametrize("n,nnz", [(200, 4000), (900, 3000)])  # 100 and 17 owners a node
@pytest.mark.parametrize("first,then", [((16, "f64"), (16, "f32")), ((16, "f32"), (16, "f64")), ((11, "f64"), (11, "f32")),
                                        ((11, "f32"), (11, "f64")), ((8, "f64"), (8, "f32"))])
def test_order5_other_precision(gpu, n, nnz, first, then):
    X, t, v = tensor(gpu, 5, n, nnz)
    Call(gpu, X, *first).eager().check(t, v)
    c = Call(gpu, X, *then)
    g = c.capture()
    g.replay()
    c.check(t, v)
    c2 = Call(gpu, X, *then, seed=5).eager()  # and afterwards without a capture
    c2.check(t, v)


@pytest.mark.parametrize("R0,R1", [(9, 8), (16, 5), (8, 8)])
def test_order4_smaller_rank(gpu, R0, R1):
    """Ranks up to 8 have a kernel and a list of work items of their own."""
    X0, t0, v0 = tensor(gpu, 4, 50, 2000, seed=3)
    Call(gpu, X0, R1, "f64").eager()  # the rank's index table, kept by the process
    X, t, v = tensor(gpu, 4, 60, 4000, s=0.0, seed=2)  # no light rows
    Call(gpu, X, R0, "f64").eager().check(t, v)
    c = Call(gpu, X, R1, "f64")
    g = c.capture()
    g.replay()
    c.check(t, v)


def test_order4_graph_outlives_a_call_at_a_smaller_rank(gpu):
    X, t, v = tensor(gpu, 4, 40, 20000, s=0.0, seed=4)  # 2,000 owners a row: split rows at any rank
    c = Call(gpu, X, 9, "f64").eager()
    g = c.capture()
    Call(gpu, X, 8, "f64").eager().check(t, v)
    import torch
    fill = torch.full((64 << 20,), float("nan"), device="cuda")  # memory freed by that call would be here
    c.Y.fill_(float("nan"))
    g.replay()
    c.check(t, v)
    assert torch.isnan(fill).all()


@pytest.mark.parametrize("R,prec", [(8, "f64"), (5, "f32"), (10, "f32")])
def test_order6(gpu, R, prec):
    """Rows of both kinds (at most 8 owners, more); a capture keeps no stream from other calls."""
    import torch
    X, t, v = tensor(gpu, 6, 400, 900, s=1.1, seed=6)
    X2, t2, v2 = tensor(gpu, 6, 300, 800, s=1.1, seed=7)
    c, o = Call(gpu, X, R, prec).eager(), Call(gpu, X2, R, prec).eager()
    g, s, s2 = torch.cuda.CUDAGraph(), torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.graph(g, stream=s, capture_error_mode="relaxed"):
        c.run(s.cuda_stream)
        o.run(s2.cuda_stream)
    c.Y.fill_(float("nan"))
    g.replay()
    c.check(t, v)
    o.check(t2, v2)
