"""The two systematic resamplers of one context share a workspace: a residual call
leaves it where a graph captured from the other call has it, and a residual call
that is first made while the stream is captured needs no allocation."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle_py as O
from tsdf_localization_gb300 import Context
from tsdf_localization_gb300 import _native as N

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


class Cloud:
    def __init__(self, ctx, m, seed):
        self.ctx, self.m = ctx, m
        self.p = np.random.default_rng(seed).normal(size=(m, 7)).astype(np.float32)
        w = np.random.default_rng(seed + 1).gamma(0.8, size=m) + 0.02
        self.p[:, 6] = (w / w.sum()).astype(np.float32)
        self.d = torch.from_numpy(self.p).cuda()
        self.out = torch.zeros((2 * m + 16, 7), device="cuda")
        self.cnt = torch.zeros(1, dtype=torch.int32, device="cuda")

    def call(self, name, u0):
        N.check(getattr(N.lib(), name)(self.ctx.handle, C.c_void_p(self.d.data_ptr()), self.m, u0,
                                       C.c_void_p(self.out.data_ptr()), self.out.shape[0],
                                       C.c_void_p(self.cnt.data_ptr())))

    def check(self, idx):
        self.ctx.sync()
        n = int(self.cnt.item())
        assert n == idx.shape[0] and np.array_equal(self.out[:n].cpu().numpy(), self.p[idx])
        self.out.zero_()
        self.cnt.zero_()
        torch.cuda.synchronize()


def workspace_bytes(ctx):
    a, b = C.c_size_t(), C.c_size_t()
    N.check(N.lib().tsdfl_ctx_workspace_bytes(ctx.handle, C.byref(a), C.byref(b)))
    return b.value


@pytest.mark.parametrize("m", [2_560, 30_011, 100_003])
def test_graph_of_the_one_call_beside_the_other(m):
    ctx, stream = Context(0), torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)
    c = Cloud(ctx, m, m)
    w = c.p[:, 6].copy()
    u = 0.3 / m
    systematic = O.resample_systematic(w, u, cap=2 * m + 16)
    residual = O.resample_residual_systematic(w, 0.3, cap=2 * m + 16)
    torch.cuda.synchronize()
    c.call("tsdfl_resample_systematic_device", u)
    c.check(systematic)
    graphs = {}
    for name, u0 in (("tsdfl_resample_systematic_device", u), ("tsdfl_resample_residual_systematic_device", 0.3)):
        graphs[name] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graphs[name], stream=stream):
            c.call(name, u0)
    before = workspace_bytes(ctx)
    c.call("tsdfl_resample_residual_systematic_device", 0.3)   # now the tables are allocated
    c.check(residual)
    assert workspace_bytes(ctx) > before
    for _ in range(2):
        with torch.cuda.stream(stream):
            graphs["tsdfl_resample_systematic_device"].replay()
        c.check(systematic)
        with torch.cuda.stream(stream):
            graphs["tsdfl_resample_residual_systematic_device"].replay()
        c.check(residual)
    c.call("tsdfl_resample_systematic_device", u)
    c.check(systematic)
    ctx.close()


def test_reserved_context_captures_the_parallel_form():
    m = 100_003
    ctx, stream = Context(0), torch.cuda.Stream()
    ctx.set_stream(stream.cuda_stream)
    ctx.reserve(m, 1_000)
    held = workspace_bytes(ctx)
    c = Cloud(ctx, m, 5)
    residual = O.resample_residual_systematic(c.p[:, 6].copy(), 0.7, cap=2 * m + 16)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    launches = N.lib().tsdfl_launch_count()
    with torch.cuda.graph(g, stream=stream):
        c.call("tsdfl_resample_residual_systematic_device", 0.7)
    assert N.lib().tsdfl_launch_count() - launches == 5 and workspace_bytes(ctx) == held
    with torch.cuda.stream(stream):
        g.replay()
    c.check(residual)
    ctx.close()
