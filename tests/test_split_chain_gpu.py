"""The chained kernels of one-slab split calls: calls queued back to back on one context, so
that each one's kernels meet the last one's in the workspace, give the bits of calls made one
at a time; with and without cut tiles, and inside a captured graph."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import project1_b200 as spx
from project1_b200 import inputs
from project1_b200.susceptibility import npack

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("real", [False, True])
@pytest.mark.parametrize("nbas,npair,nw", [(96, 160, 4), (130, 5000, 3), (403, 700, 24)])
def test_queued_calls(nbas, npair, nw, real):
    dt = torch.float64 if real else torch.complex128
    g = torch.Generator(DEV).manual_seed(nbas)
    om = torch.from_numpy(inputs.frequencies(nw)).to(DEV)
    ms = [torch.randn((nbas, npair), dtype=dt, device=DEV, generator=g) * (k + 1) for k in range(4)]
    ds = [torch.rand(npair, dtype=torch.float64, device=DEV, generator=g) + 0.1 for _ in range(4)]

    def run(ctx, k, out, stream=None, stats=False):
        call = ctx.chi0_accumulate_real_dev if real else ctx.chi0_accumulate_dev
        call(ms[k], ds[k], om, out, precision="split", stream=stream, stats=stats)

    def zeros():
        return [torch.zeros((nw, npack(nbas)), dtype=dt, device=DEV) for _ in range(4)]

    with spx.Context(0) as ctx:
        alone, queued, replayed = zeros(), zeros(), zeros()
        for k in range(4):
            run(ctx, k, alone[k], stats=True)
        torch.cuda.synchronize()
        for _ in range(2):   # two passes into the same outputs: twice the polarisation
            for k in range(4):
                run(ctx, k, queued[k])
        ctx.synchronize()
        torch.cuda.synchronize()
        for a, q in zip(alone, queued):
            assert torch.equal(q, a + a)
        graph, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=s):
            for k in range(4):
                run(ctx, k, replayed[k], stream=s.cuda_stream)
        graph.replay()
        torch.cuda.synchronize()
        for a, q in zip(alone, replayed):
            assert torch.equal(q, a)
