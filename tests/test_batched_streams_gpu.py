"""Split batches that run q by q, on several streams of one context: two batches beside each
other, a batch beside single calls, a batch captured in a graph. Each gives the bits it
gives alone."""
import pytest

torch = pytest.importorskip("torch")

import project1_b200 as spx
from project1_b200 import inputs
from project1_b200.susceptibility import npack

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
NW = 8


def _qs(shapes, seed):
    g = torch.Generator(DEV).manual_seed(seed)
    return [dict(nbas=n, npair=p, scale_all=0.5,
                 ediff=torch.rand(p, dtype=torch.float64, device=DEV, generator=g) * 30 + 0.3,
                 cprod=torch.randn((n, p), dtype=torch.complex128, device=DEV, generator=g),
                 susceph=torch.zeros((NW, npack(n)), dtype=torch.complex128, device=DEV)) for n, p in shapes]


SETS = [[(400, 9000), (300, 20000), (350, 16384)], [(330, 18000), (500, 5000)]]


@pytest.fixture(scope="module")
def case():
    om = torch.from_numpy(inputs.frequencies(NW)).to(DEV)
    sets = [_qs(s, k) for k, s in enumerate(SETS)]
    alone = []
    with spx.Context(0) as ctx:
        for qs in sets:
            assert ctx.chi0_batched(qs, om, stats=True)["kernel_launches"] > len(qs)   # q by q
            alone.append([q["susceph"].clone() for q in qs])
    return om, sets, alone


def _zero(sets):
    for qs in sets:
        for q in qs:
            q["susceph"].zero_()
    torch.cuda.synchronize()


def _check(qs, ref):
    for q, r in zip(qs, ref):
        assert torch.equal(q["susceph"], r)


def test_two_batches_on_two_streams(case):
    om, sets, alone = case
    streams = [torch.cuda.Stream() for _ in sets]
    with spx.Context(0) as ctx:
        for order in ((0, 1), (1, 0), (0, 1)):
            _zero(sets)
            for k in order:
                ctx.chi0_batched(sets[k], om, stream=streams[k].cuda_stream)
            torch.cuda.synchronize()
            for qs, ref in zip(sets, alone):
                _check(qs, ref)
        ctx.synchronize()


@pytest.mark.parametrize("precision", ["split", "fp64"])
def test_batch_beside_single_calls(case, precision):
    om, sets, alone = case
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    q = _qs([(420, 40000)], 9)[0]
    one = torch.zeros_like(q["susceph"])

    def single(ctx, out, stream=None):
        ctx.chi0_accumulate_dev(q["cprod"], q["ediff"], om, out, precision=precision, stream=stream, stats=stream is None)

    with spx.Context(0) as ctx:
        single(ctx, one)
    with spx.Context(0) as ctx:
        single(ctx, torch.zeros_like(one))
        for first in (0, 1, 0):
            _zero([sets[0], [q]])
            if first:
                single(ctx, q["susceph"], b.cuda_stream)
            ctx.chi0_batched(sets[0], om, stream=a.cuda_stream)
            if not first:
                single(ctx, q["susceph"], b.cuda_stream)
            torch.cuda.synchronize()
            assert torch.equal(q["susceph"], one)
            _check(sets[0], alone[0])
        ctx.synchronize()


def test_captured_batch(case):
    om, sets, alone = case
    with spx.Context(0) as ctx:
        for qs in sets:
            ctx.chi0_batched(qs, om, stats=True)
        graph, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=s):
            for qs in sets:
                ctx.chi0_batched(qs, om, stream=s.cuda_stream)
        for _ in range(2):
            _zero(sets)
            graph.replay()
            torch.cuda.synchronize()
            for qs, ref in zip(sets, alone):
                _check(qs, ref)
