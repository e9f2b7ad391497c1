"""The partial tiles of cut accumulations have a buffer of their own: no call grows the workspace
for them, so a call whose mandatory scratch fits runs under capture, leaves captured calls
valid, and reports nothing."""
import pytest

torch = pytest.importorskip("torch")

import project1_b200 as spx
from project1_b200 import inputs
from project1_b200.susceptibility import npack

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _case(nbas, npair, nw):
    g = torch.Generator(DEV).manual_seed(nbas + npair)
    m = torch.randn((nbas, npair), dtype=torch.complex128, device=DEV, generator=g)
    d = torch.rand(npair, dtype=torch.float64, device=DEV, generator=g) * 30 + 0.3
    return m, d, torch.from_numpy(inputs.frequencies(nw)).to(DEV), torch.zeros((nw, npack(nbas)), dtype=torch.complex128, device=DEV)


def _capture(fn):
    graph, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=s):
        fn(s.cuda_stream)
    return graph


@pytest.mark.parametrize("first", ["accumulate", "dielec"])
def test_smaller_calls_are_captured_in_a_grown_workspace(first):
    """Weights of 40000 pairs at 8 frequencies (or the scratch of an inverse) hold those of 3000 at
    24, and the head and wings, which need none."""
    m, d, om, out = _case(60, 3000, 24)
    alone = torch.zeros_like(out)
    w = torch.rand((24, 3000), dtype=torch.float64, device=DEV)
    heads = [torch.zeros((24, 6), dtype=torch.complex128, device=DEV) for _ in range(2)]
    wings = [torch.zeros((24, 60, 3), dtype=torch.complex128, device=DEV) for _ in range(2)]
    with spx.Context(0) as ctx:
        ctx.chi0_accumulate_dev(m, d, om, alone, stats=True)
        ctx.headwings_dev(m, m[:3], w, heads[0], wings[0])
        ctx.synchronize()
    with spx.Context(0) as ctx:
        if first == "accumulate":
            a = _case(40, 40000, 8)
            ctx.chi0_accumulate_dev(*a, stats=True)
        else:
            chi = torch.zeros((2, npack(300)), dtype=torch.complex128, device=DEV)
            ctx.dielec_dev(chi, torch.ones(300, dtype=torch.float64, device=DEV))
            ctx.synchronize()

        def run(s):
            ctx.chi0_accumulate_dev(m, d, om, out, stream=s)
            ctx.headwings_dev(m, m[:3], w, heads[1], wings[1], stream=s)
        graph = _capture(run)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, alone)
        assert torch.equal(heads[0], heads[1]) and torch.equal(wings[0], wings[1])


def test_captured_call_outlives_calls_that_need_no_more():
    """Both precisions; the calls between capture and replay need other partial tiles but no larger
    workspace."""
    m, d, om, out = _case(150, 30000, 6)
    expected = torch.zeros_like(out)
    with spx.Context(0) as ctx:
        ctx.chi0_accumulate_dev(m, d, om, expected, precision="split", stats=True)
        ctx.chi0_accumulate_dev(m, d, om, expected, stats=True)

        def run(s):
            ctx.chi0_accumulate_dev(m, d, om, out, precision="split", stream=s)
            ctx.chi0_accumulate_dev(m, d, om, out, stream=s)
        graph = _capture(run)
        for nbas, npair, nw in [(100, 1000, 24), (20, 5000, 12), (33, 700, 1)]:
            b = _case(nbas, npair, nw)
            for precision in ("fp64", "split"):
                ctx.chi0_accumulate_dev(*b, precision=precision, stats=True)
            r = b[0].real.contiguous()
            ctx.chi0_accumulate_real_dev(r, b[1], b[2], torch.zeros((nw, npack(nbas)), dtype=torch.float64, device=DEV),
                                         stats=True)
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, expected)


def test_limits_leave_no_message_and_refuse_nothing():
    """Limits from the mandatory scratch upwards: the call runs, with or without partial tiles,
    and no error text is left behind."""
    npair, nw = 5000, 24
    m, d, om, out = _case(120, npair, nw)
    need = 8 * nw * ((npair + 15) // 16 * 16)
    big = _case(120, 200000, nw)
    for limit in (need, need + 10**7, 3 * 10**7, 5 * 10**7, 10**8):
        with spx.Context(0, workspace_limit=limit) as ctx:
            out.zero_()
            ctx.chi0_accumulate_dev(m, d, om, out, stats=True)
            assert ctx.lib.spx_last_error(ctx.handle) == b""
            if limit >= 8 * nw * 200000:
                ctx.chi0_accumulate_dev(*big, stats=True)
                assert ctx.lib.spx_last_error(ctx.handle) == b""
            assert torch.isfinite(torch.view_as_real(out)).all()
