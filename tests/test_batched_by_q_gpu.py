"""Split batches of given products that leave kernel and slab open: q by q through the
one-call kernels, the same bits as the persistent schedule (which an explicit slab of the same
size, or a workspace limit below the largest q's scratch, still selects)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import project1_b200 as spx
from project1_b200 import _lib, inputs
from project1_b200.susceptibility import npack

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _qs(shapes, nw):
    g = torch.Generator(DEV).manual_seed(len(shapes) * 100 + nw)
    qs = []
    for i, (n, p) in enumerate(shapes):
        d = torch.rand(max(p, 1), dtype=torch.float64, device=DEV, generator=g) * 30 + 0.3
        if i % 2:
            d[::7] *= -1.0
        q = dict(nbas=n, npair=p, ediff=d, scale_all=0.5,
                 cprod=torch.randn((n, p + 3), dtype=torch.complex128, device=DEV, generator=g),
                 susceph=torch.zeros((nw, npack(n)), dtype=torch.complex128, device=DEV))
        if i == 1:
            q["wscale"] = torch.rand(max(p, 1), dtype=torch.float64, device=DEV, generator=g)
        qs.append(q)
    return qs


@pytest.mark.parametrize("shapes,nw", [([(200, 9000), (65, 16384), (130, 16385), (7, 40)], 3),
                                       ([(40, 300), (90, 0), (1, 33000), (403, 700)], 24),
                                       ([(500, 1500)], 1)])
def test_by_q_equals_persistent(shapes, nw):
    om = torch.from_numpy(inputs.frequencies(nw)).to(DEV)
    qs = _qs(shapes, nw)
    outs = []
    for limit, slab, flags, launches in [(0, 0, 0, None), (0, 0, _lib.SPX_BATCH_NOGRAPH, None), (0, 16384, 0, 1),
                                         (1 << 16, 0, 0, 1)]:
        for q in qs:
            q["susceph"].zero_()
            q["slab_pairs"] = slab
        with spx.Context(0, workspace_limit=limit) as ctx:
            st = ctx.chi0_batched(qs, om, flags=flags, stats=True)
        assert st["kernel_launches"] == 1 if launches else st["kernel_launches"] > 1
        outs.append([q["susceph"].clone() for q in qs])
    for o in outs[1:]:
        for a, b in zip(outs[0], o):
            assert torch.equal(a, b)
    assert all(torch.isfinite(torch.view_as_real(a)).all() for a in outs[0])
