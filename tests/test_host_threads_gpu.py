"""The host-pointer call's threads: they sleep while they have nothing to do, chunked and pinned
calls give the sums of the device call, and errors leave the output as it was."""
import resource
import time

import numpy as np
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
    return m, d, inputs.frequencies(nw)


def test_threads_sleep_beside_a_pinned_call():
    """At most one wake per millisecond and thread (they block about six times in a call); polling
    every 20 us or so made more than ten."""
    nbas, npair, nw = 400, 150000, 24
    m, d, om = _case(nbas, npair, nw)
    mh = torch.empty((nbas, npair), dtype=torch.complex128, pin_memory=True)
    mh.copy_(m)
    out = np.zeros((npack(nbas), nw), dtype=np.complex128, order="F")
    with spx.Context(0) as ctx:
        for _ in range(2):
            before, t = resource.getrusage(resource.RUSAGE_SELF).ru_nvcsw, time.perf_counter()
            ctx.chi0_accumulate_host_ptr(mh.data_ptr(), npair, npair, nbas, d.cpu().numpy(), om, out)
            waits, ms = resource.getrusage(resource.RUSAGE_SELF).ru_nvcsw - before, 1e3 * (time.perf_counter() - t)
    assert ms > 20 and waits <= 7 * ms


@pytest.mark.parametrize("nbas,npair,nw", [(1, 1, 1), (3, 5000, 2), (130, 7001, 9), (260, 40000, 16)])
@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("precision", ["fp64", "split"])
def test_host_sums(nbas, npair, nw, pinned, precision):
    """Chunks change the order of the FP64 sums only: (P + 8) roundings of sum |M_i||M_j||w| on
    either side. Split chunks are whole slabs: the same bits."""
    m, d, om = _case(nbas, npair, nw)
    dev = torch.zeros((nw, npack(nbas)), dtype=torch.complex128, device=DEV)
    rng = np.random.default_rng(nbas)
    out = np.asfortranarray(rng.standard_normal((npack(nbas), nw)) + 1j * rng.standard_normal((npack(nbas), nw)))
    was = out.copy()
    mh = torch.empty((nbas, npair), dtype=torch.complex128, pin_memory=pinned)
    mh.copy_(m)
    dh = d.cpu().numpy()
    with spx.Context(0) as ctx:
        ctx.chi0_accumulate_dev(m, d, torch.from_numpy(om).to(DEV), dev, precision=precision, stats=True)
        ctx.chi0_accumulate_host_ptr(mh.data_ptr(), npair, npair, nbas, dh, om, out, precision=precision)
    add = dev.cpu().numpy().T
    if precision == "split":
        assert np.array_equal(out, was + add)
        return
    w = 2.0 * dh[:, None] / (dh[:, None] ** 2 + np.asarray(om)[None, :] ** 2)
    s = np.sqrt((np.abs(mh.numpy()) ** 2) @ w)
    j, i = np.tril_indices(nbas)
    bound = np.sqrt(2) * (2 * (npair + 8) + 2) * 2.0 ** -53 * s[i] * s[j] + 2.0 ** -51 * np.abs(was)
    assert np.all(np.abs(out - was - add) <= bound)


def test_failed_call_adds_nothing():
    nbas, npair, nw = 200, 20000, 4
    m, d, om = _case(nbas, npair, nw)
    out = np.full((npack(nbas), nw), 2.0 - 1.0j, dtype=np.complex128, order="F")
    with spx.Context(0, workspace_limit=1 << 20) as ctx:
        with pytest.raises(Exception):
            ctx.chi0_accumulate(m.cpu().numpy().T, d.cpu().numpy(), om, out)
    assert np.all(out == 2.0 - 1.0j)
