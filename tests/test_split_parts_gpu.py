"""Split accumulation of wide matrices (more than 148 tiles per frequency), whose slabs are
accumulated in parts: against 64-bit sums, chunked calls against one call, and the scratch
size as a function of the pair count."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import project1_b200 as spx
from project1_b200 import _lib, inputs
from project1_b200.susceptibility import npack

DEV = "cuda:0"


def _case(nbas, npair, nw, real=False):
    g = torch.Generator(DEV).manual_seed(nbas + npair)
    m = torch.randn((nbas, npair), dtype=torch.float64 if real else torch.complex128, device=DEV, generator=g)
    d = torch.rand(npair, dtype=torch.float64, device=DEV, generator=g) * 30 + 0.3
    return m, d, torch.from_numpy(inputs.frequencies(nw)).to(DEV)


def _exact(m, d, om, scale):
    """Packed upper triangles of sum_p M_i conj(M_j) w, in 64 bits."""
    n = m.shape[0]
    j, i = torch.tril_indices(n, n, device=m.device)     # packed order: column j, rows i <= j
    out = []
    for o in om.tolist():
        w = -2.0 * d / (o * o + d * d) * scale
        out.append(((m * w) @ m.mH)[i, j])
    return torch.stack(out), i, j


@pytest.mark.gpu
@pytest.mark.parametrize("nbas,npair,real", [
    (1200, 12288, False), (1200, 12289, False), (1200, 24577, False), (1200, 32768, False), (1200, 46000, False),
    (1121, 13001, False), (2500, 13001, True), (2500, 36000, True)])
def test_parts_against_64_bits(nbas, npair, real):
    """The stated bound: 1e-6 of sqrt(chi_ii chi_jj)."""
    m, d, om = _case(nbas, npair, 2, real)
    out = torch.zeros((2, npack(nbas)), dtype=m.dtype, device=DEV)
    with spx.Context(0) as ctx:
        call = ctx.chi0_accumulate_real_dev if real else ctx.chi0_accumulate_dev
        call(m, d, om, out, scale_all=0.5, precision="split", stats=True)
    ref, i, j = _exact(m, d, om, 0.5)
    diag = ref[:, i == j].real.abs()
    assert ((out - ref).abs() <= 1e-6 * (diag[:, i] * diag[:, j]).sqrt()).all()


@pytest.mark.gpu
@pytest.mark.parametrize("nbas,npair", [(1200, 32768 + 24232), (1140, 32768 + 26000), (1140, 32768 + 13300), (1500, 32768 + 18000)])
def test_host_chunks_equal_one_call(nbas, npair):
    """The host-pointer call runs a slab and the remainder as two chunks, in scratch sized for the
    longer one, and gives the bits of the device call."""
    m, d, om = _case(nbas, npair, 1)
    dev = torch.zeros((1, npack(nbas)), dtype=torch.complex128, device=DEV)
    host = np.zeros((npack(nbas), 1), dtype=np.complex128, order="F")
    with spx.Context(0) as ctx:
        ctx.chi0_accumulate_dev(m, d, om, dev, precision="split", stats=True)
    with spx.Context(0) as ctx:
        ctx.chi0_accumulate(m.cpu().numpy().T, d.cpu().numpy(), om.cpu().numpy(), host, precision="split")
    assert np.array_equal(host.T, dev.cpu().numpy())


@pytest.mark.gpu
def test_kernel_batch_chunks_equal_one_call():
    """A batch of per-slab kernels: eight slabs, then a remainder of two longer parts."""
    nbas, npair = 1200, 8 * 32768 + 24232
    m, d, om = _case(nbas, npair, 1)
    outs = [torch.zeros((1, npack(nbas)), dtype=torch.complex128, device=DEV) for _ in range(2)]
    with spx.Context(0) as ctx:
        ctx.chi0_accumulate_dev(m, d, om, outs[0], precision="split", stats=True)
    with spx.Context(0) as ctx:
        ctx.chi0_batched([dict(nbas=nbas, npair=npair, cprod=m, ediff=d, scale_all=1.0, susceph=outs[1])], om,
                         flags=_lib.SPX_BATCH_KERNELS, stats=True)
    assert torch.equal(outs[0], outs[1])


@pytest.mark.parametrize("nbas", [64, 1140, 1200, 1500, 2000])
@pytest.mark.parametrize("slab", [8192, 32768])
def test_scratch_never_falls_with_the_pair_count(nbas, slab):
    size = getattr(_lib.load(), "_ZN3spx21split_workspace_bytesEliii")
    size.restype, size.argtypes = C.c_size_t, [C.c_int64, C.c_int, C.c_int, C.c_int]
    sizes = [size(p, nbas, 24, slab) for p in range(1, 70000, 61)]
    assert all(a <= b for a, b in zip(sizes, sizes[1:]))
