"""Split accumulation: items cut along the pairs, slab statistics in clusters, staged real
quantizer, default slabs. Sums of digit products are exact integers, so routes that differ
only in how the work is dealt agree bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle
import project1_b200 as spx
from project1_b200 import _lib, inputs
from project1_b200.susceptibility import npack

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ctx():
    c = spx.Context(0)
    yield c
    c.close()


def _case(nbas, npair, nw, real=False):
    rng = np.random.default_rng(nbas * 101 + npair + nw)
    m = rng.standard_normal((npair, nbas))
    if not real:
        m = m + 1j * rng.standard_normal((npair, nbas))
    m = np.asfortranarray(m / np.sqrt(nbas))
    d = rng.uniform(0.5, 40.0, npair)
    d[rng.integers(npair)] = 2e-7
    om = inputs.frequencies(nw)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)
    return m, d, om, t(m.T), t(d), t(om)


def _norm_error(got, ref, n):
    """The normalised error the split path states its 1e-6 bound in."""
    d = np.abs(ref[[j * (j + 1) // 2 + j for j in range(n)]].real)
    iu, ju = np.triu_indices(n)
    idx = ju * (ju + 1) // 2 + iu
    return np.max(np.abs(got - ref)[idx] / np.sqrt(d[iu] * d[ju]))


@pytest.mark.parametrize("nbas,npair,nw", [
    (1, 5000, 1), (63, 30000, 1), (96, 160, 4), (200, 40000, 3), (403, 9001, 12), (257, 2500, 30), (1000, 3000, 2),
    (80, 65, 5)])
def test_cut_items_equal_whole_items(ctx, nbas, npair, nw):
    m, d, om, md, dd, omd = _case(nbas, npair, nw)
    out = torch.zeros((nw, npack(nbas)), dtype=torch.complex128, device=DEV)
    ctx.chi0_accumulate_dev(md, dd, omd, out, scale_all=0.5, precision="split", stats=True)
    # the per-slab kernels of a batch deal whole items
    whole = torch.zeros_like(out)
    q = dict(nbas=nbas, npair=npair, cprod=md, ediff=dd, scale_all=0.5, susceph=whole)
    ctx.chi0_batched([q], omd, flags=_lib.SPX_BATCH_KERNELS | _lib.SPX_BATCH_NOGRAPH, stats=True)
    assert torch.equal(out, whole)
    # given weights: the statistics read them instead of forming them
    w = torch.empty((nw, npair), dtype=torch.float64, device=DEV)
    ctx.weights_dev(dd, omd, w, scale_all=0.5)
    given = torch.zeros_like(out)
    ctx.chi0_accumulate_w_dev(md, w, given, precision="split", stats=True)
    assert torch.equal(out, given)
    if nbas * nbas * npair * nw < 4e9:
        ref = oracle.chi0(m, oracle.weights(d, om, None, 0.5), accurate=True)
        assert _norm_error(out.cpu().numpy().T, ref, nbas) <= 1e-6


@pytest.mark.parametrize("nbas,npair,nw", [(1, 64, 1), (7, 65, 25), (128, 20000, 2), (161, 3001, 5), (300, 17000, 4)])
def test_real_split_edges(nbas, npair, nw):
    m, d, om, md, dd, omd = _case(nbas, npair, nw, real=True)
    outs = []
    for variant in (0, 1, 5):
        out = torch.zeros((nw, npack(nbas)), dtype=torch.float64, device=DEV)
        with spx.Context(0, split_variant=variant) as c:
            c.chi0_accumulate_real_dev(md, dd, omd, out, scale_all=0.5, precision="split", stats=True)
        outs.append(out)
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    ref = oracle.chi0_real(m, oracle.weights(d, om, None, 0.5))
    assert _norm_error(outs[0].cpu().numpy().T, ref, nbas) <= 1e-6


def test_signs_meet_across_the_cluster(ctx):
    """One positive weight among negative ones, in the last CTA's share of the slab: the
    frequency must take the signed operand.

    Bound: an operand is off by half a unit e_i = s_i sqrt(wmax) / (127 2^17) per part (s_i the
    column's largest |Re|, |Im|), and the dropped digit orders are at most
    (2 128^2 2^8 + 128^2) / (127 2^16)^2 s_i s_j wmax per real product; two real products per
    part and pair, P pairs. A wrong sign would be off by 2 w |M_i M_j| of one pair."""
    nbas, npair = 40, 3000
    m, _, _, md, _, _ = _case(nbas, npair, 1)
    w = np.full((npair, 1), -1.0)
    w[-1] = 2.0
    m[-1] = (1 + 1j) * np.abs(m).max()      # the pair of that weight is the columns' largest
    md[:, -1] = torch.from_numpy(m[-1].copy()).to(DEV)
    out = torch.zeros((1, npack(nbas)), dtype=torch.complex128, device=DEV)
    ctx.chi0_accumulate_w_dev(md, torch.from_numpy(np.ascontiguousarray(w.T)).to(DEV), out, precision="split")
    ref = oracle.chi0(m, w, accurate=True)
    s = np.maximum(np.abs(m.real), np.abs(m.imag)).max(axis=0)
    per = 2 * (2 * 2.0 ** -17 / 127 + (2 * 128.0 ** 2 * 256 + 128.0 ** 2) / (127.0 * 65536) ** 2)
    iu, ju = np.triu_indices(nbas)
    err = np.abs(out.cpu().numpy().T - ref)[ju * (ju + 1) // 2 + iu, 0]
    bound = np.sqrt(2.0) * npair * per * 2.0 * s[iu] * s[ju]
    wrong = 2 * 2.0 * np.abs(m[-1, iu] * m[-1, ju])
    assert np.all(bound < 0.1 * wrong)      # the bound tells a wrong sign
    assert np.all(err <= bound)
