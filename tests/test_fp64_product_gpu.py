"""The product-first FP64 accumulation (more than four frequencies): tile, chunk and
frequency-group edges, cut and whole tiles, against the extended-precision oracle."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle
import project1_b200 as spx
from project1_b200 import inputs
from project1_b200.susceptibility import npack

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _case(nbas, npair, nw, pad, mixed):
    rng = np.random.default_rng(nbas * 7919 + npair * 31 + nw)
    m = np.asfortranarray((rng.standard_normal((npair, nbas)) + 1j * rng.standard_normal((npair, nbas)))
                          / np.sqrt(nbas))
    md = torch.full((nbas, npair + pad), 3.0 + 4.0j, dtype=torch.complex128, device=DEV)  # padding is not read
    md[:, :npair] = torch.from_numpy(np.ascontiguousarray(m.T)).to(DEV)
    if mixed:
        w = rng.standard_normal((npair, nw))
        return m, md, w, None, None
    d = rng.uniform(0.5, 40.0, npair)
    d[rng.integers(npair)] = 3e-7
    om = inputs.frequencies(nw)
    return m, md, oracle.weights(d, om), torch.from_numpy(d).to(DEV), torch.from_numpy(om).to(DEV)


def _check(got, m, w):
    """Every term carries at most 6 roundings (product, weight, weight times product) and the
    sum of P terms in any order at most P - 1: |error| <= (P + 8) 2^-53 sum_p |M_i||M_j||w|
    per part, bounded by Cauchy-Schwarz with |w|-weighted column norms."""
    ref = oracle.chi0(m, w, accurate=True)
    n, (P, nw) = m.shape[1], w.shape
    s = np.sqrt(np.einsum("pi,pf->if", np.abs(m) ** 2, np.abs(w)))
    iu, ju = np.triu_indices(n)
    idx = ju * (ju + 1) // 2 + iu
    bound = 2 * (P + 8) * 2.0 ** -53 * s[iu] * s[ju]
    assert np.all(np.abs(got - ref)[idx] <= bound)


@pytest.mark.parametrize("nbas,npair,nw,pad", [
    (1, 1, 5, 0), (8, 15, 8, 1), (9, 16, 9, 0), (16, 17, 16, 3), (17, 255, 17, 0), (33, 256, 24, 0),
    (24, 257, 25, 1), (40, 1000, 29, 0), (65, 4097, 12, 5), (130, 3000, 24, 0), (403, 700, 7, 0),
    (257, 513, 36, 2), (7, 20000, 24, 0)])
@pytest.mark.parametrize("mixed", [False, True])
def test_product_form_matches_oracle(nbas, npair, nw, pad, mixed):
    m, md, w, d, om = _case(nbas, npair, nw, pad, mixed)
    out = torch.zeros((nw, npack(nbas)), dtype=torch.complex128, device=DEV)
    with spx.Context(0) as ctx:
        if mixed:
            ctx.chi0_accumulate_w_dev(md, torch.from_numpy(np.ascontiguousarray(w.T)).to(DEV), out, npair=npair,
                                      stats=True)
        else:
            ctx.chi0_accumulate_dev(md, d, om, out, npair=npair, stats=True)
    _check(out.cpu().numpy().T, m, w)


def test_product_form_without_room_for_partial_tiles():
    """A workspace_limit that holds the weights alone: the call still runs (whole tiles), and
    so does the allocation-free entry; both add into what the output holds."""
    nbas, npair, nw = 120, 5000, 24
    m, md, w, d, om = _case(nbas, npair, nw, 0, False)
    limit = 8 * 24 * ((npair + 15) // 16 * 16) + 512
    with spx.Context(0, workspace_limit=limit) as ctx:
        out = torch.zeros((nw, npack(nbas)), dtype=torch.complex128, device=DEV)
        ctx.chi0_accumulate_dev(md, d, om, out, stats=True)
        _check(out.cpu().numpy().T, m, w)
        ctx.chi0_accumulate_dev(md, d, om, out, stats=True)
        _check(0.5 * out.cpu().numpy().T, m, w)
        na = torch.zeros_like(out)
        torch.cuda.synchronize()
        rc = ctx.lib.spx_chi0_accumulate_dev_noalloc(md.data_ptr(), npair, npair, nbas, d.data_ptr(), None, 1.0,
                                                     nw, om.data_ptr(), na.data_ptr(), None)
        assert rc == 0
        _check(na.cpu().numpy().T, m, w)


@pytest.mark.parametrize("graph", [0, 1])
def test_product_form_batched_equals_per_q(graph):
    from project1_b200 import _lib
    nw = 12
    cases = [_case(n, p, nw, 0, False) for n, p in [(70, 900), (200, 3000), (1, 300)]]
    om = cases[0][4]
    qs = [dict(nbas=c[0].shape[1], npair=c[0].shape[0], cprod=c[1], ediff=c[3],
               susceph=torch.zeros((nw, npack(c[0].shape[1])), dtype=torch.complex128, device=DEV)) for c in cases]
    with spx.Context(0) as ctx:
        for _ in range(2):
            for q in qs:
                q["susceph"].zero_()
            ctx.chi0_batched(qs, om, precision="fp64", flags=0 if graph else _lib.SPX_BATCH_NOGRAPH, stats=True)
        for q, c in zip(qs, cases):
            out = torch.zeros_like(q["susceph"])
            ctx.chi0_accumulate_dev(c[1], c[3], om, out, stats=True)
            assert torch.equal(out, q["susceph"])
