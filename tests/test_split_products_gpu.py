"""Interstitial products on int8 slices: tile edges of the product GEMM, the one-pass and
two-pass operand preparation, rows of zeros, adding and storing."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle
import project1_b200 as spx
from project1_b200 import _lib, inputs
from project1_b200.wavefproducts import wavefproducts2_pw
from wfprod_util import shifted_pw, small_workload

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ctx():
    c = spx.Context(0, products=_lib.SPX_PRODUCTS_SPLIT)
    yield c
    c.close()


@pytest.mark.parametrize("kw,shifted", [
    (dict(nk=1, nocc=1, nunocc=1, ngpt=1, ngptm=1), False),
    (dict(nk=2, nocc=1, nunocc=63, ngpt=63, ngptm=64), True),
    (dict(nk=1, nocc=5, nunocc=64, ngpt=64, ngptm=13), False),       # 65 columns over two bands' edge
    (dict(nk=3, nocc=3, nunocc=65, ngpt=65, ngptm=21), True),
    (dict(nk=1, nocc=2, nunocc=130, ngpt=1025, ngptm=33), False),
    (dict(nk=1, nocc=1, nunocc=3, ngpt=4096, ngptm=3), False),       # longest one-pass row
    (dict(nk=1, nocc=2, nunocc=3, ngpt=4097, ngptm=3), False)])      # two passes
def test_split_product_edges(ctx, kw, shifted):
    w = small_workload(**kw)
    pw = shifted_pw(w, drop=0 if w.ngpt < 20 else 10) if shifted else inputs.pw_basis(w)
    c1, c2 = inputs.pw_coeffs(w, pw)
    c2[0, 0] = 0.0                                                   # a row with no scale
    ref = np.zeros((w.npair, w.ngptm), complex, order="F")
    oracle.wfprod_pw(pw, w.nk, w.nocc, w.nunocc, c1, c2, ref, 0)
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)
    rng = np.random.default_rng(w.npair)
    base = rng.standard_normal((w.ngptm, w.npair + 1)) + 1j * rng.standard_normal((w.ngptm, w.npair + 1))
    cp = d(base)
    wavefproducts2_pw(ctx, pw, d(c1), d(c2), cp, 0)
    got = cp.cpu().numpy()
    assert np.array_equal(got[:, w.npair:], base[:, w.npair:])
    add = (got[:, :w.npair] - base[:, :w.npair]).T
    # the smaller operand keeps 3 digits: half a unit 2^-17/127 of its row's largest part per value,
    # the dropped digit orders as much again, two real products per part over ng terms
    # against the other operand's largest value; alpha = 1/sqrt(vol). The convolved operand
    # is bounded by sum |cstep| times the occupied coefficients' largest value.
    big1 = np.abs(c1).max() * np.abs(pw["cstep"]).sum()
    big2 = np.abs(c2).max(axis=2)                                    # (nk, nunocc)
    ng = c2.shape[2]
    bound = 4 * np.sqrt(2) * ng * (2.0 ** -17 / 127) * 2 * big1 / np.sqrt(w.vol) * \
        np.broadcast_to(big2[:, None, :], (w.nk, w.nocc, w.nunocc)).reshape(-1)
    assert np.all(np.abs(add - ref) <= bound[:, None] + 2.0 ** -50 * np.abs(base[:, :w.npair].T))
    assert np.all(add[np.broadcast_to(big2[:, None, :] == 0, (w.nk, w.nocc, w.nunocc)).reshape(-1)] == 0)
