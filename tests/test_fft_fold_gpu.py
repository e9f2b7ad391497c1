"""The FFT branch of the interstitial products: folded passes (mixed-basis vectors within 7 of
the origin) at grid edges, slot and band-group remainders, and the direct and line-FFT
passes for other sets, against the numpy restatement of the reference's FFT branch."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle
import project1_b200 as spx
from project1_b200 import inputs
from project1_b200.wavefproducts import wavefproducts2_pw
from wfprod_util import shifted_pw, small_workload

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def ctx():
    c = spx.Context(0)
    yield c
    c.close()


def _bound(pw, c1, c2, n):
    """Per pair: every output is a sum over the n^3 grid points of products whose factors are
    themselves sums over at most 2 n terms an axis; each axis adds at most 2 n roundings per term
    and the factors 6 each, on both sides of the comparison, so |error| <=
    2 (6 n + 40) 2^-53 n^3 sum|c1| sum|c2| sum|cstep| / (n^3 sqrt(vol)) with the factors bounded by
    their coefficient sums; sqrt(2) for the two parts."""
    s1, s2 = np.abs(c1).sum(-1), np.abs(c2).sum(-1)          # (nk, nocc), (nk, nunocc)
    cs = np.abs(pw["cstep"]).sum()
    return np.sqrt(2) * 2 * (6 * n + 40) * 2.0 ** -53 * cs / np.sqrt(pw["vol"]) * \
        (s1[:, :, None] * s2[:, None, :]).reshape(-1)


def _run(ctx, w, pw, n):
    c1, c2 = inputs.pw_coeffs(w, pw)
    ref = oracle.wfprod_pw_fft(pw, w.nk, w.nocc, w.nunocc, c1, c2, n)
    rng = np.random.default_rng(n)
    ng = pw["gptm"].shape[0]
    base = rng.standard_normal((ng, w.npair + 2)) + 1j * rng.standard_normal((ng, w.npair + 2))
    cp = torch.from_numpy(base).to(DEV)
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)
    wavefproducts2_pw(ctx, dict(pw, nfft=n), d(c1), d(c2), cp, 0)
    got = cp.cpu().numpy()
    assert np.array_equal(got[:, w.npair:], base[:, w.npair:])            # rows past npair
    add = got[:, :w.npair] - base[:, :w.npair]                            # the call adds
    assert np.all(np.abs(add.T - ref) <= _bound(pw, c1, c2, n)[:, None] + 2.0 ** -52 * np.abs(base[:, :w.npair]).T)


@pytest.mark.parametrize("n", [16, 17, 18, 23, 32, 33, 40, 48, 50, 63, 64])
@pytest.mark.parametrize("shifted", [False, True])
def test_folded_passes_grid_edges(ctx, n, shifted):
    w = small_workload(nk=2, nocc=5, nunocc=7, ngpt=60, ngptm=27)
    _run(ctx, w, shifted_pw(w, shift=(0, 1, 0), gshift=(1, -2, 0), drop=5) if shifted else inputs.pw_basis(w), n)


@pytest.mark.parametrize("nk,nocc,nunocc", [(1, 1, 1), (1, 4, 4), (3, 2, 5), (1, 9, 3), (2, 3, 130)])
@pytest.mark.parametrize("n", [24, 60])
def test_folded_passes_band_groups(ctx, nk, nocc, nunocc, n):
    w = small_workload(nk=nk, nocc=nocc, nunocc=nunocc, ngpt=60, ngptm=19)
    _run(ctx, w, inputs.pw_basis(w), n)


@pytest.mark.parametrize("n", [16, 21, 36, 48])
def test_folded_passes_full_reach(ctx, n):
    """Components up to +-7 on every axis, in no order, with repeats and lone signs."""
    w = small_workload(nk=1, nocc=2, nunocc=3, ngpt=60)
    g = np.array([[7, 0, 0], [-7, 1, 0], [0, 7, -7], [0, -7, 7], [0, 0, 7], [3, -7, -7], [7, 7, 7], [0, 0, 0],
                  [5, 2, -1], [7, 0, 0]], np.int32)
    _run(ctx, w, dict(inputs.pw_basis(w), gptm=g), n)


@pytest.mark.parametrize("n", [12, 19, 30, 32, 48])
def test_sets_beyond_the_folded_reach(ctx, n):
    """A sphere away from the origin (components 2 .. 10): direct sums and the line FFT."""
    w = small_workload(nk=2, nocc=3, nunocc=5, ngpt=60, ngptm=27)
    pw = inputs.pw_basis(w)
    pw["gptm"] = np.ascontiguousarray(pw["gptm"] + np.array([6, 0, -8], np.int32))
    pw["gshift"] = np.array([1, 0, 0], np.int32)
    _run(ctx, w, pw, n)
