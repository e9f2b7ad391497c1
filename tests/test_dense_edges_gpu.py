"""Tile and block edges of the dense FP64 kernels: the product GEMM behind the transform,
the Hermitian block sweep of the dielectric inverse, and head and wings."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle
import project1_b200 as spx
from project1_b200.susceptibility import npack

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
U = 2.0 ** -53


@pytest.fixture(scope="module")
def ctx():
    c = spx.Context(0)
    yield c
    c.close()


def _d(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(DEV)


def _z(rng, *shape):
    return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)


@pytest.mark.parametrize("npair,nbas,dim", [(1, 1, 1), (63, 15, 64), (64, 16, 63), (65, 17, 65), (700, 33, 129),
                                            (40000, 70, 66)])
@pytest.mark.parametrize("inplace", [False, True])
def test_transform_tile_edges(ctx, npair, nbas, dim, inplace):
    rng = np.random.default_rng(npair + nbas)
    if inplace:
        dim = min(dim, nbas)
    c, t = _z(rng, npair, nbas), _z(rng, nbas, dim)
    ref = oracle.trafo(c, t)
    # each part: 2 nbas products and their sum, |error| <= (2 nbas + 2) u sum |c||t|, twice for re and im;
    # the oracle's own sum carries as much
    bound = 4 * (2 * nbas + 2) * U * (np.abs(c) @ np.abs(t))
    cd = torch.full((nbas, npair + 3), 5.0 + 0j, dtype=torch.complex128, device=DEV)
    cd[:, :npair] = _d(c.T)
    out = cd if inplace else torch.full((dim, npair + 1), 9.0 + 0j, dtype=torch.complex128, device=DEV)
    ctx.trafo_dev(cd, _d(t.T), out=None if inplace else out, npair=npair)
    got = out.cpu().numpy()
    assert np.all(np.abs(got[:dim, :npair].T - ref) <= bound)
    assert np.all(got[:dim, npair:] == (5.0 if inplace else 9.0))   # padding untouched


@pytest.mark.parametrize("n,nw", [(1, 1), (15, 2), (63, 3), (64, 1), (65, 2), (127, 1), (129, 2), (200, 3)])
def test_dielectric_inverse_block_edges(ctx, n, nw):
    rng = np.random.default_rng(n)
    chi = np.zeros((npack(n), nw), complex)
    iu, ju = np.triu_indices(n)
    for f in range(nw):
        b = _z(rng, n, n) / np.sqrt(2 * n)
        chi[ju * (ju + 1) // 2 + iu, f] = -(b @ b.conj().T)[iu, ju]
    coul = rng.uniform(0.5, 3.0, n)
    ref = oracle.dielec(chi, coul)
    eps = _d(chi.T)
    ctx.dielec_dev(eps, _d(coul))
    got = eps.cpu().numpy().T
    # eps = 1 + positive semi-definite: |inverse| <= 1; Gauss-Jordan on such a matrix is backward
    # stable, forward error <= c n kappa u with kappa <= |eps| <= 1 + 3 |b|^2 < 20, c a small constant
    assert np.abs(got - ref).max() <= 10 * n * 20 * U + 1e-15


@pytest.mark.parametrize("npair,dim,nw,pad", [(1, 1, 2, 0), (17, 3, 8, 1), (255, 64, 9, 0), (256, 65, 24, 1),
                                              (5000, 63, 25, 0), (20000, 129, 30, 3), (3000, 0, 17, 0),
                                              (1000, 500, 1, 0)])
def test_headwings_group_edges(ctx, npair, dim, nw, pad):
    rng = np.random.default_rng(npair + dim)
    c, d, w = _z(rng, npair, dim), _z(rng, npair, 3), rng.standard_normal((npair, nw))
    href, gref = oracle.headwings(c, d, w)
    wd = torch.full((nw, npair + pad), 1e300, dtype=torch.float64, device=DEV)
    wd[:, :npair] = _d(w.T)
    head = torch.zeros((nw, 6), dtype=torch.complex128, device=DEV)
    wing = torch.zeros((nw, dim, 3), dtype=torch.complex128, device=DEV)
    cd = _d(c.T) if dim else torch.zeros((0, npair), dtype=torch.complex128, device=DEV)
    ctx.headwings_dev(cd, _d(d.T), wd, head, wing, npair=npair)
    # as the accumulation: (P + 8) u sum |x||y||w| per part, and as much for the oracle's sum
    scale = 4 * (npair + 8) * U
    hb = np.array([(np.abs(d[:, k1]) * np.abs(d[:, k2])) @ np.abs(w) for k2 in range(3) for k1 in range(k2 + 1)])
    assert np.all(np.abs(head.cpu().numpy().T - href) <= scale * hb)
    for k in range(3):
        gb = (np.abs(c) * np.abs(d[:, k])[:, None]).T @ np.abs(w)
        assert np.all(np.abs(wing.cpu().numpy()[:, :, k].T - gref[k]) <= scale * gb)
