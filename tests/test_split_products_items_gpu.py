"""The int8 product GEMM with several tiles per CTA and a last row block that is not full: lanes
of the missing rows store nothing and still take part in the next tile."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import project1_b200 as spx
from project1_b200 import _lib, inputs
from project1_b200.wavefproducts import wavefproducts2_pw
from wfprod_util import small_workload

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("nunocc", [65, 100, 127])
def test_ragged_rows_over_many_tiles(nunocc):
    """2 x 161 tiles for 148 CTAs, against the FP64 GEMM: half a unit 2^-17/127 of each operand
    row's largest part per value, the dropped digit orders as much again, two real products per
    part over the plane waves; the FP64 side's roundings are far below that."""
    w = small_workload(nk=1, nocc=40, nunocc=nunocc, ngpt=60, ngptm=257)
    pw = inputs.pw_basis(w)
    c1, c2 = inputs.pw_coeffs(w, pw)
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)
    outs = []
    for products in (_lib.SPX_PRODUCTS_FP64, _lib.SPX_PRODUCTS_SPLIT):
        cp = torch.zeros((w.ngptm, w.npair), dtype=torch.complex128, device=DEV)
        with spx.Context(0, products=products) as ctx:
            for _ in range(2):   # adds
                wavefproducts2_pw(ctx, pw, d(c1), d(c2), cp, 0)
            ctx.synchronize()
        outs.append(cp.cpu().numpy())
    big1 = np.abs(c1).max() * np.abs(pw["cstep"]).sum()
    big2 = np.abs(c2).max(axis=2)[:, None, :]
    bound = 2 * 4 * np.sqrt(2) * c2.shape[2] * (2.0 ** -17 / 127) * 2 * big1 / np.sqrt(w.vol) * \
        np.broadcast_to(big2, (1, w.nocc, nunocc)).reshape(-1)
    assert np.all(np.abs(outs[1] - outs[0]) <= bound[None, :])
