"""FP64 accumulation with inversion symmetry (real products): both sides of the rule that picks
the kernel, tile and chunk remainders and frequency groups, against the extended-precision oracle."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle
import project1_b200 as spx
from project1_b200 import inputs
from project1_b200.susceptibility import npack

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("nbas,npair,nw", [(1, 1, 1), (16, 255, 8), (17, 256, 9), (64, 257, 24), (65, 1000, 25),
                                           (200, 321, 16), (300, 900, 48), (700, 130, 2), (900, 260, 24)])
@pytest.mark.parametrize("odd", [0, 1])
def test_real_products(nbas, npair, nw, odd):
    rng = np.random.default_rng(nbas + nw)
    m = np.asfortranarray(rng.standard_normal((npair, nbas)) / np.sqrt(nbas))
    d = rng.uniform(0.2, 3.0, npair)
    om = inputs.frequencies(nw)
    buf = torch.zeros((nbas, npair + odd), dtype=torch.float64, device=DEV)
    buf[:, :npair] = torch.from_numpy(np.ascontiguousarray(m.T))
    out = torch.zeros((nw, npack(nbas)), dtype=torch.float64, device=DEV)
    with spx.Context(0) as ctx:
        ctx.chi0_accumulate_real_dev(buf, torch.from_numpy(d).to(DEV), torch.from_numpy(om).to(DEV), out,
                                     scale_all=0.5, npair=npair, stats=True)
    w = oracle.weights(d, om, None, 0.5)
    ref = oracle.chi0_real(m, w)
    # 2 roundings a term, P - 1 of the sum, and 4 of the weight: (P + 8) 2^-53 sum |M_i||M_j||w|
    s = np.sqrt(np.einsum("pi,pf->if", m ** 2, np.abs(w)))
    iu, ju = np.triu_indices(nbas)
    err = np.abs(out.cpu().numpy().T - ref)[ju * (ju + 1) // 2 + iu]
    assert np.all(err <= 2 * (npair + 8) * 2.0 ** -53 * s[iu] * s[ju])
