"""FP64 accumulation of up to four frequencies (and remainders of that size): both sides of
the rule that picks the tile form, against the extended-precision oracle."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle
import project1_b200 as spx
from project1_b200.susceptibility import npack

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("nbas,npair,nw", [(5, 300, 1), (64, 255, 4), (64, 256, 3), (300, 1000, 2), (600, 260, 1),
                                           (600, 260, 3), (900, 257, 2), (130, 900, 26)])
def test_few_frequencies(nbas, npair, nw):
    rng = np.random.default_rng(nbas + nw)
    m = np.asfortranarray((rng.standard_normal((npair, nbas)) + 1j * rng.standard_normal((npair, nbas)))
                          / np.sqrt(nbas))
    w = rng.standard_normal((npair, nw))
    md = torch.from_numpy(np.ascontiguousarray(m.T)).to(DEV)
    out = torch.zeros((nw, npack(nbas)), dtype=torch.complex128, device=DEV)
    with spx.Context(0) as ctx:
        ctx.chi0_accumulate_w_dev(md, torch.from_numpy(np.ascontiguousarray(w.T)).to(DEV), out, stats=True)
    ref = oracle.chi0(m, w, accurate=True)
    # at most 6 roundings a term and P - 1 of the sum, per part: (P + 8) 2^-53 sum |M_i||M_j||w|
    s = np.sqrt(np.einsum("pi,pf->if", np.abs(m) ** 2, np.abs(w)))
    iu, ju = np.triu_indices(nbas)
    err = np.abs(out.cpu().numpy().T - ref)[ju * (ju + 1) // 2 + iu]
    assert np.all(err <= 2 * (npair + 8) * 2.0 ** -53 * s[iu] * s[ju])
