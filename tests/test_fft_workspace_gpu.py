"""The FFT branch's scratch: the band grids' pass buffers and the pairs' half-transformed grids
share one region, and unpadded (unfolded) passes step in where a limit has no room for folded
ones, so the call fits where it fitted with separate buffers and unpadded lines."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import project1_b200 as spx
from project1_b200 import inputs
from project1_b200.wavefproducts import wavefproducts2_pw
from test_fft_fold_gpu import _bound
from wfprod_util import shifted_pw, small_workload

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _separate(pw, nk, nocc, nunocc, n):
    """Bytes with every buffer apart and lines of n points, all k points at once (small cases)."""
    up = lambda x: (x + 255) // 256 * 256
    dim = lambda g: g.max(0) - g.min(0) + 1
    d1, d2 = dim(pw["gpt1"]), dim(pw["gpt2"])
    nb = max(nocc, nunocc)
    ks = [len(set(((pw["gptm"] - pw["gshift"]) % n)[:, c])) for c in range(3)]
    perk = up(16 * nb * max(d1.prod(), d2.prod())) + up(16 * nb * n * max(d1[1] * d1[2], d2[1] * d2[2])) + \
        up(16 * nb * n * n * max(d1[2], d2[2])) + up(16 * (nocc + nunocc) * n ** 3) + \
        up(16 * nocc * nunocc * n * ks[1] * ks[2]) + 16 * n * n * 18 + 2048
    return 16 * n ** 3 + 80 * 1024 + 4 * (len(pw["gpt1"]) + len(pw["gpt2"]) + 2 * len(pw["gptm"])) + nk * perk


@pytest.mark.parametrize("n", [16, 24, 30, 48, 60, 64])
@pytest.mark.parametrize("nk,nocc,nunocc", [(1, 1, 1), (1, 3, 4), (2, 3, 4), (2, 5, 40), (1, 16, 16)])
def test_fits_where_separate_buffers_did(n, nk, nocc, nunocc):
    w = small_workload(nk=nk, nocc=nocc, nunocc=nunocc, ngpt=257 if n > 16 else 57, ngptm=57)
    pw = shifted_pw(w, drop=7)
    c1, c2 = (torch.from_numpy(c).to(DEV) for c in inputs.pw_coeffs(w, pw))
    outs = []
    for limit in (0, int(_separate(pw, nk, nocc, nunocc, n))):
        cp = torch.zeros((w.ngptm, w.npair), dtype=torch.complex128, device=DEV)
        with spx.Context(0, workspace_limit=limit) as ctx:
            wavefproducts2_pw(ctx, dict(pw, nfft=n), c1, c2, cp, 0)
            ctx.synchronize()
        outs.append(cp.cpu().numpy())
    # folded and direct sums of the same numbers: test_fft_fold_gpu's bound, for each of the two
    bound = _bound(pw, c1.cpu().numpy(), c2.cpu().numpy(), n)
    assert np.all(np.abs(outs[0] - outs[1]) <= 2 * bound[None, :])

