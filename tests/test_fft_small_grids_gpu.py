"""The FFT branch on grids of a few points: the line transforms run over boxes many times as
wide as the grid."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle
import project1_b200 as spx
from project1_b200 import inputs
from project1_b200.wavefproducts import wavefproducts2_pw
from test_fft_fold_gpu import _bound
from wfprod_util import small_workload

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("n", [2, 3, 4, 5])
def test_smallest_grids_take_wide_boxes(n):
    """One plane wave per grid point, with components up to +-40: n values of an axis's box of
    about 80 are occupied, so the 2 n terms an axis of _bound hold."""
    w = small_workload(nk=1, nocc=2, nunocc=3, ngptm=27, step_radius=0)
    k = 40 // n
    axis = np.array([r + n * (k if r % 2 == 0 else -k) for r in range(n)], np.int32)
    g = np.ascontiguousarray(np.stack(np.meshgrid(axis, axis, axis, indexing="ij"), -1).reshape(-1, 3))
    pw = dict(inputs.pw_basis(w), gpt1=g, gpt2=g.copy())
    rng = np.random.default_rng(n)
    c1, c2 = (rng.standard_normal((1, nb, n ** 3)) + 1j * rng.standard_normal((1, nb, n ** 3))
              for nb in (w.nocc, w.nunocc))
    ref = oracle.wfprod_pw_fft(pw, 1, w.nocc, w.nunocc, c1, c2, n)
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)
    cp = torch.zeros((w.ngptm, w.npair), dtype=torch.complex128, device=DEV)
    with spx.Context(0) as ctx:
        wavefproducts2_pw(ctx, dict(pw, nfft=n), d(c1), d(c2), cp, 0)
        ctx.synchronize()
    assert np.all(np.abs(cp.cpu().numpy().T - ref) <= _bound(pw, c1, c2, n)[:, None])
