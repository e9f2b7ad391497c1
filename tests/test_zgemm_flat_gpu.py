"""The FP64 GEMM's form for one run of columns: the dielectric inverse at sizes around its
64-wide blocks and 16-deep chunks (rank 16 and less takes the general form), one and several
matrices per batch, against numpy."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

import project1_b200 as spx
from project1_b200.susceptibility import npack

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("n", [16, 17, 64, 65, 80, 81, 129, 145, 200])
@pytest.mark.parametrize("nw", [1, 5])
def test_inverse(n, nw):
    rng = np.random.default_rng(n + nw)
    chi = np.zeros((nw, npack(n)), dtype=np.complex128)
    eps = []
    iu, ju = np.triu_indices(n)
    v = rng.uniform(0.5, 1.5, n)
    for f in range(nw):
        b = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) / np.sqrt(n)
        x = -(b @ b.conj().T)
        chi[f, ju * (ju + 1) // 2 + iu] = x[iu, ju]
        eps.append(np.eye(n) - np.sqrt(v)[:, None] * x * np.sqrt(v)[None, :])
    p = torch.from_numpy(chi).to(DEV)
    with spx.Context(0) as ctx:
        ctx.dielec_dev(p, torch.from_numpy(v).to(DEV), invert=True)
    got = p.cpu().numpy()
    for f in range(nw):
        a = np.zeros((n, n), dtype=np.complex128)
        a[iu, ju] = got[f, ju * (ju + 1) // 2 + iu]
        a = a + np.triu(a, 1).conj().T
        # Gauss-Jordan on a positive definite matrix: residual within a few n 2^-53 of the
        # condition number (at most 1 + 1.5 * 4.5, the edge of the Wishart spectrum taken at 4.5)
        assert np.abs(a @ eps[f] - np.eye(n)).max() <= 8 * n * 2.0 ** -53 * 8
