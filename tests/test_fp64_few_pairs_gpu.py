"""FP64 accumulations of few pairs, between the two forms of the kernel: which form the rule
takes, and its sums against the extended-precision oracle."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import oracle
import project1_b200 as spx
from project1_b200 import _lib, inputs
from project1_b200.susceptibility import npack


def _on_k1(real, nbas, npair, nw, part=True):
    fn = getattr(_lib.load(), "_ZN3spx10fp64_on_k1Ebibili")
    fn.restype, fn.argtypes = C.c_int, [C.c_bool, C.c_int, C.c_bool, C.c_int, C.c_int64, C.c_int]
    return fn(real, 148, part, nbas, npair, nw)


# measured: the frequency-by-frequency form is faster by 10 % or more ...
FIRST = [(False, 65, 80, 36), (False, 300, 8, 36), (False, 640, 16, 12), (False, 1250, 16, 36), (False, 1500, 12800, 4),
         (True, 65, 80, 48), (True, 150, 108, 48), (True, 900, 16, 36), (True, 1250, 1, 5), (True, 1500, 12800, 4)]
# ... and the product-first form
SECOND = [(False, 150, 80, 48), (False, 640, 80, 24), (False, 1500, 80, 48), (False, 400, 12800, 4), (False, 1200, 128000, 24),
          (True, 300, 80, 24), (True, 300, 10000, 24), (True, 900, 10000, 48), (True, 89, 4000, 12)]


@pytest.mark.parametrize("shape", FIRST)
def test_rule_takes_the_first_form(shape):
    assert _on_k1(*shape) == shape[3]


@pytest.mark.parametrize("shape", SECOND)
def test_rule_takes_the_product_form(shape):
    assert _on_k1(*shape) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("real", [False, True])
@pytest.mark.parametrize("nbas,npair,nw", [(1, 1, 1), (17, 2, 36), (64, 6, 25), (65, 16, 48), (150, 108, 48), (33, 39, 32),
                                           (100, 64, 24), (100, 65, 24), (130, 255, 41), (130, 256, 41), (403, 80, 27)])
def test_few_pairs_against_the_oracle(nbas, npair, nw, real):
    """At most 6 roundings a term and P - 1 of the sum, either form: |error| <= (P + 8) 2^-53
    sum_p |M_i||M_j||w| per part, bounded by the |w|-weighted column norms."""
    rng = np.random.default_rng(nbas + npair + nw)
    m = rng.standard_normal((npair, nbas))
    if not real:
        m = m + 1j * rng.standard_normal((npair, nbas))
    m = np.asfortranarray(m / np.sqrt(nbas))
    d = rng.uniform(0.5, 40.0, npair)
    om = inputs.frequencies(nw)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to("cuda:0")
    out = torch.zeros((nw, npack(nbas)), dtype=torch.float64 if real else torch.complex128, device="cuda:0")
    with spx.Context(0) as ctx:
        call = ctx.chi0_accumulate_real_dev if real else ctx.chi0_accumulate_dev
        call(t(m.T), t(d), t(om), out, stats=True)
    w = oracle.weights(d, om)
    ref = oracle.chi0_real(m, w) if real else oracle.chi0(m, w, accurate=True)
    s = np.sqrt(np.einsum("pi,pf->if", np.abs(m) ** 2, np.abs(w)))
    j, i = np.tril_indices(nbas)
    # (the real oracle sums in FP64 too)
    assert np.all(np.abs(out.cpu().numpy().T - ref) <= (4 if real else 2) * (npair + 8) * 2.0 ** -53 * s[i] * s[j])
