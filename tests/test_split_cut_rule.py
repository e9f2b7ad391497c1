"""How the last items of the split accumulation are cut along the pairs, and the bits of calls at
the edges of that rule."""
import ctypes as C

import pytest

torch = pytest.importorskip("torch")

import project1_b200 as spx
from project1_b200 import _lib, inputs
from project1_b200.susceptibility import npack

SMS = 148


@pytest.mark.parametrize("real", [False, True])
@pytest.mark.parametrize("nitems", [1, 2, 28, 147, 148, 149, 150, 170, 295, 296, 297, 336, 443])
def test_shares_are_worth_their_partial_tiles(nitems, real):
    """The last round's time in stages, an item's partial tiles counting one each: never more than a
    whole item's, and the saving covers the cost of the sum (64 or 128 stages)."""
    fn = getattr(_lib.load(), "_ZN3spx14split_cut_ctasEiiib")
    fn.restype, fn.argtypes = C.c_int, [C.c_int, C.c_int, C.c_int, C.c_bool]
    for nk in list(range(1, 200)) + [256, 300, 511, 512]:
        n = fn(nitems, nk, SMS, real)
        assert 0 <= n <= SMS
        if n == 0:
            continue
        left = nitems % SMS
        longest = -(-left * nk // n)
        assert left * nk // n >= 8 and longest < nk
        assert longest + nk / (left * nk / n) <= nk
        assert nk - longest >= (126 if real else 62)


@pytest.mark.gpu
@pytest.mark.parametrize("nbas,npair,nw", [(320, 4160, 10), (320, 4700, 10), (64, 4700, 149), (64, 9000, 150), (64, 32768, 149),
                                           (64, 32768, 1), (130, 8200, 27)])
@pytest.mark.parametrize("real", [False, True])
def test_cut_and_whole_items_give_the_same_bits(nbas, npair, nw, real):
    """A workspace_limit without room for partial tiles keeps the items whole."""
    g = torch.Generator("cuda:0").manual_seed(nbas + npair)
    m = torch.randn((nbas, npair), dtype=torch.float64 if real else torch.complex128, device="cuda:0", generator=g)
    d = torch.rand(npair, dtype=torch.float64, device="cuda:0", generator=g) * 30 + 0.3
    d[::5] *= -1.0
    om = torch.from_numpy(inputs.frequencies(nw)).to("cuda:0")
    size = getattr(_lib.load(), "_ZN3spx26split_workspace_bytes_realElii" if real else "_ZN3spx21split_workspace_bytesElii")
    size.restype, size.argtypes = C.c_size_t, [C.c_int64, C.c_int, C.c_int]
    outs, counts = [], []
    for limit in (0, size(npair, nbas, nw) + 1024):
        out = torch.zeros((nw, npack(nbas)), dtype=m.dtype, device="cuda:0")
        with spx.Context(0, workspace_limit=limit) as ctx:
            call = ctx.chi0_accumulate_real_dev if real else ctx.chi0_accumulate_dev
            counts.append(call(m, d, om, out, precision="split", stats=True)["kernel_launches"])
        outs.append(out)
    assert counts[1] == 3 and counts[0] in (3, 4)
    assert torch.equal(outs[0], outs[1])
