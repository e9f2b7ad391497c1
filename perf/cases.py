"""Performance cases of the polarisation library: what a user's program calls, over the
sizes it is called with.

Each case is a dict of plain values. `prepare` makes the inputs on the GPU (host arrays
for the host-pointer call) from a seed, `run` is one pass through the public entry points,
`work` the bytes and operations a pass cannot do without, and `exact` the same outputs
in plain 64-bit torch. Kinds:

  host      susceptibility() on numpy arrays, the drop-in call of a host program
  chi0      chi0_accumulate_dev, complex M on the device, "fp64" or "split"
  real      chi0_accumulate_real_dev (the inversion-symmetric build: real M)
  batched   chi0_batched, several q points of uneven sizes in one launch
  products  wavefproducts2_mt + wavefproducts2_pw (explicit convolution, FP64)
  fft       wavefproducts2_pw through the FFT branch
  fused     chi0_from_coeffs: products and polarisation in one call
  gamma     q -> 0: dcprod, transform to the Coulomb eigenbasis, weights, head and wings
  dielec    dielectric matrices and their inverses, with head and wings
"""
from __future__ import annotations

import math

import numpy as np
import torch

import project1_b200 as spx
from project1_b200 import inputs
from project1_b200 import wavefproducts as wf

DEV = "cuda:0"
C128 = torch.complex128
F64 = torch.float64
_CTX = None


def _context():
    """The one context a program keeps for its device."""
    global _CTX
    if _CTX is None:
        _CTX = spx.Context(0)
    return _CTX


# ---------------------------------------------------------------------------
# the cases


def listed():
    return [
        # one q point of a small crystal from a host program (SPEX's own call surface):
        # 400 mixed-basis functions, 8 k points, 20 x 80 bands, 12 frequencies, pageable arrays
        dict(name="host_fp64_small", kind="host", precision="fp64", nbas=400, nk=8, nocc=20,
             nunocc=80, nw=12, kweights=False),
        # the plain FP64 drop-in on a medium crystal: 1200 functions, 40 x 400 bands,
        # 24 frequencies, the 8 irreducible k points of one q
        dict(name="fp64_medium", kind="chi0", precision="fp64", nbas=1200, nk=8, nocc=40,
             nunocc=400, nw=24, pad=0, kweights=True, degenerate=0.0),
        # the smallest calls: one packet of a molecule-sized basis, where latency counts
        dict(name="split_tiny", kind="chi0", precision="split", nbas=96, nk=2, nocc=4,
             nunocc=20, nw=4, pad=0, kweights=False, degenerate=0.05),
        # an ordinary small q point with odd sizes and a padded leading dimension
        dict(name="split_small", kind="chi0", precision="split", nbas=403, nk=7, nocc=21,
             nunocc=83, nw=12, pad=3, kweights=True, degenerate=0.01),
        # the largest single call: 1200 functions, 64 k x 40 x 400 bands, 24 frequencies,
        # 1 % near-degenerate pairs
        dict(name="split_large", kind="chi0", precision="split", nbas=1200, nk=64, nocc=40,
             nunocc=400, nw=24, pad=0, kweights=False, degenerate=0.01),
        # a crystal with inversion symmetry: real M and real polarisation
        dict(name="real_split", kind="real", precision="split", nbas=900, nk=16, nocc=24,
             nunocc=200, nw=24, pad=0, kweights=True, degenerate=0.01),
        # several q points of uneven sizes in one call
        dict(name="batched_split", kind="batched", precision="split", nq=8, nbas_lo=300,
             nbas_hi=900, nk=8, occ_lo=10, occ_hi=30, unocc_lo=60, unocc_hi=150, nw=24),
        # the wave-function products alone (muffin tin and explicit convolution), FP64:
        # 2 atoms, lmax 8, 3 radial functions, 3000 plane waves, 40 x 300 bands
        dict(name="products_fp64", kind="products", lcut=8, nrad=3, ngpt=3000, ngptm=1014, nk=4,
             nocc=40, nunocc=300, drop=0),
        # the interstitial products on the 48^3 grid
        dict(name="products_fft", kind="fft", ngpt=3000, ngptm=1014, nfft=48, nk=2, nocc=40,
             nunocc=300),
        # products and split polarisation in one call, 27 k points, 1500 functions
        dict(name="fused_split", kind="fused", precision="split", lcut=8, nrad=3, ngpt=3000,
             ngptm=1014, nk=27, nocc=40, nunocc=300, nw=24),
        # the Gamma point: momentum matrix, transform to the Coulomb eigenbasis, head, wings
        dict(name="gamma", kind="gamma", nbas=1200, dim=1100, lcut=8, nrad=3, ngpt=1500, nk=4,
             nocc=40, nunocc=300, nw=24),
        # 24 dielectric matrices of 1200 and their inverses
        dict(name="dielec_inverse", kind="dielec", nbas=1200, nw=24),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host", "chi0", "chi0", "real", "batched", "products", "fft", "fused",
                       "gamma", "dielec"])
    nw = rng.choice([1, 4, 6, 8, 11, 12, 16, 20, 24, 24, 31, 36])
    if kind in ("host", "chi0", "real"):
        prec = rng.choice(["fp64", "split"])
        while True:
            c = dict(kind=kind, precision=prec, nbas=_log(rng, 60, 500 if kind == "host" else 1500),
                     nk=_log(rng, 1, 8 if kind == "host" else 64), nocc=_log(rng, 4, 40),
                     nunocc=_log(rng, 20, 120 if kind == "host" else 400), nw=nw,
                     pad=rng.choice([0, 0, 1, 3, 16]), kweights=rng.random() < 0.5,
                     degenerate=rng.choice([0.0, 0.01]))
            P = c["nk"] * c["nocc"] * c["nunocc"]
            # at most the cost of the listed FP64 / split calls, 8 GB of M
            cap = 3.4e13 if prec == "fp64" else 2.8e14
            if 8.0 * c["nbas"] ** 2 * P * nw <= cap and 16 * c["nbas"] * P <= 8e9:
                return c
    if kind == "batched":
        lo = _log(rng, 60, 600)
        occ, un = _log(rng, 5, 20), _log(rng, 30, 120)
        return dict(kind=kind, precision="split", nq=rng.randint(2, 12), nbas_lo=lo,
                    nbas_hi=lo + rng.randint(0, 500), nk=rng.randint(1, 12), occ_lo=occ,
                    occ_hi=occ + 12, unocc_lo=un, unocc_hi=un + 60, nw=min(nw, 24))
    if kind in ("products", "fused"):
        lcut = rng.choice([3, 4, 6, 8])
        c = dict(kind=kind, lcut=lcut, nrad=rng.choice([2, 3]), ngpt=_log(rng, 300, 3000),
                 ngptm=_log(rng, 60, 1014), nk=rng.randint(1, 6 if kind == "products" else 16),
                 nocc=rng.randint(5, 40), nunocc=_log(rng, 40, 300))
        if kind == "fused":
            c.update(precision="split", nw=min(nw, 24))
        else:
            c.update(drop=rng.choice([0, 0, 7, 10]))
        return c
    if kind == "fft":
        nfft = rng.choice([32, 48, 48, 40, 64])
        # spheres whose products and mixed-basis vectors do not wrap on the grid
        ngpt = _log(rng, 200, 600 if nfft < 48 else 3000)
        return dict(kind=kind, ngpt=ngpt, ngptm=_log(rng, 50, 257 if nfft < 48 else 1014), nfft=nfft,
                    nk=rng.randint(1, 2), nocc=rng.randint(4, 40), nunocc=_log(rng, 30, 300))
    if kind == "gamma":
        nbas = _log(rng, 100, 1200)
        return dict(kind=kind, nbas=nbas, dim=rng.randint(nbas * 2 // 3, nbas), lcut=rng.choice([4, 6, 8]),
                    nrad=rng.choice([2, 3]), ngpt=_log(rng, 200, 1500), nk=rng.randint(1, 4),
                    nocc=rng.randint(5, 40), nunocc=_log(rng, 40, 300), nw=min(nw, 24))
    return dict(kind="dielec", nbas=_log(rng, 60, 1300), nw=min(nw, 24))


# ---------------------------------------------------------------------------
# inputs


def _gen(seed, salt=0):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 1000003 + salt)
    return g


def _normal(shape, g, scale=1.0):
    """Complex normals, real and imaginary part of standard deviation `scale`."""
    z = torch.empty(shape, dtype=C128, device=DEV)
    torch.view_as_real(z).normal_(0.0, scale, generator=g)
    return z


def _uniform(shape, lo, hi, g):
    return torch.empty(shape, dtype=F64, device=DEV).uniform_(lo, hi, generator=g)


def _ediff(nk, nocc, nunocc, degenerate, g):
    """e_n'(k+q) - e_n(k) of sorted bands (eV), n' fastest; some near-degenerate pairs."""
    occ = _uniform((nk, nocc), -10.0, 0.0, g).sort(dim=1).values
    un = _uniform((nk, nunocc), 0.5, 40.0, g).sort(dim=1).values
    d = (un[:, None, :] - occ[:, :, None]).reshape(-1)
    if degenerate > 0:
        n = max(1, int(round(degenerate * d.numel())))
        sel = torch.randperm(d.numel(), device=DEV, generator=g)[:n]
        d[sel] = _uniform((n,), 0.0, 1e-6, g)
    return d.contiguous()


def _omega(nw):
    return torch.from_numpy(inputs.frequencies(nw)).to(DEV)


def _wscale(case, seed):
    """nkpts(k) per pair: the number of k points an irreducible one stands for."""
    if not case.get("kweights"):
        return None
    n = np.random.default_rng([seed, 17]).integers(1, 9, case["nk"]).astype(np.float64)
    return torch.from_numpy(np.repeat(n, case["nocc"] * case["nunocc"])).to(DEV)


def _npair(case):
    return case["nk"] * case["nocc"] * case["nunocc"]


def _chi0_inputs(case, seed):
    g = _gen(seed)
    P, N = _npair(case), case["nbas"]
    ldc = P + case.get("pad", 0)
    if case["kind"] == "real":
        m = torch.empty((N, ldc), dtype=F64, device=DEV).normal_(0.0, 1.0 / math.sqrt(N), generator=g)
    else:
        m = _normal((N, ldc), g, 1.0 / math.sqrt(N))
    return dict(m=m, ediff=_ediff(case["nk"], case["nocc"], case["nunocc"], case.get("degenerate", 0.0), g),
                omega=_omega(case["nw"]), ws=_wscale(case, seed), scale=1.0 / case["nk"])


def _batched_inputs(case, seed):
    # the sizes belong to the case, the values to the seed
    r = np.random.default_rng([case["nq"], case["nbas_lo"], case["nbas_hi"], case["nk"], 23])
    g = _gen(seed)
    sizes = [(int(r.integers(case["nbas_lo"], case["nbas_hi"] + 1)),
              int(r.integers(case["occ_lo"], case["occ_hi"] + 1)),
              int(r.integers(case["unocc_lo"], case["unocc_hi"] + 1))) for _ in range(case["nq"])]
    qs = []
    for n, no, nu in sizes:
        P = case["nk"] * no * nu
        qs.append(dict(nbas=n, npair=P, cprod=_normal((n, P), g, 1.0 / math.sqrt(n)),
                       ediff=_ediff(case["nk"], no, nu, 0.01, g), scale_all=1.0 / case["nk"]))
    return qs


def _workload(case, seed):
    return inputs.WfprodWorkload("case", lcut=case.get("lcut", 2), lcutm=case.get("lcut", 2),
                                 nrad=case.get("nrad", 2), nradm=case.get("nrad", 2), ngpt=case["ngpt"],
                                 ngptm=case["ngptm"], nk=case["nk"], nocc=case["nocc"],
                                 nunocc=case["nunocc"], nw=case.get("nw", 1), seed=int(seed) % (1 << 31))


def _coeff_inputs(case, seed):
    """Basis descriptors (host) and coefficients (device) of the products."""
    w = _workload(case, seed)
    g = _gen(seed)
    pw = inputs.pw_basis(w)
    drop = case.get("drop", 0)
    if drop:   # k+q: another, shorter sphere and a backfolding vector
        pw["gpt2"] = np.ascontiguousarray(pw["gpt1"][: pw["gpt1"].shape[0] - drop] + np.array([1, 0, 0], np.int32))
        pw["gshift"] = np.array([0, 1, 0], np.int32)
    if case.get("nfft"):
        pw["nfft"] = case["nfft"]
    out = dict(w=w, pw=pw)
    for key, gpt, nb in (("p1", pw["gpt1"], case["nocc"]), ("p2", pw["gpt2"], case["nunocc"])):
        damp = torch.from_numpy(np.exp(-(gpt.astype(float) ** 2).sum(1) / 50.0)).to(DEV)
        out[key] = _normal((case["nk"], nb, gpt.shape[0]), g) * damp
    if "lcut" in case:
        out["mt"] = inputs.mt_basis(w)
        out["c1"] = _normal((case["nk"], case["nocc"], w.natom, w.maxlm), g)
        out["c2"] = _normal((case["nk"], case["nunocc"], w.natom, w.maxlm), g)
    return out


def _gamma_inputs(case, seed):
    g = _gen(seed)
    r = np.random.default_rng([seed, 29])
    natom, lcut, nrad, nk = 2, case["lcut"], case["nrad"], case["nk"]
    maxlm, N, P = (lcut + 1) ** 2 * nrad, case["nbas"], _npair(case)
    w = _workload(dict(case, ngptm=1), seed)
    basis = inputs.pw_basis(w)
    damp = torch.from_numpy(np.exp(-(basis["gpt1"].astype(float) ** 2).sum(1) / 50.0)).to(DEV)
    mom = dict(natom=natom, lcut=lcut, nrad=nrad, qmat1=r.standard_normal((nrad, nrad, lcut + 1)),
               qmat2=r.standard_normal((nrad, nrad, lcut + 1)), gpt=basis["gpt1"],
               kpt=r.uniform(-0.5, 0.5, (nk, 3)),
               rlat=2 * np.pi / 10.0 * (np.eye(3) + 0.1 * r.standard_normal((3, 3))),
               cstep=basis["cstep"], step_radius=basis["step_radius"], vol=1000.0)
    return dict(mom=mom, c1=_normal((nk, case["nocc"], natom, maxlm), g),
                c2=_normal((nk, case["nunocc"], natom, maxlm), g),
                p1=_normal((nk, case["nocc"], case["ngpt"]), g) * damp,
                p2=_normal((nk, case["nunocc"], case["ngpt"]), g) * damp,
                cprod=_normal((N, P), g, 1.0 / math.sqrt(N)),
                trafo=_normal((case["dim"], N), g, 1.0 / math.sqrt(2 * N)),
                ediff=_ediff(nk, case["nocc"], case["nunocc"], 0.0, g), omega=_omega(case["nw"]))


def _tri(n):
    """Packed index j(j+1)/2 + i and (i, j) of the upper triangle, in packed order."""
    j = torch.arange(n, device=DEV).repeat_interleave(torch.arange(1, n + 1, device=DEV))
    i = torch.arange(j.numel(), device=DEV) - j * (j + 1) // 2
    return i, j


def _dielec_inputs(case, seed):
    """Negative semi-definite chi decaying with frequency, 4 pi / |q + G|^2 Coulomb values."""
    g = _gen(seed)
    n, nw = case["nbas"], case["nw"]
    i, j = _tri(n)
    chi = torch.empty((nw, n * (n + 1) // 2), dtype=C128, device=DEV)
    om = _omega(nw)
    b = _normal((n, n), g, 1.0 / math.sqrt(n))
    for f in range(nw):
        s = (-0.3 / (1.0 + float(om[f]) / 15.0)) * _uniform((n,), 0.2, 1.0, g)
        chi[f] = ((b * s) @ b.conj().T)[i, j]
    coul = 4 * math.pi / (0.4 * torch.arange(1, n + 1, device=DEV, dtype=F64) ** (2.0 / 3.0))
    return dict(chi=chi, coul=coul, head=_normal((nw, 6), g, 0.1), wing=_normal((nw, n, 3), g, 0.1))


def prepare(case, seed):
    ctx = _context()
    kind = case["kind"]
    st = dict(ctx=ctx, case=case)
    if kind == "host":
        a = _chi0_inputs(case, seed)
        st.update(m=np.asfortranarray(a["m"][:, :_npair(case)].cpu().numpy().T),
                  ediff=a["ediff"].cpu().numpy(), frqh=1j * a["omega"].cpu().numpy(),
                  nkpts=None if a["ws"] is None else a["ws"].cpu().numpy())
        return st
    if kind in ("chi0", "real"):
        a = _chi0_inputs(case, seed)
        st.update(a)
        n = case["nbas"]
        st["out"] = torch.zeros((case["nw"], n * (n + 1) // 2), dtype=F64 if kind == "real" else C128, device=DEV)
    elif kind == "batched":
        qs = _batched_inputs(case, seed)
        sizes = [case["nw"] * q["nbas"] * (q["nbas"] + 1) // 2 for q in qs]
        flat = torch.zeros((sum(sizes),), dtype=C128, device=DEV)
        off = 0
        for q, s in zip(qs, sizes):
            q["susceph"] = flat[off:off + s].view(case["nw"], -1)
            off += s
        st.update(qs=qs, flat=flat, omega=_omega(case["nw"]))
    elif kind in ("products", "fft", "fused"):
        a = _coeff_inputs(case, seed)
        st.update(p1=a["p1"], p2=a["p2"], pw=wf.PwDesc(a["pw"]))
        if "mt" in a:
            st.update(mt=wf.MtDesc(a["mt"]), c1=a["c1"], c2=a["c2"])
        w = a["w"]
        if kind == "fused":
            n = w.nbas
            st.update(ediff=_ediff(case["nk"], case["nocc"], case["nunocc"], 0.0, _gen(seed, 1)),
                      omega=_omega(case["nw"]),
                      out=torch.zeros((case["nw"], n * (n + 1) // 2), dtype=C128, device=DEV))
        else:
            st["col0"] = w.nbasp if kind == "products" else 0
            st["cprod"] = torch.zeros((st["col0"] + case["ngptm"], _npair(case)), dtype=C128, device=DEV)
    elif kind == "gamma":
        a = _gamma_inputs(case, seed)
        P, nw, dim = _npair(case), case["nw"], case["dim"]
        st.update(a, mom=wf.MomDesc(a["mom"]),
                  dc=torch.zeros((3, P), dtype=C128, device=DEV), body=torch.zeros((dim, P), dtype=C128, device=DEV),
                  w=torch.zeros((nw, P), dtype=F64, device=DEV), head=torch.zeros((nw, 6), dtype=C128, device=DEV),
                  wing=torch.zeros((nw, dim, 3), dtype=C128, device=DEV))
    elif kind == "dielec":
        a = _dielec_inputs(case, seed)
        st.update(a, eps=torch.empty_like(a["chi"]), h=torch.empty_like(a["head"]), g=torch.empty_like(a["wing"]))
    return st


# ---------------------------------------------------------------------------
# one pass


def run(st):
    ctx, case = st["ctx"], st["case"]
    kind = case["kind"]
    if kind == "host":
        return spx.susceptibility(ctx, st["m"], st["ediff"], st["frqh"], nkpt=case["nk"], nkpts=st["nkpts"],
                                  precision=case["precision"])
    if kind == "chi0":
        st["out"].zero_()       # intent(out): zeroed on entry, then accumulated
        ctx.chi0_accumulate_dev(st["m"], st["ediff"], st["omega"], st["out"], wscale=st["ws"],
                                scale_all=st["scale"], precision=case["precision"], npair=_npair(case))
        return st["out"]
    if kind == "real":
        st["out"].zero_()
        ctx.chi0_accumulate_real_dev(st["m"], st["ediff"], st["omega"], st["out"], wscale=st["ws"],
                                     scale_all=st["scale"], precision=case["precision"], npair=_npair(case))
        return st["out"]
    if kind == "batched":
        st["flat"].zero_()
        ctx.chi0_batched(st["qs"], st["omega"], precision=case["precision"])
        return [q["susceph"] for q in st["qs"]]
    if kind == "products":
        st["cprod"].zero_()     # the products add into cprod
        wf.wavefproducts2_mt(ctx, st["mt"], st["c1"], st["c2"], st["cprod"])
        wf.wavefproducts2_pw(ctx, st["pw"], st["p1"], st["p2"], st["cprod"], st["col0"])
        return st["cprod"]
    if kind == "fft":
        st["cprod"].zero_()
        wf.wavefproducts2_pw(ctx, st["pw"], st["p1"], st["p2"], st["cprod"], 0)
        return st["cprod"]
    if kind == "fused":
        st["out"].zero_()
        wf.chi0_from_coeffs(ctx, st["mt"], st["pw"], st["c1"], st["c2"], st["p1"], st["p2"], st["ediff"],
                            st["omega"], st["out"], scale_all=1.0 / case["nk"], precision=case["precision"])
        return st["out"]
    if kind == "gamma":
        wf.dcprod_dev(ctx, st["mom"], case["nk"], case["nocc"], case["nunocc"], st["c1"], st["c2"], st["p1"],
                      st["p2"], st["dc"], ediff=st["ediff"])
        ctx.trafo_dev(st["cprod"], st["trafo"], out=st["body"])
        ctx.weights_dev(st["ediff"], st["omega"], st["w"], scale_all=1.0 / case["nk"])
        st["head"].zero_()
        st["wing"].zero_()
        ctx.headwings_dev(st["body"], st["dc"], st["w"], st["head"], st["wing"])
        return dict(dcprod=st["dc"], cprod=st["body"], head=st["head"], wing=st["wing"])
    st["eps"].copy_(st["chi"])  # in place: the program keeps chi
    st["h"].copy_(st["head"])
    st["g"].copy_(st["wing"])
    ctx.dielec_dev(st["eps"], st["coul"], invert=True, head=st["h"], wing=st["g"])
    return dict(inverse=st["eps"], head=st["h"], wing=st["g"])


# ---------------------------------------------------------------------------
# work: every input read once, every output written once; the operations of the sums
# themselves (a product of two M per pair and element, then one multiply-add per part
# and frequency)


def _chi0_work(N, P, nw, real=False):
    npk = N * (N + 1) // 2
    if real:
        return 8.0 * N * P + 8.0 * P + 8.0 * npk * nw, npk * float(P) * (1 + 2 * nw)
    return 16.0 * N * P + 8.0 * P + 16.0 * npk * nw, npk * float(P) * (6 + 4 * nw)


def _sphere_extent(n):
    return 2.0 * math.ceil((3 * n / (4 * math.pi)) ** (1 / 3)) + 1


def work(case):
    kind = case["kind"]
    if kind in ("host", "chi0", "real"):
        b, f = _chi0_work(case["nbas"], _npair(case), case["nw"], kind == "real")
    elif kind == "batched":
        n = 0.5 * (case["nbas_lo"] + case["nbas_hi"])
        P = case["nk"] * 0.25 * (case["occ_lo"] + case["occ_hi"]) * (case["unocc_lo"] + case["unocc_hi"])
        b, f = (case["nq"] * x for x in _chi0_work(int(n), int(P), case["nw"]))
    elif kind in ("products", "fft", "fused"):
        P, nk, no, nu = _npair(case), case["nk"], case["nocc"], case["nunocc"]
        b = 16.0 * nk * (no + nu) * case["ngpt"]
        cols = case["ngptm"]
        if kind == "fft":
            n, lg = case["nfft"], math.log2(case["nfft"])
            k = min(n, _sphere_extent(case["ngptm"]))
            f = P * (6.0 * n ** 3 + 5.0 * lg * (n ** 3 + k * n ** 2 + k * k * n))
        else:
            f = 8.0 * P * case["ngptm"] * case["ngpt"]
        if "lcut" in case:
            lm = (case["lcut"] + 1) ** 2 * case["nrad"]
            b += 16.0 * nk * (no + nu) * 2 * lm
            f += 8.0 * P * 2 * lm * lm
            cols += 2 * lm
        if kind == "fused":
            npk = cols * (cols + 1) // 2
            b += 8.0 * P + 16.0 * npk * case["nw"]
            f += npk * float(P) * (6 + 4 * case["nw"])
        else:
            b += 16.0 * P * cols
    elif kind == "gamma":
        P, N, dim, nw, ng = _npair(case), case["nbas"], case["dim"], case["nw"], case["ngpt"]
        lm = (case["lcut"] + 1) ** 2 * case["nrad"]
        b = 16.0 * (P * (N + dim + 3) + N * dim + case["nk"] * (case["nocc"] + case["nunocc"]) * (ng + 2 * lm)) + \
            16.0 * nw * (6 + 3 * dim)
        f = 8.0 * P * N * dim + 24.0 * P * (ng + 2 * lm) + 3.0 * (dim + 2) * P * (6 + 4 * nw)
    else:
        n, nw = case["nbas"], case["nw"]
        b = 2 * 16.0 * nw * (n * (n + 1) // 2 + 6 + 3 * n) + 8.0 * n
        f = 4.0 * n ** 3 * nw
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# the same outputs in plain 64-bit torch


def _weights_exact(ediff, omega, ws, scale):
    w = -2.0 * ediff / (omega[:, None] ** 2 + ediff ** 2) * scale
    return w if ws is None else w * ws


def _gram_add(G, m, w):
    """G[f] += m diag(w[f]) m^H for m (N, p), chunked over the pairs."""
    for p0 in range(0, m.shape[1], 32768):
        mc = m[:, p0:p0 + 32768]
        mh = mc.conj().T.contiguous() if mc.is_complex() else mc.T.contiguous()
        for f in range(w.shape[0]):
            G[f] += (mc * w[f, p0:p0 + 32768]) @ mh


def _gram_exact(m, w):
    G = torch.zeros((w.shape[0], m.shape[0], m.shape[0]), dtype=m.dtype, device=DEV)
    _gram_add(G, m, w)
    i, j = _tri(m.shape[0])
    return G[:, i, j]


def _mt_exact(mt, c1, c2, k):
    """cprod columns (natom*maxllm, nocc*nunocc) of k point k, muffin-tin part."""
    L, Lm, nr, nrm, na = mt["lcut"], mt["lcutm"], mt["nrad"], mt["nradm"], mt["natom"]
    if "T" not in mt:
        maxlm, maxllm = (L + 1) ** 2 * nr, (Lm + 1) ** 2 * nrm
        T = np.zeros((maxlm, maxllm, maxlm))
        gt, integ = np.asarray(mt["gaunt"]), np.asarray(mt["integral"])
        for l1, l, LL, mi, Mi in np.argwhere(gt != 0.0):
            m, M = mi - L, Mi - Lm
            m1 = m + M
            if abs(m) > l or abs(M) > LL or abs(m1) > l1:
                continue
            o, I, i = nr * (l1 * l1 + l1 + m1), nrm * (LL * LL + LL + M), nr * (l * l + l + m)
            ln1 = nr * ((l1 - abs(l - LL)) // 2)
            blk = integ[l * nr:(l + 1) * nr, ln1:ln1 + nr, LL * nrm:(LL + 1) * nrm]   # (i, j, nn)
            T[o:o + nr, I:I + nrm, i:i + nr] += gt[l1, l, LL, mi, Mi] * np.transpose(blk, (1, 2, 0))
        mt["T"] = torch.from_numpy(np.ascontiguousarray(np.transpose(T, (1, 0, 2)))).to(DEV)   # (I, o, i)
    T = mt["T"]
    nI, no_, ni = T.shape
    cols = []
    for a in range(na):
        c = c1[k, :, a, :]                                       # (nocc, i)
        t = T.reshape(nI * no_, ni)
        mat = torch.complex(t @ c.real.T.contiguous(), t @ c.imag.T.contiguous()).reshape(nI, no_, -1)
        blk = torch.einsum("po,Ion->Inp", c2[k, :, a, :], mat.conj().resolve_conj())
        cols.append(complex(mt["cexp"][a]) * blk.reshape(nI, -1))
    return torch.cat(cols)


def _pw_exact(pw, p1, p2, k):
    """cprod columns (ngptm, nocc*nunocc) of k point k, interstitial part:
    sum over G1, G2 of cpw2(G2) conj(cstep(G2 - GM + g - G1) cpw1(G1)) / sqrt(vol)."""
    g1, g2, gm = (torch.from_numpy(np.asarray(pw[n]).astype(np.int64)).to(DEV) for n in ("gpt1", "gpt2", "gptm"))
    g = torch.from_numpy(np.asarray(pw["gshift"]).astype(np.int64)).to(DEV)
    sr = int(pw["step_radius"])
    cs = np.asarray(pw["cstep"]).reshape((2 * sr + 1,) * 3, order="F")
    lo = torch.minimum(g2.min(0).values - gm.max(0).values + g, g1.min(0).values - sr)
    hi = torch.maximum(g2.max(0).values - gm.min(0).values + g, g1.max(0).values + sr)
    dim = [int(x) for x in hi - lo + 1]
    nocc = p1.shape[1]
    a = torch.zeros((nocc, *dim), dtype=C128, device=DEV)
    x = g1 - lo
    a[:, x[:, 0], x[:, 1], x[:, 2]] = p1[k]
    b = torch.zeros_like(a)
    l1, h1 = [int(v) for v in x.min(0).values], [int(v) for v in x.max(0).values]
    src = a[:, l1[0]:h1[0] + 1, l1[1]:h1[1] + 1, l1[2]:h1[2] + 1].clone()
    for dx in range(-sr, sr + 1):
        for dy in range(-sr, sr + 1):
            for dz in range(-sr, sr + 1):
                c = complex(cs[dx + sr, dy + sr, dz + sr])
                if c != 0:
                    b[:, l1[0] + dx:h1[0] + 1 + dx, l1[1] + dy:h1[1] + 1 + dy, l1[2] + dz:h1[2] + 1 + dz] += c * src
    idx = (g2[None, :, :] - gm[:, None, :] + g - lo)
    lin = (idx[..., 0] * dim[1] + idx[..., 1]) * dim[2] + idx[..., 2]       # (ngptm, ngpt2)
    b = b.reshape(nocc, -1)
    out = torch.empty((gm.shape[0], nocc, p2.shape[1]), dtype=C128, device=DEV)
    for n in range(nocc):
        out[:, n, :] = b[n][lin].conj().resolve_conj() @ p2[k].T / math.sqrt(pw["vol"])
    return out.reshape(gm.shape[0], -1)


def _dcprod_exact(a, case):
    mom = a["mom"]
    L, nr, natom, nk, ng = mom["lcut"], mom["nrad"], mom["natom"], case["nk"], case["ngpt"]
    maxlm = (L + 1) ** 2 * nr
    A = np.zeros((3, maxlm, maxlm))
    q1, q2 = mom["qmat1"], mom["qmat2"]
    at = lambda l, m: nr * (l * l + l + m)
    for l in range(L + 1):
        for m in range(-l, l + 1):
            d1 = 2 * (2 * l + 1) * (2 * l + 3)
            f = [-math.sqrt((l + m + 1) * (l + m + 2) / d1), math.sqrt((l - m + 1) * (l + m + 1) * 2 / d1),
                 -math.sqrt((l - m + 1) * (l - m + 2) / d1)]
            for x in range(3):
                m1, o = m + 1 - x, at(l, m)
                if l < L:
                    A[x, o:o + nr, at(l + 1, m1):at(l + 1, m1) + nr] += f[x] * q2[:, :, l].T
                if l > 0 and abs(m1) <= l - 1:
                    d0 = 2 * (2 * l - 1) * (2 * l + 1)
                    gg = [math.sqrt((l - m) * (l - m - 1) / d0) if x == 0 else 0.0,
                          math.sqrt((l - m) * (l + m) * 2 / d0) if x == 1 else 0.0,
                          math.sqrt((l + m) * (l + m - 1) / d0) if x == 2 else 0.0][x]
                    A[x, o:o + nr, at(l - 1, m1):at(l - 1, m1) + nr] += gg * q1[:, :, l].T
    A = torch.from_numpy(A).to(DEV).to(C128)
    out = torch.zeros((3, nk, case["nocc"], case["nunocc"]), dtype=C128, device=DEV)
    gp = torch.from_numpy(np.asarray(mom["gpt"]).astype(np.int64)).to(DEV)
    sr = int(mom["step_radius"])
    ns = 2 * sr + 1
    cs = torch.from_numpy(np.asarray(mom["cstep"])).to(DEV)                 # x fastest
    dd = gp[None, :, :] - gp[:, None, :] + sr                               # G_j - G_i
    inside = ((dd >= 0) & (dd < ns)).all(-1)
    lin = (dd[..., 0] + ns * (dd[..., 1] + ns * dd[..., 2])).clamp(0, ns ** 3 - 1)
    O = torch.where(inside, cs[lin], torch.zeros((), dtype=C128, device=DEV)).conj().resolve_conj()
    rlat = torch.from_numpy(np.ascontiguousarray(mom["rlat"])).to(DEV)
    for k in range(nk):
        for at_ in range(natom):
            c = torch.einsum("xoi,ni->xno", A, a["c1"][k, :, at_, :])
            v = torch.einsum("xno,po->xnp", c.conj().resolve_conj(), a["c2"][k, :, at_, :]) / 1j
            out[0, k] += (v[0] - v[2]) / math.sqrt(2.0)
            out[1, k] -= (v[0] + v[2]) / math.sqrt(2.0) * 1j
            out[2, k] += v[1]
        vec = a["p1"][k] @ O.T
        kk = torch.from_numpy(np.asarray(mom["kpt"][k])).to(DEV)
        qg = (gp.to(F64) + kk) @ rlat.T                                     # (ng, 3)
        for x in range(3):
            out[x, k] += (vec.conj().resolve_conj() * qg[:, x]) @ a["p2"][k].T
    return out.reshape(3, -1) / math.sqrt(mom["vol"]) / a["ediff"]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("host", "chi0", "real"):
        a = _chi0_inputs(case, seed)
        ref = _gram_exact(a["m"][:, :_npair(case)], _weights_exact(a["ediff"], a["omega"], a["ws"], a["scale"]))
        return (2.0 * ref).cpu().numpy().T if kind == "host" else ref
    if kind == "batched":
        om = _omega(case["nw"])
        return [_gram_exact(q["cprod"], _weights_exact(q["ediff"], om, None, q["scale_all"]))
                for q in _batched_inputs(case, seed)]
    if kind in ("products", "fft", "fused"):
        a = _coeff_inputs(case, seed)
        P = case["nocc"] * case["nunocc"]
        cols = lambda k: torch.cat(([_mt_exact(a["mt"], a["c1"], a["c2"], k)] if "mt" in a else []) +
                                   [_pw_exact(a["pw"], a["p1"], a["p2"], k)])
        if kind != "fused":
            return torch.cat([cols(k) for k in range(case["nk"])], dim=1)
        w = _weights_exact(_ediff(case["nk"], case["nocc"], case["nunocc"], 0.0, _gen(seed, 1)),
                           _omega(case["nw"]), None, 1.0 / case["nk"])
        n = a["w"].nbas
        G = torch.zeros((case["nw"], n, n), dtype=C128, device=DEV)
        for k in range(case["nk"]):
            _gram_add(G, cols(k), w[:, k * P:(k + 1) * P])
        i, j = _tri(n)
        return G[:, i, j]
    if kind == "gamma":
        a = _gamma_inputs(case, seed)
        dc = _dcprod_exact(a, case)
        body = a["trafo"].conj().resolve_conj() @ a["cprod"]
        w = _weights_exact(a["ediff"], a["omega"], None, 1.0 / case["nk"])
        head = torch.stack([(dc[k1] * dc[k2].conj()) .to(C128) @ w.T.to(C128)
                            for k2 in range(3) for k1 in range(k2 + 1)], dim=1)
        wing = torch.stack([torch.stack([body @ (dc[k2].conj() * w[f]) for k2 in range(3)], dim=1)
                            for f in range(case["nw"])])
        return dict(dcprod=dc, cprod=body, head=head, wing=wing)
    a = _dielec_inputs(case, seed)
    n = case["nbas"]
    i, j = _tri(n)
    sq = a["coul"].sqrt()
    inv = torch.empty_like(a["chi"])
    for f in range(case["nw"]):
        x = torch.zeros((n, n), dtype=C128, device=DEV)
        x[j, i] = a["chi"][f].conj()
        x[i, j] = a["chi"][f]
        x = torch.eye(n, dtype=C128, device=DEV) - sq[:, None] * x * sq[None, :]
        inv[f] = torch.linalg.inv(x)[i, j]
    head = -4 * math.pi * a["head"]
    head[:, [0, 2, 5]] += 1.0
    wing = -math.sqrt(4 * math.pi) * sq[None, :, None] * a["wing"]
    return dict(inverse=inv, head=head, wing=wing)
