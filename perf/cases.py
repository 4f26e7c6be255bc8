"""Performance cases of the QSGW inner loops: the calls a driver makes for one q point, from a small
test cell to the largest streamed one.

`kind` says which part of the path a case runs, through the public Python entry points of
`ecalj_b200.lib` (device arrays, as a driver that keeps its data on the GPU passes them):

  chain    chi0(i w), chi0(w), W(i w), W(w) and Sigma_c of one small cell, call after call
  chi0     chi0(i w) of every k and frequency with the Lorentzian pair weights
  hist     the tetrahedron route: x0gemm per k from pair/bin lists, then the Hilbert transform
  wimag    W - v on the imaginary axis with both basis changes
  wreal    W - v on the real axis (general matrices, pivoted inverse)
  sigc     Sigma_c of one or several tasks (k, rotation, state batch) of one q point
  zmel     <psi|psi M>: muffin-tin part, interstitial part, change to the Coulomb basis
  coulomb  eigenvectors of the Coulomb matrix and v^(1/2) from them
  interp   the W_c frequency interpolator: inference on one q's block and one gradient

`prec` is the library's precision switch ("fp64", or "i8" with `ns` int8 slices).
"""
import math

import numpy as np
import torch

from ecalj_b200 import lib, sched, synth

_PREC = {"fp64": lib.PREC_FP64, "i8": lib.PREC_SPLIT_I8}
C128 = torch.complex128


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # a two-atom test cell: every call is short, so launches and host tables count
        dict(name="chain_n96", kind="chain", N=96, nk=8, nocc=4, nun0=10, nun1=20, niw=6, nreal=40, ntq=6, nm=20,
             prec="fp64"),
        # Si, 4x4x4 k points, 12 frequencies, plain FP64 chi0
        dict(name="chi0_si_fp64", kind="chi0", N=260, nk=64, nocc=4, nun0=40, nun1=60, niw=12, prec="fp64", ns=1),
        # GaAs-like cell, 6x6x6 k points with uneven band windows, the int8 path of the benchmark
        dict(name="chi0_gaas_i8", kind="chi0", N=600, nk=216, nocc=9, nun0=100, nun1=300, niw=24, prec="i8", ns=3),
        # tetrahedron histogram of an odd-sized cell, 16 k points, both frequency axes
        dict(name="hist_n233_fp64", kind="hist", N=233, nk=16, nocc=4, nun=50, nwhis=96, niw=12, nw=60, width=3,
             prec="fp64", ns=1),
        # W at every imaginary frequency of the GaAs-like cell
        dict(name="wimag_n600", kind="wimag", N=600, niw=24),
        # W on the real axis of the Si cell
        dict(name="wreal_n260", kind="wreal", N=260, nw=50),
        # Sigma_c of one Si task in plain FP64
        dict(name="sigc_si_fp64", kind="sigc", N=260, ntq=20, nm=150, niw=12, nreal=50, ntask=1, prec="fp64", ns=1,
             keepwv=False),
        # Sigma_c of the benchmark: 8 tasks of 40 x 400 states, int8
        dict(name="sigc_gaas_i8", kind="sigc", N=600, ntq=40, nm=400, niw=24, nreal=50, ntask=8, prec="i8", ns=3,
             keepwv=False),
        # one task of the large streamed cell at the most accurate slice count, W kept packed
        dict(name="sigc_large_i8x4", kind="sigc", N=1500, ntq=40, nm=200, niw=32, nreal=50, ntask=1, prec="i8", ns=4,
             keepwv=True),
        # matrix elements of a two-atom cell, one (q, k) pair
        dict(name="zmel_n500", kind="zmel", natom=2, nc=3, nv=25, mdim=150, ngc=200, ngp=150, nm=200, ntp0=40,
             prec="fp64", ns=1),
        # the Coulomb eigenproblem of the Si cell
        dict(name="coulomb_n260", kind="coulomb", N=260),
        # the interpolator: 32 predicted points of a 64 x 64 block, and one training batch
        dict(name="interp_block64", kind="interp", rows=262144, batch=8192),
    ]


def _logu(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the same ranges: sizes over their logarithm, odd ones among them."""
    kind = rng.choice(["chain", "chi0", "chi0", "hist", "wimag", "wreal", "sigc", "sigc", "sigc", "zmel", "coulomb",
                       "interp"])
    prec = rng.choice(["fp64", "i8", "i8"])
    ns = 1 if prec == "fp64" else rng.choice([3, 4])
    if kind == "chain":
        nun0 = rng.randint(6, 20)
        return dict(kind=kind, N=_logu(rng, 40, 160), nk=rng.randint(2, 16), nocc=rng.randint(2, 6), nun0=nun0,
                    nun1=nun0 + rng.randint(0, 20), niw=rng.randint(4, 12), nreal=rng.randint(30, 50),
                    ntq=rng.randint(4, 12), nm=rng.randint(12, 60), prec="fp64")
    if kind == "chi0":
        while True:
            nun0 = rng.randint(20, 150)
            c = dict(kind=kind, N=_logu(rng, 96, 640), nk=_logu(rng, 8, 216), nocc=rng.randint(3, 12), nun0=nun0,
                     nun1=nun0 + rng.randint(0, 120), niw=rng.randint(6, 32), prec=prec, ns=ns)
            if work(c)["flops"] <= (1e12 if prec == "fp64" else 6e12):
                return c
    if kind == "hist":
        nwhis = rng.randint(60, 120)
        return dict(kind=kind, N=_logu(rng, 80, 320), nk=rng.randint(4, 16), nocc=rng.randint(2, 8),
                    nun=rng.randint(20, 80), nwhis=nwhis, niw=rng.randint(6, 24), nw=rng.randint(20, nwhis - 2),
                    width=rng.randint(1, 6), prec=prec, ns=1 if prec == "fp64" else 4)
    if kind == "wimag":
        return dict(kind=kind, N=_logu(rng, 96, 640), niw=rng.randint(4, 32))
    if kind == "wreal":
        return dict(kind=kind, N=_logu(rng, 64, 320), nw=rng.randint(16, 60))
    if kind == "sigc":
        while True:
            c = dict(kind=kind, N=_logu(rng, 96, 1500), ntq=rng.randint(8, 48), nm=_logu(rng, 40, 400),
                     niw=rng.randint(6, 32), nreal=rng.randint(40, 60), ntask=rng.choice([1, 1, 2, 4, 8]), prec=prec,
                     ns=ns, keepwv=rng.random() < 0.25)
            if work(c)["flops"] <= (1e12 if prec == "fp64" else 6e12) and c["N"] ** 2 * c["ntask"] <= 5e6:
                return c
    if kind == "zmel":
        return dict(kind=kind, natom=rng.randint(1, 4), nc=rng.randint(0, 4), nv=rng.randint(9, 36),
                    mdim=rng.randint(30, 160), ngc=_logu(rng, 40, 240), ngp=_logu(rng, 40, 180), nm=_logu(rng, 20, 300),
                    ntp0=rng.randint(4, 48), prec=prec, ns=ns)
    if kind == "coulomb":
        return dict(kind=kind, N=_logu(rng, 64, 300))
    return dict(kind=kind, rows=_logu(rng, 4096, 262144), batch=_logu(rng, 512, 16384))


# ------------------------------------------------------------------ inputs
_started = False


def _start(case):
    global _started
    if not _started:
        lib.load()
        lib.init(0)
        lib.share_torch_stream()
        _started = True
    p = case.get("prec", "fp64")
    lib.set_precision(_PREC[p], case["ns"] if p != "fp64" else 1)


class _Rand:
    """Seeded inputs: a numpy generator for tables and a device generator for the large arrays."""

    def __init__(self, seed):
        self.np = np.random.default_rng(seed)
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed)

    def cplx(self, *shape, scale=1.0):
        x = torch.randn(*shape, 2, dtype=torch.float64, device="cuda", generator=self.g)
        return torch.view_as_complex(x.mul_(scale))


def _bands(case, r):
    nocc, nun, eo, eu = synth.chi0_spectrum(r.np, case["nk"], case["nocc"], (case["nun0"], case["nun1"]))
    return nocc, nun, np.concatenate(eo) * 0.5, np.concatenate(eu) * 0.5


def _unitary(n, r):
    return torch.linalg.qr(r.cplx(n, n))[0].contiguous()


def _vcousq(n, r):
    return np.sqrt(10.0 ** r.np.uniform(-2.0, 3.0, n))


def _wc_stack(n, freq, r, real_axis):
    """W - v of a plasmon-pole model, (slot, N, N): -B diag(a f(w)) B^H with a pole per mode; on the real
    axis f is complex (W not Hermitian), as a broadened response is."""
    b = r.cplx(n, n, scale=1.0 / math.sqrt(n))
    a = torch.from_numpy(10.0 ** r.np.uniform(-1.0, 2.0, n)).cuda()
    wp = torch.from_numpy(r.np.uniform(0.2, 2.0, n)).cuda()
    out = torch.empty(len(freq), n, n, dtype=C128, device="cuda")
    for i, w in enumerate(freq):
        f = wp ** 2 / ((wp ** 2 - (w + 0.05j) ** 2) if real_axis else (wp ** 2 + w * w))
        out[i] = torch.matmul(b * (-a * f).to(C128)[None, :], b.conj().T)
    return out


def _sigc_task(case, r):
    n, ntq, nm = case["N"], case["ntq"], case["nm"]
    mesh = synth.imag_mesh(case["niw"])
    omega = np.sort(r.np.uniform(-1.0, 1.0, ntq))
    ekc = np.sort(r.np.uniform(-1.0, 4.0, nm))
    fr = synth.freq_r_mesh(case["nreal"])
    ef, esmr = 0.0, 0.01
    nwxi, nwx, ntmax = sched.get_nwx(omega, ekc, fr, ef, esmr)
    zmel = r.cplx(ntq, nm, n, scale=1.0 / math.sqrt(n))
    return dict(zsec=torch.zeros(ntq * ntq, dtype=C128, device="cuda"), zmel=zmel, ns1=1, ns2=nm,
                ns2r=min(nm, ntmax), nwxi=nwxi, nwx=nwx, ntqxx=ntq, wc_imag=None, wc_real=None, omega=omega, ekc=ekc,
                nctot=0, ef=ef, esmr=esmr, wkkr=1.0 / 8, ua=mesh["ua"], freqx=mesh["x"], wwx=mesh["wx"],
                expa=mesh["expa"], freq_r=fr, keepwv=bool(case.get("keepwv")), nblochpmx=n, ngb=n, ntq=ntq), mesh


def _pack_upper(w):
    """Packed upper triangles (column by column) of a stack whose torch layout is (slot, column, row)."""
    n = w.shape[-1]
    j, i = torch.tril_indices(n, n, device=w.device)
    return w[:, j, i].contiguous()


def _hermitian_part(w):
    return (w + w.transpose(-1, -2).conj()) * 0.5


def _chi0_like(n, freq, r, eta=None):
    """chi0 of n random pairs per row at the given frequencies, (slot, N, N)."""
    g = r.cplx(n, 2 * n, scale=1.0 / math.sqrt(n))
    de = torch.from_numpy(r.np.uniform(0.05, 2.4, 2 * n)).cuda()
    out = torch.empty(len(freq), n, n, dtype=C128, device="cuda")
    for i, w in enumerate(freq):
        if eta is None:
            f = -2.0 * de / (de * de + w * w)
        else:
            f = 1.0 / (w - de + 1j * eta) - 1.0 / (w + de + 1j * eta)
        out[i] = torch.matmul(g * f.to(C128)[None, :], g.conj().T)
    return out


def _zmel_tables(case, r):
    atoms, ppb = [], []
    ias = ims = 1
    ics = 0
    for _ in range(case["natom"]):
        nc, nv, md = case["nc"], case["nv"], case["mdim"]
        p = torch.randn(md, nc + nv, nc + nv, dtype=torch.float64, device="cuda", generator=r.g)
        ppb.append(p)
        atoms.append(dict(nc=nc, nv=nv, ias=ias, ics=ics, ims=ims, ncore=nc, nlnm=nc + nv, mdim=md,
                          phase=complex(np.exp(2j * math.pi * r.np.random())), ppb_d=p))
        ias += nv
        ims += md
        ics += nc
    return atoms, ppb


def prepare(case, seed):
    _start(case)
    r = _Rand(seed)
    kind = case["kind"]
    s = dict(case=case)
    if kind in ("chain", "chi0"):
        s["bands"] = _bands(case, r)
        npair = int(np.sum(s["bands"][0] * s["bands"][1]))
        s["z"] = r.cplx(npair, case["N"], scale=1.0 / math.sqrt(case["N"]))
        s["freq"] = synth.imag_mesh(case["niw"])["freq_i"]
    n = case.get("N", 0)
    if kind == "chi0":
        s["chi"] = torch.empty(case["niw"], n, n, dtype=C128, device="cuda")
    elif kind == "chain":
        s["task"], mesh = _sigc_task(case, r)
        s["freq"] = np.concatenate([[0.0], mesh["freq_i"]])
        s["vsq"], s["m2e"] = _vcousq(n, r), _unitary(n, r)
        s["eta"] = 0.05
        nr = case["nreal"]
        s["chi"] = torch.empty(case["niw"] + 1, n, n, dtype=C128, device="cuda")
        s["chir"] = torch.empty(nr, n, n, dtype=C128, device="cuda")
        s["wi"], s["wr"] = torch.empty_like(s["chi"]), torch.empty_like(s["chir"])
        s["task"].update(wc_imag=s["wi"], wc_real=s["wr"])
    elif kind == "hist":
        nm, nq, nb, npair = case["nocc"], case["nun"], case["nwhis"], case["nocc"] * case["nun"]
        s["z"] = r.cplx(case["nk"], nq, nm, n, scale=1.0 / math.sqrt(n))
        s["frhis"] = 0.02 * (np.exp(0.04 * np.arange(nb + 1)) - 1.0)
        s["freq_i"] = synth.imag_mesh(case["niw"])["freq_i"]
        s["freq_r"] = np.concatenate([[0.0], 0.5 * (s["frhis"][:-1] + s["frhis"][1:])])[:case["nw"] + 1]
        tabs = []
        for _ in range(case["nk"]):
            ini = r.np.integers(1, nb + 2 - case["width"], npair)
            end = ini + r.np.integers(0, case["width"], npair)
            cnt = end - ini + 1
            it, itp = np.meshgrid(np.arange(1, nm + 1), np.arange(1, nq + 1))
            tabs.append(tuple(np.ascontiguousarray(a, dtype=np.int32) for a in (
                it.ravel(), itp.ravel(), np.ones(npair), ini, end, np.concatenate([[1], 1 + np.cumsum(cnt)[:-1]])))
                + (r.np.uniform(0.01, 1.0, int(cnt.sum())),))
        s["tabs"] = tabs
        s["rcxq"] = torch.empty(nb + 1, n, n, dtype=C128, device="cuda")
        s["zxqi"] = torch.empty(case["niw"], n, n, dtype=C128, device="cuda")
        s["zxq"] = torch.empty(case["nw"] + 1, n, n, dtype=C128, device="cuda")
    elif kind == "wimag":
        s["chi"] = _chi0_like(n, synth.imag_mesh(case["niw"])["freq_i"], r)
        s["vsq"], s["m2e"] = _vcousq(n, r), _unitary(n, r)
        s["w"] = torch.empty_like(s["chi"])
    elif kind == "wreal":
        s["chi"] = _chi0_like(n, synth.freq_r_mesh(case["nw"]), r, eta=0.1)
        s["vsq"] = _vcousq(n, r)
        s["w"] = torch.empty_like(s["chi"])
    elif kind == "sigc":
        s["tasks"], s["mesh"] = [], None
        for _ in range(case["ntask"]):
            t, s["mesh"] = _sigc_task(case, r)
            wi = _wc_stack(n, np.concatenate([[0.0], s["mesh"]["freq_i"]]), r, False)
            wr = _wc_stack(n, t["freq_r"], r, True)
            if t["keepwv"]:
                wi, wr = _pack_upper(_hermitian_part(wi)), _pack_upper(_hermitian_part(wr))
            t.update(wc_imag=wi, wc_real=wr)
            s["tasks"].append(t)
    elif kind == "zmel":
        s["atoms"], s["ppb"] = _zmel_tables(case, r)
        nbl = case["natom"] * case["mdim"]
        nda, ntp0, nm, ngp = case["natom"] * case["nv"], case["ntp0"], case["nm"], case["ngp"]
        s["nbloch"], s["ndima"] = nbl, nda
        s["cphim"], s["cphiq"] = r.cplx(nm, nda), r.cplx(ntp0, nda)
        s["geigq"], s["dgeigqk"] = r.cplx(ntp0, ngp), r.cplx(nm, ngp)
        pts = np.stack(np.meshgrid(*[np.arange(-3, 4)] * 3, indexing="ij")).reshape(3, -1).astype(np.int32)
        near = pts[:, np.argsort((pts ** 2).sum(0), kind="stable")]
        s["b1"], s["b2"] = near[:, :ngp].copy(), near[:, :ngp].copy()
        s["gc"] = near[:, :case["ngc"]].copy()
        comp = np.concatenate([(s["gc"][:, :, None] + s["b2"][:, None, :]).reshape(3, -1),
                               (s["gc"][:, :, None] - s["b1"][:, None, :]).reshape(3, -1)], axis=1)
        s["comp"] = np.ascontiguousarray(np.unique(comp, axis=1).astype(np.int32))
        box = np.stack(np.meshgrid(*[np.arange(-9, 10)] * 3, indexing="ij")).reshape(3, -1).astype(np.int32)
        s["nvggg"] = np.ascontiguousarray(box[:, r.np.random(box.shape[1]) < 0.8])
        k = s["nvggg"].shape[1]
        s["ggg"] = r.np.standard_normal(k) + 1j * r.np.standard_normal(k)
        s["phase"] = np.exp(-2j * np.pi * r.np.random(case["ngc"]))
        ngb = nbl + case["ngc"]
        s["m2e"] = _unitary(ngb, r)
        s["zt"] = torch.empty(ntp0, nm, ngb, dtype=C128, device="cuda")
        s["mt"] = torch.empty(ntp0, nm, nbl, dtype=C128, device="cuda")
        s["zmel"] = torch.empty_like(s["zt"])
    elif kind == "coulomb":
        q = _unitary(n, r)
        lam = torch.from_numpy(10.0 ** r.np.uniform(-2.0, 3.0, n)).cuda()
        v = torch.matmul(q * lam.to(C128)[None, :], q.conj().T)
        s["v"] = _hermitian_part(v).contiguous()
        s["x"], s["out"] = torch.empty_like(s["v"]), torch.empty_like(s["v"])
    elif kind == "interp":
        _interp_parameters()
        for name, m in (("inf", case["rows"]), ("trn", case["batch"])):
            x = torch.rand(m, 16, dtype=torch.float32, device="cuda", generator=r.g) * 2 - 1
            x[:, 15] = 0.0
            s["x_" + name] = x.contiguous()
            s["t_" + name] = torch.randint(0, 64, (m,), dtype=torch.int32, device="cuda", generator=r.g)
        s["y_trn"] = torch.randn(case["batch"], dtype=torch.float32, device="cuda", generator=r.g)
        s["w_trn"] = torch.rand(case["batch"], dtype=torch.float32, device="cuda", generator=r.g) + 0.1
        s["y"] = torch.empty(case["rows"], dtype=torch.float32, device="cuda")
    return s


def _interp_values():
    rng = np.random.default_rng(99)
    p = rng.standard_normal(16 * 256 + 256 + 256 * 256 + 256 + 256 + 1 + 128 * 16) * 0.06
    return p.astype(np.float32)


def _interp_parameters():
    """The network's trained parameters: one network per process, the same for every state."""
    lib.wsurr_init(1)
    lib.wsurr_params(_interp_values())


# ------------------------------------------------------------------ one pass
def run(s):
    c = s["case"]
    kind, n = c["kind"], c.get("N", 0)
    if kind == "chi0":
        lib.chi0_lorentz_d(s["chi"], n, c["niw"], s["freq"], c["nk"], *s["bands"], s["z"])
        return s["chi"]
    if kind == "chain":
        m = c["niw"] + 1
        lib.chi0_lorentz_d(s["chi"], n, m, s["freq"], c["nk"], *s["bands"], s["z"])
        lib.chi0_lorentz_real_d(s["chir"], n, c["nreal"], s["task"]["freq_r"], s["eta"], c["nk"], *s["bands"], s["z"])
        lib.wvi_llw(s["chi"], 2, s["vsq"], s["m2e"], True, True, 2, zw=s["wi"], device=True, ngb=n, niw=m)
        lib.wvr_llw_d(s["chir"], n, c["nreal"], 2, s["vsq"], s["m2e"], True, True, 2, s["wr"])
        s["task"]["zsec"].zero_()
        lib.sxcf_correlation(**s["task"], device=True)
        return [s["chi"], s["chir"], s["wi"], s["wr"], s["task"]["zsec"]]
    if kind == "hist":
        nm, nq = c["nocc"], c["nun"]
        s["rcxq"].zero_()
        for k in range(c["nk"]):
            it, itp, jpm, ini, end, off, whw = s["tabs"][k]
            lib.x0gemm(s["rcxq"], n, 1, n, c["nwhis"], 1, 1, nm, s["z"][k], 1, 1, len(it), it, itp, jpm, ini, end,
                       off, whw, zmel_shape=(n, nm, nq), device=True)
        lib.dpsion_chiq_d(s["rcxq"], n, n, c["nwhis"], s["frhis"], s["freq_i"], s["freq_r"], zxqi=s["zxqi"],
                          zxq=s["zxq"])
        return [s["rcxq"], s["zxqi"], s["zxq"]]
    if kind == "wimag":
        return lib.wvi_llw(s["chi"], 2, s["vsq"], s["m2e"], True, True, 2, zw=s["w"], device=True, ngb=n, niw=c["niw"])
    if kind == "wreal":
        return lib.wvr_llw_d(s["chi"], n, c["nw"], 2, s["vsq"], None, False, False, 2, s["w"])
    if kind == "sigc":
        for t in s["tasks"]:
            t["zsec"].zero_()
        if len(s["tasks"]) == 1:
            return lib.sxcf_correlation(**s["tasks"][0], device=True)
        return lib.sxcf_correlation_batch_d(s["tasks"])
    if kind == "zmel":
        nm, ntp0, nbl, ngc, ngp = c["nm"], c["ntp0"], s["nbloch"], c["ngc"], c["ngp"]
        ngb = nbl + ngc
        s["mt"].zero_()
        lib.zmel_mt_d(s["mt"], nbl, 1, nm, 0, ntp0, s["cphim"], s["ndima"], s["cphiq"], s["ndima"], s["atoms"])
        s["zt"][:, :, :nbl] = s["mt"]
        lib.zmel_ipw_d(s["zt"], ngb, nbl, 1, nm, 1, nm, ntp0, s["geigq"], ngp, s["dgeigqk"], ngp, s["b1"], s["b2"],
                       s["gc"], s["comp"], s["nvggg"], s["ggg"], (0, 0, 0), s["phase"])
        return lib.zmel_m2e_d(s["zmel"], s["zt"], ngb, ngb, nm, ntp0, s["m2e"], False, True)
    if kind == "coulomb":
        s["x"].copy_(s["v"])
        vcoud = lib.zhegv_d(s["x"], n)
        zs = s["x"] * torch.from_numpy(np.sqrt(vcoud)).to("cuda").to(C128)[:, None]
        lib.zmm(zs, s["x"], s["out"], n, n, n, 0, 2, beta=0.0, device=True)
        return [vcoud, s["out"]]
    lib.wsurr_forward_d(s["x_inf"], s["t_inf"], s["y"], c["rows"])
    loss, grad = lib.wsurr_grad_d(s["x_trn"], s["t_trn"], s["y_trn"], c["batch"], s["w_trn"])
    return [s["y"], loss, grad]


# ------------------------------------------------------------------ what a pass cannot do without
def _chi0_work(c, slots, npair):
    n = c["N"]
    # Hermitian output: half of the 8 N^2 flops a pair and frequency
    return 16.0 * n * npair + 16.0 * n * n * slots, 4.0 * n * n * npair * slots


def _w_work(n, slots, basis):
    # inverse 8 N^3, each basis change two products of 8 N^3
    return 32.0 * n * n * slots, slots * 8.0 * n ** 3 * (1 + 4 * basis)


def _sigc_work(c):
    n, ncol, slots = c["N"], c["ntq"] * c["nm"], c["niw"] + 1
    pole = 0.12 * ncol                      # states between the target energy and the Fermi level, 3 records each
    rec = 0.5 if c.get("keepwv") else 1.0
    b = 16.0 * n * ncol + 16.0 * n * n * (slots + 0.7 * c["nreal"]) * rec
    f = 8.0 * n * n * (ncol * slots + 3 * pole) + 8.0 * n * c["nm"] * c["ntq"] ** 2
    return b, f


def work(case):
    c, kind, n = case, case["kind"], case.get("N", 0)
    if kind in ("chi0", "chain"):
        npair = c["nk"] * c["nocc"] * (c["nun0"] + c["nun1"]) / 2
    if kind == "chi0":
        b, f = _chi0_work(c, c["niw"], npair)
    elif kind == "chain":
        b, f = _chi0_work(c, c["niw"] + 1 + 2 * c["nreal"], npair)
        for x in (_w_work(n, c["niw"] + 1 + c["nreal"], True), _sigc_work(c)):
            b, f = b + x[0], f + x[1]
    elif kind == "hist":
        npair = c["nk"] * c["nocc"] * c["nun"]
        b = 16.0 * n * npair + 16.0 * n * n * (c["nwhis"] + 1 + c["niw"] + c["nw"] + 1)
        # the transform matrix is real: 4 flops an element
        f = 4.0 * n * n * npair * (c["width"] + 1) / 2 + 4.0 * n * n * c["nwhis"] * (c["niw"] + c["nw"] + 1)
    elif kind == "wimag":
        b, f = _w_work(n, c["niw"], True)
    elif kind == "wreal":
        b, f = _w_work(n, c["nw"], False)
    elif kind == "sigc":
        b, f = (c["ntask"] * x for x in _sigc_work(c))
    elif kind == "zmel":
        nbl, ncol, ngp = c["natom"] * c["mdim"], c["nm"] * c["ntp0"], c["ngp"]
        ngb = nbl + c["ngc"]
        b = 16.0 * ncol * ngb + 16.0 * ngb * ngb + 8.0 * c["natom"] * c["mdim"] * c["nv"] ** 2
        first = min(c["nm"], c["ntp0"])
        f = (8.0 * nbl * c["nv"] * ncol + 4.0 * nbl * c["nv"] ** 2 * c["ntp0"] + 8.0 * ngb * ngb * ncol
             + 8.0 * c["ngc"] * ngp * (ngp * first + ncol))
    elif kind == "coulomb":
        # tridiagonalisation and back transformation, then v^(1/2)
        b, f = 64.0 * n * n, 4.0 * (9.0 + 2.0) * n ** 3
    else:
        per = 2.0 * (16 * 256 + 256 * 256 + 256 + 16)
        b, f = 72.0 * (c["rows"] + c["batch"]), per * (c["rows"] + 3 * c["batch"])
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------ how far another correct implementation may be
def tolerance(case):
    """About four times the distance of two roundings of the same sums, measured against `exact`."""
    kind = case["kind"]
    if case.get("prec") == "i8":
        three = case["ns"] == 3
        if kind in ("chi0", "hist"):                 # 7 bits a slice: 5e-6 / 6e-7 from 64 bits
            return {"rel": 2e-5, "max": 2e-3} if three else {"rel": 2e-6, "max": 2e-4}
        # 8 bits a slice: 3e-7 / 2e-9
        return {"rel": 1.5e-6, "max": 1.5e-4} if three else {"rel": 1e-8, "max": 1e-6}
    if kind in ("wimag", "wreal", "chain"):
        return {"rel": 1e-11, "max": 1e-9}           # condition of eps~: 1e-12
    if kind == "interp":
        return {"rel": 4e-3, "max": 0.1}             # BF16 operands of the hidden layer: 1e-2 from 64 bits
    return {"rel": 1e-12, "max": 1e-10}


# ------------------------------------------------------------------ the same results in 64 bits, plain torch / numpy
def _exact_chi0(z, bands, freq, nk, eta=None):
    nocc, nun, eo, eu = bands
    de, a, b = [], 0, 0
    for k in range(nk):
        de.append((eu[b:b + nun[k], None] - eo[None, a:a + nocc[k]]).ravel())
        a, b = a + nocc[k], b + nun[k]
    de = torch.from_numpy(np.concatenate(de)).cuda()
    out = []
    for w in freq:
        f = -2.0 * de / (de * de + w * w) if eta is None else 1 / (w - de + 1j * eta) - 1 / (w + de + 1j * eta)
        # chi0(i, j) = sum_p f conj(z_pi) z_pj, stored (j, i)
        out.append(torch.matmul((z * (f / nk).to(C128)[:, None]).T, z.conj()))
    return torch.stack(out)


def _exact_w(chi, vsq, m2e, basis):
    """chi stored (slot, column, row); W - v the same way."""
    v = torch.from_numpy(vsq).cuda().to(C128)
    x = chi.transpose(1, 2)
    q = m2e.T if basis else None
    if basis:
        x = q.conj().T @ x @ q
    eps = torch.eye(len(vsq), dtype=C128, device="cuda") - v[:, None] * x * v[None, :]
    w = v[:, None] * torch.linalg.inv(eps) * v[None, :] - torch.diag(v * v)
    if basis:
        w = q @ w @ q.conj().T
    return w.transpose(1, 2).contiguous()


def _gauss_window(a, b, e, sm):
    lo, hi = min(a, b), max(a, b)
    return 0.5 * math.erfc((e - hi) / math.sqrt(2) / sm) - 0.5 * math.erfc((e - lo) / math.sqrt(2) / sm)


def _exact_sigc(t, unpack):
    n, ntq, nm, sm, ef = t["ngb"], t["ntq"], t["ns2"], t["esmr"], t["ef"]
    x, wt, ex, ua, fr = t["freqx"], t["wwx"], t["expa"], t["ua"], t["freq_r"]
    om, ek = t["omega"], t["ekc"]
    we = 0.5 * (om[:, None] - ek[None, :nm]).ravel()                    # column c = it + nm itp
    sig2 = 2.0 * (0.5 * sm) ** 2
    o2 = (1.0 / x - 1.0)[None, :] ** 2 + we[:, None] ** 2
    cons = -np.expm1(-o2 / sig2) / o2
    wg = np.empty((len(we), len(x) + 1))
    wg[:, 1:] = -we[:, None] * cons * (wt / x ** 2 / np.pi)[None, :]
    erfc = lambda y: torch.special.erfc(torch.from_numpy(y)).numpy()
    aw = np.abs(ua * we)
    wg[:, 0] = (we * (cons * (ex * wt / x ** 2)[None, :]).sum(1) / np.pi
                + np.where(np.signbit(we), -0.5, 0.5) * np.exp(aw ** 2)
                * (erfc(np.sqrt(aw ** 2 + we ** 2 / sig2)) - erfc(aw)))
    wg = torch.from_numpy(wg * t["wkkr"]).cuda()
    z = t["zmel"].reshape(-1, n)
    cz = torch.zeros_like(z)
    wi, wr = t["wc_imag"], t["wc_real"]
    for i in range(len(x) + 1):
        w = unpack(wi[i])
        cz += (z * wg[:, i].to(C128)[:, None]) @ w.conj().T
    # poles: three records around |omega - e| / 2, quadratic in the frequency squared
    nt0p = int(np.sum(ek < ef + 10 * sm))
    nt0m = int(np.sum(ek < ef - 10 * sm))
    bins = {}
    for q in range(ntq):
        lo, hi = (nt0m, t["ns2r"]) if om[q] >= ef else (0, min(nt0p, t["ns2r"]))
        for i in range(lo, hi):
            wf = _gauss_window(om[q], ef, ek[i], sm)
            if abs(om[q] - ef) < 1e-6 or wf < 1e-8:
                continue
            a, b = min(om[q], ef), max(om[q], ef)
            ebar = ek[i] + sm / math.sqrt(2 * math.pi) * (math.exp(-(a - ek[i]) ** 2 / (2 * sm * sm))
                                                          - math.exp(-(b - ek[i]) ** 2 / (2 * sm * sm))) / wf
            e = 0.5 * abs(om[q] - ebar)
            k = int(np.nonzero(fr[1:] > e)[0][0]) + 1
            f2 = fr[k - 1:k + 2] ** 2
            for j in range(3):
                l = [m for m in range(3) if m != j]
                c3 = (e * e - f2[l[0]]) * (e * e - f2[l[1]]) / ((f2[j] - f2[l[0]]) * (f2[j] - f2[l[1]]))
                bins.setdefault(k - 1 + j, []).append((i + nm * q, c3 * wf * t["wkkr"] * (1 if om[q] >= ef else -1)))
    for b, ent in bins.items():
        cols = torch.tensor([e[0] for e in ent], device="cuda")
        wts = torch.tensor([e[1] for e in ent], dtype=torch.float64, device="cuda").to(C128)
        w = _hermitian_part(unpack(wr[b]))
        cz[cols] += (z[cols] * wts[:, None]) @ w.conj().T
    s = t["zmel"].reshape(ntq, -1) @ cz.reshape(ntq, -1).conj().T        # stored (column, row)
    d = s.diagonal()
    s = s - torch.diag(torch.clamp(d.imag, min=0.0) * 1j)
    return s.reshape(-1)


def _unpacker(n):
    j, i = torch.tril_indices(n, n, device="cuda")

    def f(p):
        w = torch.zeros(n, n, dtype=C128, device="cuda")
        w[j, i] = p                               # the upper triangle, stored (column, row)
        d = torch.diag(w.diagonal())
        return w + w.conj().T - d.real.to(C128)
    return f


def _exact_hilbert(frhis, zs):
    """rows z, columns bins 1..nwhis: the weights of f(bin centre) in int f(w) / (w - z) dw, f odd in w and
    linear between the centres, zero at w = 0 and beyond the last edge."""
    nb = len(frhis) - 1
    c = 0.5 * (frhis[:-1] + frhis[1:])
    z = (np.asarray(zs, dtype=np.complex128) + 1e-13j)[:, None]

    def piece(a, b, f0, f1):                      # int_a^b of the line through (a', f0), (b', f1)
        da, db = z - a, z - b
        ok = (np.abs(da) > 1e-8) & (np.abs(db) > 1e-8)
        lg = np.where(ok, np.log(np.where(ok, db, 1) / np.where(ok, da, 1)), 0)
        return np.where(ok, z * lg + (b - a), 0), lg

    def side(cc, left, right, first, last):
        out = np.zeros((len(zs), nb), np.complex128)
        for k in range(nb):
            prev = first if k == 0 else cc[k - 1]
            nxt = last if k == nb - 1 else cc[k + 1]
            m, g = piece(left[k], cc[k], 0, 0)
            out[:, k:k + 1] += (m - g * prev) / (cc[k] - prev)
            if k > 0:
                out[:, k - 1:k] += (g * cc[k] - m) / (cc[k] - prev)
            m, g = piece(cc[k], right[k], 0, 0)
            out[:, k:k + 1] += (g * nxt - m) / (nxt - cc[k])
            if k < nb - 1:
                out[:, k + 1:k + 2] += (m - g * cc[k]) / (nxt - cc[k])
        return out

    pos = side(c, frhis[:-1], frhis[1:], 0.0, frhis[-1])
    neg = side(-c[::-1], -frhis[:0:-1], -frhis[-2::-1], -frhis[-1], 0.0)[:, ::-1]
    return (pos - neg).real / np.pi


def exact(case, seed):
    s = prepare(case, seed)
    c, kind, n = case, case["kind"], case.get("N", 0)
    if kind == "chi0":
        return _exact_chi0(s["z"], s["bands"], s["freq"], c["nk"])
    if kind == "chain":
        chi = _exact_chi0(s["z"], s["bands"], s["freq"], c["nk"])
        chir = _exact_chi0(s["z"], s["bands"], s["task"]["freq_r"], c["nk"], s["eta"])
        wi, wr = _exact_w(chi, s["vsq"], s["m2e"], True), _exact_w(chir, s["vsq"], s["m2e"], True)
        return [chi, chir, wi, wr, _exact_sigc(dict(s["task"], wc_imag=wi, wc_real=wr), lambda w: w)]
    if kind == "hist":
        nm = c["nocc"]
        rc = torch.zeros_like(s["rcxq"])
        for k in range(c["nk"]):
            it, itp, _, ini, end, off, whw = s["tabs"][k]
            z = s["z"][k].reshape(-1, n)
            col = (it - 1) + nm * (itp - 1)
            for b in range(1, c["nwhis"] + 1):
                e = np.nonzero((ini <= b) & (end >= b))[0]
                if len(e):
                    zc = z[torch.from_numpy(col[e].astype(np.int64)).cuda()]
                    w = torch.from_numpy(whw[b - ini[e] + off[e] - 1]).cuda().to(C128)
                    rc[b] += (zc * w[:, None]).T @ zc.conj()
        fh = s["frhis"]
        norm = torch.from_numpy(-1.0 / np.diff(fh)).cuda().to(C128)
        r = rc.clone()
        r[1:] *= norm[:, None, None]
        flat = r[1:].reshape(c["nwhis"], -1)
        mi = torch.from_numpy(_exact_hilbert(fh, 1j * s["freq_i"])).cuda().to(C128)
        mr = torch.from_numpy(_exact_hilbert(fh, s["freq_r"])).cuda().to(C128)
        return [rc, (mi @ flat).reshape(-1, n, n), 1j * r[:c["nw"] + 1] + (mr @ flat).reshape(-1, n, n)]
    if kind == "wimag":
        return _exact_w(s["chi"], s["vsq"], s["m2e"], True)
    if kind == "wreal":
        return _exact_w(s["chi"], s["vsq"], None, False)
    if kind == "sigc":
        out = [_exact_sigc(t, _unpacker(n) if t["keepwv"] else (lambda w: w)) for t in s["tasks"]]
        return out[0] if len(out) == 1 else out
    if kind == "zmel":
        nm, ntp0, nv = c["nm"], c["ntp0"], c["nv"]
        rows = []
        for a, p in zip(s["atoms"], s["ppb"]):
            v = p[:, c["nc"]:, c["nc"]:].to(C128)                        # (i, column, row) of ppb
            cm = s["cphim"][:, a["ias"] - 1:a["ias"] - 1 + nv]
            cq = s["cphiq"][:, a["ias"] - 1:a["ias"] - 1 + nv]
            # sum_ab conj(cm_a) ppb(b, a) cq_b
            rows.append(a["phase"] * torch.einsum("ta,iab,qb->qti", cm.conj(), v, cq))
        lo = s["nvggg"].min(1) - 12
        dim = s["nvggg"].max(1) - lo + 13
        lut = np.zeros(dim, np.complex128)
        lut[tuple(s["nvggg"] - lo[:, None])] = s["ggg"]
        g = torch.empty(ntp0, nm, c["ngc"], dtype=C128, device="cuda")
        for i in range(c["ngc"]):
            d = s["b1"][:, :, None] - s["b2"][:, None, :] - s["gc"][:, i][:, None, None] - lo[:, None, None]
            inside = np.all((d >= 0) & (d < dim[:, None, None]), axis=0)
            d = np.where(inside[None], d, 0)
            m = torch.from_numpy(np.where(inside, lut[tuple(d)], 0)).cuda()
            g[:, :, i] = s["phase"][i] * (s["geigq"] @ m @ s["dgeigqk"].T)
        zt = torch.cat(rows + [g], dim=2)
        return (zt @ s["m2e"].conj().T).conj().resolve_conj()
    if kind == "coulomb":
        lam, q = torch.linalg.eigh(s["v"].T.contiguous())
        out = (q * lam.sqrt().to(C128)[None, :]) @ q.conj().T
        return [lam.flip(0).cpu().numpy(), out.T.contiguous()]
    p = torch.from_numpy(_interp_values()).cuda()
    cut = np.cumsum([16 * 256, 256, 256 * 256, 256, 256, 1])
    w = [x.to(torch.bfloat16).double().requires_grad_(True) for x in torch.tensor_split(p, cut.tolist())[:6]]
    head = p[cut[-1]:].double().requires_grad_(True)

    def net(x, t):
        x = x.double()
        h = torch.relu(x @ w[0].view(16, 256) + w[1])
        h = torch.relu(h @ w[2].view(256, 256) + w[3])
        return h @ w[4] + w[5] + (head.view(128, 16)[t.long()] * x).sum(1)

    with torch.no_grad():
        y = net(s["x_inf"], s["t_inf"])
    e = net(s["x_trn"], s["t_trn"]) - s["y_trn"].double()
    wt = s["w_trn"].double()
    loss = (wt * e * e).sum() / wt.sum()
    grads = torch.autograd.grad(loss, w + [head])
    return [y, float(loss.detach()), torch.cat([x.reshape(-1) for x in grads]).cpu().numpy()]
