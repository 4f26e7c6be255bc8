"""CUDA graph of a recorded call sequence: chi0 -> W -> Sigma_c recorded once
and replayed gives the eager results, reads device inputs at replay time, and
refuses to grow scratch while recording."""
import numpy as np
import pytest

from ecalj_b200 import synth
from oracle import sxcf
from tests.conftest import rel_fro

pytestmark = pytest.mark.gpu


def _problem(lib, torch):
    p = synth.chi0_problem(N=96, nk=4, nocc=3, nun=(10, 20), niw=6, seed=31)
    N, niw = p["N"], p["niw"]
    vsq, q = synth.coulomb(N, 32)
    t = synth.sigc_task(N, 6, 20, niw, 30, seed=33, esmr=0.02, ef=0.05)
    nt0p, nt0m = sxcf.nt0pm(t["ekc"], t["ef"], t["esmr"])
    nwxi, nwx, ntmax = sxcf.get_nwx(t["omega"], 6, nt0p, nt0m, 20, t["freq_r"], t["esmr"], t["ef"], t["ekc"], 0)
    freqs = np.concatenate([[0.0], p["freq_i"]])
    d = dict(p=p, t=t, N=N, niw=niw, vsq=vsq, freqs=freqs, nwxi=nwxi, nwx=nwx, ns2r=min(20, ntmax),
             z=lib.to_device(p["zcols"]), m2e=lib.to_device(q), zmel=lib.to_device(t["zmel"]),
             chi=torch.zeros(N * N * (niw + 1), dtype=torch.complex128, device="cuda"),
             zw=torch.zeros(N * N * (niw + 1), dtype=torch.complex128, device="cuda"),
             wr=torch.zeros(N * N * len(t["freq_r"]), dtype=torch.complex128, device="cuda"),
             zsec=torch.zeros(36, dtype=torch.complex128, device="cuda"))
    return d


def _step(lib, d):
    p, t, N, niw = d["p"], d["t"], d["N"], d["niw"]
    d["zsec"].zero_()
    lib.chi0_lorentz_d(d["chi"], N, niw + 1, d["freqs"], p["nk"], p["nocc"], p["nun"], p["eocc_h"], p["eun_h"], d["z"])
    lib.wvi_llw(d["chi"], 2, d["vsq"], d["m2e"], True, True, 2, zw=d["zw"], device=True, ngb=N, niw=niw + 1)
    d["wr"].view(-1, N * N)[:] = d["zw"][:N * N]          # real-axis W = W(0) on every record
    lib.sxcf_correlation(d["zsec"], d["zmel"], 1, 20, d["ns2r"], d["nwxi"], d["nwx"], 6, d["zw"], d["wr"],
                         t["omega"], t["ekc"], 0, t["ef"], t["esmr"], 1.0 / 8, t["ua"], t["x"], t["wx"], t["expa"],
                         t["freq_r"], nblochpmx=N, device=True, ngb=N, ntq=6)


@pytest.mark.parametrize("prec", ["fp64", "split"])
def test_graph_replay_matches_eager(qsgw, prec):
    import torch
    lib = qsgw
    lib.set_precision(lib.PREC_SPLIT_F16 if prec == "split" else lib.PREC_FP64)
    try:
        d = _problem(lib, torch)
        _step(lib, d)                                     # eager (also sizes every scratch buffer)
        lib.synchronize()
        ref = {k: d[k].clone() for k in ("chi", "zw", "zsec")}
        lib.graph_begin()
        _step(lib, d)
        lib.graph_end()
        for k in ("chi", "zw", "zsec"):
            d[k].fill_(7.0)                               # the replay must rewrite everything
        for _ in range(2):
            lib.graph_launch()
        lib.synchronize()
        tol = 1e-12 if prec == "fp64" else 1e-9
        for k in ("chi", "zw", "zsec"):
            assert rel_fro(d[k].cpu().numpy(), ref[k].cpu().numpy()) <= tol, k
        # device inputs are read at replay time: z -> 2 z gives chi0 -> 4 chi0
        d["z"].mul_(2.0)
        lib.graph_launch()
        lib.synchronize()
        assert rel_fro(d["chi"].cpu().numpy(), 4 * ref["chi"].cpu().numpy()) <= tol
        lib.graph_destroy()
    finally:
        lib.set_precision(lib.PREC_FP64)


def test_graph_refuses_scratch_growth(qsgw):
    import torch
    lib = qsgw
    # more pairs x frequencies than any test collected before this one (the full-size chi0
    # test is collected after it): the weight scratch must grow
    p = synth.chi0_problem(N=64, nk=64, nocc=8, nun=(100, 120), niw=12, seed=35)
    N, niw = p["N"], p["niw"]
    chi = torch.zeros(N * N * niw, dtype=torch.complex128, device="cuda")
    z = lib.to_device(p["zcols"])
    lib.graph_begin()
    with pytest.raises(lib.QSGWError) as e:
        lib.chi0_lorentz_d(chi, N, niw, p["freq_i"], p["nk"], p["nocc"], p["nun"], p["eocc_h"], p["eun_h"], z)
    assert e.value.code == -7 and "graph" in str(e.value)
    try:
        lib.graph_end()
    except lib.QSGWError:
        pass
    lib.graph_destroy()
    # eager use works again and sizes the buffers
    lib.chi0_lorentz_d(chi, N, niw, p["freq_i"], p["nk"], p["nocc"], p["nun"], p["eocc_h"], p["eun_h"], z)
    lib.synchronize()
    assert float(torch.linalg.vector_norm(chi)) > 0


def _replays_as_recorded(lib, call, out, spoil=lambda: None):
    """`call` recorded, its host tables spoilt and their memory reused: the replay still gives the eager result."""
    call()                                                # sizes the scratch
    lib.synchronize()
    ref = out.clone()
    lib.graph_begin()
    call()
    lib.graph_end()
    spoil()
    junk = [np.full(50000, 7) for _ in range(20)]
    out.zero_()
    lib.graph_launch()
    lib.synchronize()
    lib.graph_destroy()
    assert len(junk) == 20 and float(ref.abs().max()) > 0
    assert rel_fro(out.cpu().numpy(), ref.cpu().numpy()) <= 1e-13


def _rc(rng, *shape):
    return np.asfortranarray(rng.standard_normal(shape) + 1j * rng.standard_normal(shape))


def test_muffin_tin_elements_recorded_in_a_graph(qsgw):
    import torch
    rng = np.random.default_rng(3)
    nlnm, md, nm, ntp0 = 7, 5, 4, 3
    ppb = [torch.from_numpy(rng.standard_normal(nlnm * nlnm * md)).cuda() for _ in range(2)]
    atoms = [dict(nlnm=nlnm, nc=1, nv=6, ias=1 + 6 * i, ics=0, ims=1 + md * i, mdim=md, ncore=0, phase=1j ** i, ppb_d=p)
             for i, p in enumerate(ppb)]
    cphim, cphiq = qsgw.to_device(_rc(rng, 12, nm)), qsgw.to_device(_rc(rng, 12, ntp0))
    zt = torch.zeros(2 * md * nm * ntp0, dtype=torch.complex128, device="cuda")
    _replays_as_recorded(qsgw, lambda: qsgw.zmel_mt_d(zt, 2 * md, 1, nm, 0, ntp0, cphim, 12, cphiq, 12, atoms), zt)


def test_imaginary_axis_weights_recorded_in_a_graph(qsgw):
    import torch
    t = synth.sigc_task(8, 3, 10, 6, 30, seed=2, esmr=0.02, ef=0.05)
    tabs = [np.array(t[k]) for k in ("omega", "ekc", "x", "wx", "expa")]
    om, ek, x, wx, ex = tabs
    out = torch.zeros(7 * 10 * 3, dtype=torch.float64, device="cuda")

    def spoil():
        for a in tabs:
            a[:] = 0.5

    _replays_as_recorded(qsgw, lambda: qsgw.sxcf_wgtim_d(out, 6, 1, 10, 3, 0, om, ek, t["esmr"], 1 / 8, t["ua"], x, wx,
                                                         ex), out, spoil)


def test_exchange_recorded_in_a_graph(qsgw):
    import torch
    rng = np.random.default_rng(5)
    ngb, nm, ntq = 20, 9, 4
    z = qsgw.to_device(_rc(rng, ngb, nm, ntq))
    vcoud, ekc = 10 ** rng.uniform(-2, 3, ngb), np.sort(rng.uniform(-1, 1, nm))
    zsec = torch.zeros(ntq * ntq, dtype=torch.complex128, device="cuda")

    def call():
        zsec.zero_()
        qsgw.sxcf_exchange_d(zsec, ntq, z, ngb, 1, nm, ntq, vcoud, ekc, 0, 0.1, 0.02, 0.125)

    def spoil():
        vcoud[:] = 1.0

    _replays_as_recorded(qsgw, call, zsec, spoil)


def test_scratch_outgrown_after_recording_is_kept(qsgw):
    """Later calls of a larger shape take new scratch; the graph goes on with the one it was recorded with."""
    import torch
    rng = np.random.default_rng(9)

    def problem(ngb, nm, ntq):
        z = qsgw.to_device(_rc(rng, ngb, nm, ntq))
        vcoud, ekc = 10 ** rng.uniform(-2, 3, ngb), np.sort(rng.uniform(-1, 1, nm))
        zsec = torch.zeros(ntq * ntq, dtype=torch.complex128, device="cuda")
        x = torch.from_numpy(rng.uniform(-1, 1, (ngb, 16)).astype(np.float32).ravel()).cuda()
        buf = torch.zeros(ngb * 16 + 4, dtype=torch.float32, device="cuda")
        buf[1:1 + ngb * 16] = x                               # not 16-byte aligned: the layer-by-layer route
        y, tix = torch.zeros(ngb, device="cuda"), torch.zeros(ngb, dtype=torch.int32, device="cuda")

        def call():
            zsec.zero_()
            qsgw.sxcf_exchange_d(zsec, ntq, z, ngb, 1, nm, ntq, vcoud, ekc, 0, 0.1, 0.02, 0.125)
            qsgw.wsurr_forward_d(buf[1:1 + ngb * 16], tix, y, ngb)
        return call, zsec, y

    qsgw.wsurr_init(3)
    small, zs, ys = problem(20, 9, 4)
    large, zl, yl = problem(70001, 2, 3)
    small()
    qsgw.synchronize()
    ref = zs.clone(), ys.clone()
    qsgw.graph_begin()
    small()
    qsgw.graph_end()
    for _ in range(2):
        large()
    fill = [torch.full((1 << 22,), 3.0, device="cuda") for _ in range(8)]      # whatever reuses released memory
    out = zl.clone(), yl.clone()
    ys.zero_()
    qsgw.graph_launch()
    large()
    qsgw.synchronize()
    qsgw.graph_destroy()
    assert len(fill) == 8
    for a, b in zip((zs, ys, zl, yl), ref + out):
        assert rel_fro(a.cpu().numpy(), b.cpu().numpy()) <= 1e-12 and float(b.abs().max()) > 0
