"""The int8 kernels at the edges of their tiles and splits, against the CPU emulation of the same digits and kept
slice pairs.

Bounds: the integer products are exact, so kernel and emulation differ by the FP64 rounding of the scaled sums: some
eps of the terms that are added, whatever the slice count."""
import numpy as np
import pytest

from ecalj_b200 import sched, synth
from oracle import sxcf
from tests import ozaki_emul

pytestmark = pytest.mark.gpu


def _rc(rng, *shape):
    return np.asfortranarray(rng.standard_normal(shape) + 1j * rng.standard_normal(shape))


@pytest.fixture
def i8(qsgw):
    yield lambda ns: qsgw.set_precision(qsgw.PREC_SPLIT_I8, ns)
    qsgw.set_precision(qsgw.PREC_FP64, 1)


# largest element over rms of a normal sample of these sizes: under 5
PEAK = 5.0


@pytest.mark.parametrize("ns", [2, 3, 4])
@pytest.mark.parametrize("n", [1, 63, 64, 65, 127, 128, 129, 192, 193])
def test_chi0_hermitian_tiles(qsgw, i8, n, ns):
    """Diagonal tiles half a tile wide, their mirror, one and several K parts."""
    import torch
    for nun in (3, 40):
        p = synth.chi0_problem(N=n, nk=3, nocc=2, nun=(nun, nun + 2), niw=3, seed=n + nun)
        oo, uo = (np.concatenate([[0], np.cumsum(p[k])]) for k in ("nocc", "nun"))
        de = np.concatenate([(p["eun_h"][uo[k]:uo[k + 1]][None, :] - p["eocc_h"][oo[k]:oo[k + 1]][:, None])
                             .reshape(-1, order="F") for k in range(3)])
        w = -2.0 * de[None, :] / (de[None, :] ** 2 + p["freq_i"][:, None] ** 2) / 3
        emu = ozaki_emul.chi0_dense(p["zcols"], w, ns)
        i8(ns)
        chi = torch.zeros(n * n * 3, dtype=torch.complex128, device="cuda")
        qsgw.chi0_lorentz_d(chi, n, 3, p["freq_i"], 3, p["nocc"], p["nun"], p["eocc_h"], p["eun_h"],
                            qsgw.to_device(p["zcols"]))
        qsgw.synchronize()
        got = qsgw.from_device(chi, (n, n, 3))
        for iw in range(3):
            assert np.linalg.norm(got[:, :, iw] - emu[:, :, iw]) <= 1e-12 * np.linalg.norm(emu[:, :, iw])
            assert np.array_equal(got[:, :, iw], got[:, :, iw].conj().T)


@pytest.mark.parametrize("ncoun", [60, 640, 1500, 3000])      # FP64 up to 300 pairs a bin, int8 at 600
@pytest.mark.parametrize("npr,ipr_col,npr_col", [(130, 1, 130), (70, 3, 129)])
def test_x0gemm_bins_add_to_what_is_there(qsgw, i8, npr, ipr_col, npr_col, ncoun):
    rng = np.random.default_rng(npr)
    nbb, nm, nq, nwhis = 140, 4, 6, 5
    z = _rc(rng, nbb, nm, nq)
    tabs = (rng.integers(1, nm + 1, ncoun), rng.integers(1, nq + 1, ncoun), np.ones(ncoun, int),
            *(2 * [rng.integers(1, nwhis + 1, ncoun)]), np.arange(1, ncoun + 1))
    w = rng.uniform(-1, 1, ncoun)
    r0 = _rc(rng, npr, npr_col, nwhis + 1)
    out = []
    for ns in (0, 4):
        if ns:
            i8(ns)
        r = r0.copy(order="F")
        qsgw.x0gemm(r, npr, ipr_col, npr_col, nwhis, 1, 1, nm, z, 1, 1, ncoun, *tabs, w)
        out.append(r)
    inc = np.linalg.norm(out[0] - r0)
    assert np.linalg.norm(out[1] - out[0]) <= 6 * 2.0 * PEAK * np.sqrt(80.0) * 2.0 ** -28 * inc + 1e-14 * np.linalg.norm(r0)


def _bins(rng, cnts, nm, nq):
    """Pair tables of bins with the given pair counts, in mixed order; weights of both signs."""
    bin_ = rng.permutation(np.repeat(np.arange(1, len(cnts) + 1), cnts))
    n = len(bin_)
    return n, (rng.integers(1, nm + 1, n), rng.integers(1, nq + 1, n), np.ones(n, int), bin_, bin_,
               np.arange(1, n + 1)), rng.uniform(-1, 1, n)


@pytest.mark.parametrize("cnts,fp64,int8", [([128] * 5, 1, 0),             # short bins
                                            ([129] * 5, 1, 0),             # longer ones that do not pay
                                            ([10] * 40 + [513], 1, 1),     # one long bin among short ones
                                            ([600, 700, 513], 0, 1)])
def test_x0gemm_route_by_bins(qsgw, i8, cnts, fp64, int8):
    """In the int8 mode each bin runs where it is faster; every bin is added once."""
    import torch
    rng = np.random.default_rng(len(cnts))
    n, nm, nq = 70, 4, 6
    z = _rc(rng, n, nm, nq)
    ncoun, tabs, w = _bins(rng, cnts, nm, nq)
    r0 = _rc(rng, n, n, len(cnts) + 1)
    out = []
    for ns in (0, 4):
        if ns:
            i8(ns)
        r = qsgw.to_device(r0)
        qsgw.profile(True)
        qsgw.x0gemm(r, n, 1, n, len(cnts), 1, 1, nm, qsgw.to_device(z), 1, 1, ncoun, *tabs, w, zmel_shape=(n, nm, nq),
                    device=True)
        qsgw.synchronize()
        launches = [qsgw.profile_get(t)[1] for t in ("chi0_dmma", "chi0_tc")]
        qsgw.profile(False)
        out.append(qsgw.from_device(r, r0.shape))
    assert launches == [fp64, 2 * int8]                        # one int8 launch per sign of the weights
    for b, c in enumerate(cnts, 1):
        inc = np.linalg.norm(out[0][:, :, b] - r0[:, :, b])
        tol = 1e-13 if c <= 128 or not int8 else 6 * 2.0 * PEAK * np.sqrt(80.0) * 2.0 ** -28
        assert np.linalg.norm(out[1][:, :, b] - out[0][:, :, b]) <= tol * inc + 1e-14 * np.linalg.norm(r0[:, :, b])


@pytest.mark.parametrize("ns", [2, 3, 4])
@pytest.mark.parametrize("npr,ipr_col,npr_col", [(130, 1, 130), (70, 3, 129)])
def test_x0gemm_chunk_remainders(qsgw, i8, npr, ipr_col, npr_col, ns):
    """Pair counts at the edges of the 128-, 64- and 32-pair pieces of a chunk, columns gathered from a list."""
    rng = np.random.default_rng(ns)
    cnts = [640, 641, 672, 673, 704, 705, 767]
    nbb, nm, nq = 140, 5, 60
    z = _rc(rng, nbb, nm, nq)
    ncoun, tabs, w = _bins(rng, cnts, nm, nq)
    r0 = _rc(rng, npr, npr_col, len(cnts) + 1)
    got = r0.copy(order="F")
    i8(ns)
    qsgw.x0gemm(got, npr, ipr_col, npr_col, len(cnts), 1, 1, nm, z, 1, 1, ncoun, *tabs, w)
    zf = z.reshape(nbb, -1, order="F")
    zmax = np.maximum(np.abs(zf.real), np.abs(zf.imag)).max(axis=1)
    for b in range(1, len(cnts) + 1):
        sel = tabs[3] == b
        col = (tabs[0] - 1 + nm * (tabs[1] - 1))[sel]
        emu = ozaki_emul.chi0_dense(zf[:, col], w[sel][None, :], ns, zmax)[:npr, ipr_col - 1:ipr_col - 1 + npr_col, 0]
        err = np.linalg.norm(got[:, :, b] - r0[:, :, b] - emu)
        assert err <= 1e-12 * np.linalg.norm(emu) + 1e-15 * np.linalg.norm(r0[:, :, b])


@pytest.mark.parametrize("ncoun", [60, 3000])                # the FP64 engine's route and the int8 one
def test_x0gemm_recorded_in_a_graph(qsgw, i8, ncoun):
    """A recorded call replays with its own copy of the pair tables."""
    import torch
    rng = np.random.default_rng(ncoun)
    n, nm, nq, nwhis = 40, 4, 6, 5
    z = qsgw.to_device(_rc(rng, n, nm, nq))
    tabs = [rng.integers(1, nm + 1, ncoun), rng.integers(1, nq + 1, ncoun), np.ones(ncoun, int),
            *(2 * [rng.integers(1, nwhis + 1, ncoun)]), np.arange(1, ncoun + 1)]
    w = rng.uniform(0.1, 1, ncoun)
    r = torch.zeros(n * n * (nwhis + 1), dtype=torch.complex128, device="cuda")
    i8(4)
    call = lambda: qsgw.x0gemm(r, n, 1, n, nwhis, 1, 1, nm, z, 1, 1, ncoun, *tabs, w, zmel_shape=(n, nm, nq),
                               device=True)
    call()
    qsgw.synchronize()
    once = r.clone()
    qsgw.graph_begin()
    call()
    qsgw.graph_end()
    w[:] = 0.0
    junk = [np.full(200000, 7) for _ in range(20)]             # whatever reuses the host tables' memory
    r.zero_()
    for _ in range(2):
        qsgw.graph_launch()
    qsgw.synchronize()
    qsgw.graph_destroy()
    assert len(junk) == 20
    assert torch.linalg.vector_norm(r - 2 * once) <= 1e-12 * torch.linalg.vector_norm(once)


def _sigma(qsgw, t, wi, wr, n, nm, ntq, keepwv=False):
    nwxi, nwx, ntmax = sched.get_nwx(t["omega"], t["ekc"], t["freq_r"], t["ef"], t["esmr"])
    if keepwv:
        pack = lambda w: np.asfortranarray(np.stack([np.concatenate([w[:j + 1, j, k] for j in range(n)])
                                                     for k in range(w.shape[2])], axis=1))
        wi, wr = pack(wi), pack(wr)
    zs = np.zeros((ntq, ntq), complex, order="F")
    qsgw.sxcf_correlation(zs, t["zmel"], 1, nm, min(nm, ntmax), nwxi, nwx, ntq, wi, wr, t["omega"], t["ekc"], 0, t["ef"],
                          t["esmr"], 1 / 8, t["ua"], t["x"], t["wx"], t["expa"], t["freq_r"], keepwv=keepwv)
    return zs


@pytest.mark.parametrize("ns", [2, 3, 4])
@pytest.mark.parametrize("n,nm,ntq", [(1, 3, 2), (31, 5, 2), (32, 40, 3), (33, 40, 4), (64, 60, 5), (65, 9, 2),
                                      (96, 70, 2), (97, 33, 6)])
def test_sigma_segment_splits_and_chunks(qsgw, i8, n, nm, ntq, ns):
    """K extents of one, one and a half and two chunks; few tiles (segments split over CTAs); the paired last row tile
    alone (n <= 32), beside full ones (65, 96) and absent (64)."""
    t = synth.sigc_task(n, ntq, nm, 11, 30, seed=n, esmr=0.02, ef=0.05)
    rng = np.random.default_rng(n)
    w = _rc(rng, n, n, 12)
    wi, wr = np.asfortranarray(w + w.conj().transpose(1, 0, 2)), _rc(rng, n, n, 30)
    i8(ns)
    got = _sigma(qsgw, t, wi, wr, n, nm, ntq)
    nwxi, nwx, ntmax = sched.get_nwx(t["omega"], t["ekc"], t["freq_r"], t["ef"], t["esmr"])
    emu = np.zeros((ntq, ntq), complex, order="F")
    ozaki_emul.correlation_block(emu, t["zmel"], 1, nm, min(nm, ntmax), nwxi, nwx, ntq, wi, wr, t["omega"], t["ekc"], 0,
                                 t["ef"], t["esmr"], 1 / 8, t["ua"], t["x"], t["wx"], t["expa"], t["freq_r"], ns=ns)
    # Sigma adds nm n terms of czmelwc^H zmel; its elements cancel, so the scale is that of the unsigned sum
    wg = sxcf.wgtim(t["omega"], t["ekc"], 0, 1, nm, ntq, t["esmr"], 1 / 8, t["ua"], t["x"], t["wx"], t["expa"])
    scale = np.abs(wg).sum(0).max() * np.linalg.norm(t["zmel"]) ** 2 * max(np.linalg.norm(x, 2) for x in
                                                                          wi.transpose(2, 0, 1))
    assert np.linalg.norm(got - emu) <= 1e-14 * scale


@pytest.mark.parametrize("n", [1, 31, 32, 33, 65])
def test_packed_w_equals_full_w(qsgw, n):
    """Packed upper triangles are unpacked to the matrices they came from (Hermitian, real diagonal)."""
    t = synth.sigc_task(n, 3, 12, 5, 30, seed=n, esmr=0.02, ef=0.05)
    rng = np.random.default_rng(n)
    herm = lambda k: np.asfortranarray((lambda w: w + w.conj().transpose(1, 0, 2))(_rc(rng, n, n, k)))
    wi, wr = herm(6), herm(30)
    full = _sigma(qsgw, t, wi, wr, n, 12, 3)
    packed = _sigma(qsgw, t, wi, wr, n, 12, 3, keepwv=True)
    assert np.linalg.norm(full - packed) <= 1e-13 * np.linalg.norm(full)
