"""The FP64 engine at the edges of its tiles (16 x 8 fragments, 64 x 64 tiles, K chunks of 16 in halves of
8), of its split over K and of its in-place accumulation, against numpy.

Bound: every element is a sum of k complex products, so its rounding error is at most (k + 4) eps sqrt(8)
times the sum of |a||b| (+ |c|); the Frobenius norms below bound that sum."""
import numpy as np
import pytest

from oracle import sxcf, x0
from ecalj_b200 import sched, synth
from tests.conftest import rel_fro

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


def _rc(rng, *shape):
    return np.asfortranarray(rng.standard_normal(shape) + 1j * rng.standard_normal(shape))


@pytest.mark.parametrize("opa,opb", [(0, 0), (0, 2), (2, 0), (1, 1)])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (16, 8, 8), (17, 9, 9), (48, 24, 16), (63, 65, 17), (65, 63, 31),
                                   (128, 64, 33), (33, 40, 1000)])
def test_zmm_edges(qsgw, m, n, k, opa, opb):
    rng = np.random.default_rng(m + 3 * n + 5 * k)
    a = _rc(rng, m, k) if opa == 0 else _rc(rng, k, m)
    b = _rc(rng, k, n) if opb == 0 else _rc(rng, n, k)
    c0 = _rc(rng, m, n)
    op = lambda x, o: x if o == 0 else (x.T if o == 1 else x.conj().T)
    bound = (k + 4) * EPS * np.sqrt(8) * (np.linalg.norm(a) * np.linalg.norm(b) + np.linalg.norm(c0))
    for alpha, beta in ((1.0, 0.0), (-1.0, 1.0), (1.0, 1.0), (1.0, 0.5)):     # +-1, 1: C starts the sums
        c = c0.copy(order="F")
        if beta == 0.0:
            c[:] = np.nan                                                    # must not be read
        qsgw.zmm(a, b, c, m, n, k, opa, opb, alpha, beta)
        ref = alpha * (op(a, opa) @ op(b, opb)) + beta * c0
        assert np.linalg.norm(c - ref) <= bound, (alpha, beta)


@pytest.mark.parametrize("npr", [15, 33, 64, 65, 130])
@pytest.mark.parametrize("ncoun", [1, 8, 9, 17, 600])
def test_x0gemm_bins_of_few_pairs(qsgw, npr, ncoun):
    """Hermitian bins whose pair counts straddle the K halves; every element of both triangles is checked."""
    rng = np.random.default_rng(npr + ncoun)
    nm, nq, nwhis = 5, 7, 3
    z = _rc(rng, npr + 2, nm, nq)
    itc, itpc = rng.integers(1, nm + 1, ncoun), rng.integers(1, nq + 1, ncoun)
    ini = rng.integers(1, nwhis + 1, ncoun)
    tabs = (itc, itpc, np.ones(ncoun, int), ini, ini, np.arange(1, ncoun + 1))
    w = rng.uniform(-1, 1, ncoun)
    r0 = _rc(rng, npr, npr, nwhis + 1)
    ref, got = r0.copy(order="F"), r0.copy(order="F")
    x0.x0gemm(ref, npr, 1, npr, nwhis, 1, 1, nm, z, 1, 1, ncoun, *tabs, w)
    qsgw.x0gemm(got, npr, 1, npr, nwhis, 1, 1, nm, z, 1, 1, ncoun, *tabs, w)
    bound = (ncoun + 4) * EPS * np.sqrt(8) * (np.linalg.norm(z) ** 2 * ncoun + np.linalg.norm(r0))
    assert np.linalg.norm(got - ref) <= bound


@pytest.mark.parametrize("n,nm,ntq", [(24, 5, 2), (64, 16, 4), (70, 33, 5)])
def test_sigma_segments_split_over_blocks(qsgw, n, nm, ntq):
    """Few column tiles: the segments of one tile are dealt to several blocks that add into the output."""
    t = synth.sigc_task(n, ntq, nm, 9, 30, seed=n, esmr=0.02, ef=0.05)
    rng = np.random.default_rng(n)
    w = _rc(rng, n, n, 10)
    wi = np.asfortranarray(w + w.conj().transpose(1, 0, 2))
    wr = _rc(rng, n, n, 30)
    nwxi, nwx, ntmax = sched.get_nwx(t["omega"], t["ekc"], t["freq_r"], t["ef"], t["esmr"])
    args = (1, nm, min(nm, ntmax), nwxi, nwx, ntq, wi, wr, t["omega"], t["ekc"], 0, t["ef"], t["esmr"], 1 / 8,
            t["ua"], t["x"], t["wx"], t["expa"], t["freq_r"])
    ref, got = (np.zeros((ntq, ntq), complex, order="F") for _ in range(2))
    sxcf.correlation_block(ref, t["zmel"], *args)
    qsgw.sxcf_correlation(got, t["zmel"], *args)
    assert rel_fro(got, ref) < 1e-11
