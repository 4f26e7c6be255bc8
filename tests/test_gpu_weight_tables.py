"""Weight tables formed on the device or with shortcuts on the host: pole weights of levels around the points where
the smeared window saturates, core levels, and k-points without pairs."""
import numpy as np
import pytest

from ecalj_b200 import synth
from oracle import sxcf
from tests.conftest import rel_fro

pytestmark = pytest.mark.gpu


def _rc(rng, *shape):
    return np.asfortranarray(rng.standard_normal(shape) + 1j * rng.standard_normal(shape))


@pytest.mark.parametrize("nctot", [0, 3])
def test_pole_weights_around_the_window_ends(qsgw, nctot):
    n, esmr, ef = 12, 0.02, 0.05
    far = 6.5 * np.sqrt(2.0) * esmr
    omega = np.array([-0.9, -0.3, ef, 0.4, 1.0])
    # levels at, just inside and just outside the saturation points of every window end
    ends = np.concatenate([omega, [ef]])
    ekc = np.sort(np.concatenate([ends + s * far * f for s in (-1, 1) for f in (0.5, 0.999, 1.001)] + [ends]))
    nm, ntq = len(ekc), len(omega)
    rng = np.random.default_rng(nctot)
    z = _rc(rng, n, nm, ntq)
    mesh = synth.imag_mesh(4)
    fr = synth.freq_r_mesh(40)
    wi, wr = _rc(rng, n, n, 5), _rc(rng, n, n, 40)
    args = (1, nm, nm, 0, 39, ntq, wi, wr, omega, ekc, nctot, ef, esmr, 1 / 8, mesh["ua"], mesh["x"], mesh["wx"],
            mesh["expa"], fr)
    ref, got = (np.zeros((ntq, ntq), complex, order="F") for _ in range(2))
    sxcf.correlation_block(ref, z, *args)
    qsgw.sxcf_correlation(got, z, *args)
    assert rel_fro(got, ref) < 1e-12


def test_k_points_without_pairs(qsgw):
    import torch
    n, niw = 9, 3
    nocc, nun = np.array([0, 2, 3, 0, 1, 2]), np.array([4, 0, 5, 0, 3, 2])
    rng = np.random.default_rng(3)
    eo, eu = rng.uniform(-0.4, 0.0, nocc.sum()), rng.uniform(-0.1, 2.0, nun.sum())      # some negative energies
    npair = int((nocc * nun).sum())
    z = _rc(rng, n, npair)
    fi = synth.imag_mesh(niw)["freq_i"]
    chi = torch.zeros(n * n * niw, dtype=torch.complex128, device="cuda")
    qsgw.chi0_lorentz_d(chi, n, niw, fi, 6, nocc, nun, eo, eu, qsgw.to_device(z))
    qsgw.synchronize()
    de, a, b = [], 0, 0
    for k in range(6):
        de.append((eu[b:b + nun[k], None] - eo[None, a:a + nocc[k]]).ravel())
        a, b = a + nocc[k], b + nun[k]
    de = np.concatenate(de)
    ref = np.stack([np.conj(z) @ np.diag(-2 * de / (de * de + w * w) / 6) @ z.T for w in fi], axis=2)
    assert rel_fro(qsgw.from_device(chi, (n, n, niw)), ref) < 1e-13
