"""The Hilbert transform matrix formed on the GPU, element by element, against the host's: a histogram with
one unit entry per bin returns the matrix itself."""
import numpy as np
import pytest

from ecalj_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nwhis,niw,nw,ecut", [(1, 1, 0, 1e10), (2, 3, 1, 1e10), (37, 5, 36, 0.8), (96, 12, 60, 1e10),
                                               (64, 0, 10, 1e10), (20, 4, -1, 1e10)])
def test_transform_matrix_elements(qsgw, nwhis, niw, nw, ecut):
    import torch
    frhis = 0.02 * (np.exp(0.04 * np.arange(nwhis + 1)) - 1.0)
    fi = synth.imag_mesh(niw)["freq_i"] if niw else np.zeros(0)
    fr = None if nw < 0 else np.concatenate([[0.0], 0.5 * (frhis[:-1] + frhis[1:])])[:nw + 1]
    ref = qsgw.dpsion_matrix(frhis, fi, fr, ecut=ecut)
    unit = torch.eye(nwhis + 1, dtype=torch.complex128, device="cuda")
    zi, zr = qsgw.dpsion_chiq_d(unit.reshape(-1), nwhis + 1, 1, nwhis, frhis, fi, fr, ecut)
    qsgw.synchronize()
    got = np.concatenate([z.cpu().numpy().reshape(nwhis + 1, -1, order="F") for z in (zi, zr) if z is not None], axis=1)
    # both sides lose z log + (b - a) to cancellation: eps |z| / (bin width) of an element of order 1 / width
    width = np.diff(frhis).min()
    z = np.abs(np.concatenate([fi, [] if fr is None else fr]))
    bound = 64 * np.finfo(float).eps * (1.0 + z / width) / width
    assert np.all(np.abs(got - ref).max(axis=0) <= bound)
