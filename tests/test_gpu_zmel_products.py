"""The two products of the muffin-tin part at the sizes where their blocks change: 16 target columns, 96
valence channels (the largest accepted), atoms of different sizes, core states split by the window."""
import numpy as np
import pytest

from oracle import zmel
from tests.conftest import rel_fro

pytestmark = pytest.mark.gpu


def _rc(rng, *shape):
    return np.asfortranarray(rng.standard_normal(shape) + 1j * rng.standard_normal(shape))


@pytest.mark.parametrize("ntp0", [1, 16, 17])
@pytest.mark.parametrize("nm1,nm2,nctot", [(1, 1, 0), (2, 5, 4), (1, 70, 4), (5, 37, 4)])
def test_muffin_tin_products(qsgw, nm1, nm2, nctot, ntp0):
    import torch
    rng = np.random.default_rng(nm2 + ntp0)
    atoms = [dict(nc=3, nv=96, ias=1, ics=0, ims=1, ncore=3), dict(nc=1, nv=1, ias=97, ics=3, ims=34, ncore=1)]
    ppb = [rng.standard_normal((99, 99, 33)), rng.standard_normal((2, 2, 1))]
    ph = np.exp(1j * rng.uniform(0, 6.28, 2))
    nbloch, ndima = 36, 97
    nmv = max(0, nm2 - max(nm1, nctot + 1) + 1)
    cphim, cphiq = _rc(rng, ndima, max(nmv, 1)), _rc(rng, ndima, ntp0)
    ref = zmel.zmel_mt(cphim, cphiq, ppb, atoms, nbloch, nm1, nm2, nctot, ntp0, ph)
    nm = nm2 - nm1 + 1
    zt = torch.zeros(nbloch * nm * ntp0, dtype=torch.complex128, device="cuda")
    dat = [dict(a, nlnm=p.shape[0], mdim=p.shape[2], phase=f,
                ppb_d=torch.from_numpy(p.reshape(-1, order="F").copy()).cuda()) for a, p, f in zip(atoms, ppb, ph)]
    qsgw.zmel_mt_d(zt, nbloch, nm1, nm2, nctot, ntp0, qsgw.to_device(cphim), ndima, qsgw.to_device(cphiq), ndima, dat)
    qsgw.synchronize()
    assert rel_fro(qsgw.from_device(zt, (nbloch, nm, ntp0)), ref) < 1e-13
    for conj in (False, True):                                # the conjugate comes from the same product
        m2e = _rc(rng, nbloch, 35)
        out = torch.zeros(35 * nm * ntp0, dtype=torch.complex128, device="cuda")
        qsgw.zmel_m2e_d(out, zt, nbloch, 35, nm, ntp0, qsgw.to_device(m2e), False, conj)
        qsgw.synchronize()
        assert rel_fro(qsgw.from_device(out, (35, nm, ntp0)), zmel.zmel_m2e(ref, m2e, False, conj)) < 1e-13


@pytest.mark.parametrize("nv,mdim,nm,ntp0", [(1, 1, 1, 65600),      # more targets than one batch of the grid takes
                                             (96, 1500, 2, 300)])   # 690 MB of first products: several slabs
def test_muffin_tin_target_slabs(qsgw, nv, mdim, nm, ntp0):
    import torch
    rng = np.random.default_rng(ntp0)
    atom = dict(nc=0, nv=nv, ias=1, ics=0, ims=1, ncore=0)
    ppb = rng.standard_normal((nv, nv, mdim))
    cphim, cphiq = _rc(rng, nv, nm), _rc(rng, nv, ntp0)
    t = np.tensordot(ppb, cphiq, axes=(0, 0))                 # (a, i, itp)
    ref = np.tensordot(cphim.conj(), t, axes=(0, 0)).transpose(1, 0, 2)
    zt = torch.zeros(mdim * nm * ntp0, dtype=torch.complex128, device="cuda")
    dat = [dict(atom, nlnm=nv, mdim=mdim, phase=1.0, ppb_d=torch.from_numpy(ppb.reshape(-1, order="F").copy()).cuda())]
    m, q = qsgw.to_device(cphim), qsgw.to_device(cphiq)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    qsgw.zmel_mt_d(zt, mdim, 1, nm, 0, ntp0, m, nv, q, nv, dat)
    qsgw.synchronize()
    assert free - torch.cuda.mem_get_info()[0] <= 300 << 20
    assert rel_fro(qsgw.from_device(zt, (mdim, nm, ntp0)), ref) < 1e-13
