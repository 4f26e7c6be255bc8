"""The Jacobi steps at odd sizes, at the edges of their 16-pair and 64-row blocks, and with a padded leading
dimension: residual, orthonormality and eigenvalues against LAPACK within 64 n eps of the matrix norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,pad", [(3, 0), (31, 2), (32, 0), (33, 0), (34, 1), (63, 0), (65, 3), (129, 0)])
def test_jacobi_block_edges(qsgw, n, pad):
    rng = np.random.default_rng(n)
    g = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    v = g @ g.conj().T * 10.0 ** rng.uniform(-3, 3)
    v = 0.5 * (v + v.conj().T)
    v[0, :] = v[:, 0] = 0.0                                   # a decoupled state: no rotation at all
    v[0, 0] = 1.0
    buf = np.full((n + pad, n), 7.0 + 0j, order="F")
    buf[:n] = v
    d = qsgw.to_device(buf)
    lam = qsgw.zhegv_d(d, n, lda=n + pad)
    z = qsgw.from_device(d, buf.shape)
    tol = 64 * n * np.finfo(float).eps
    norm = np.linalg.norm(v, 2)
    assert np.abs(lam - np.linalg.eigvalsh(v)[::-1]).max() <= tol * norm
    assert np.abs(v @ z[:n] - z[:n] * lam).max() <= tol * norm
    assert np.abs(z[:n].conj().T @ z[:n] - np.eye(n)).max() <= tol
    assert np.all(z[n:] == 7.0)


@pytest.mark.parametrize("n", [48, 130, 257])
def test_jacobi_equal_eigenvalues(qsgw, n):
    """Four distinct eigenvalues: rotations within an eigenspace are arbitrary, the spaces are not."""
    rng = np.random.default_rng(n)
    q, _ = np.linalg.qr(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)))
    lam = np.repeat([7.0, 5.0, 2.0, 1.0], (n + 3) // 4)[:n]
    v = (q * lam) @ q.conj().T
    v = np.asfortranarray(0.5 * (v + v.conj().T))
    d = qsgw.to_device(v)
    got = qsgw.zhegv_d(d, n)
    z = qsgw.from_device(d, v.shape)
    tol = 64 * n * np.finfo(float).eps
    assert np.abs(got - lam).max() <= tol * lam[0]
    assert np.abs((z * got) @ z.conj().T - v).max() <= tol * lam[0]
    assert np.abs(z.conj().T @ z - np.eye(n)).max() <= tol


def test_jacobi_equal_eigenvalues_of_the_largest_cell(qsgw):
    """n = 1500, two distinct eigenvalues: the most sweeps met (44 of the 60 allowed)."""
    import torch
    n = 1500
    g = torch.Generator(device="cuda").manual_seed(n)
    q, _ = torch.linalg.qr(torch.randn(n, n, dtype=torch.complex128, device="cuda", generator=g))
    lam = torch.repeat_interleave(torch.tensor([3.0, 1.0], dtype=torch.float64, device="cuda"), n // 2)
    v = (q * lam) @ q.conj().T
    v = 0.5 * (v + v.conj().T)
    d = v.T.contiguous().reshape(-1).clone()                 # column-major
    got = torch.from_numpy(qsgw.zhegv_d(d, n)).cuda()
    z = d.view(n, n).T
    tol = 64 * n * np.finfo(float).eps
    assert (got - lam).abs().max() <= tol * 3
    assert ((z * got) @ z.conj().T - v).abs().max() <= tol * 3
    assert (z.conj().T @ z - torch.eye(n, device="cuda")).abs().max() <= tol


@pytest.mark.parametrize("exp10", [-140, -155, -200, -300, 100])
def test_jacobi_small_and_large_entries(qsgw, exp10):
    """Rotations are chosen from squares of the entries: a small matrix is solved as its multiple of order one."""
    n = 40
    rng = np.random.default_rng(n)
    g = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    v = g + g.conj().T
    d = qsgw.to_device(np.asfortranarray(v * 10.0 ** exp10))
    lam = qsgw.zhegv_d(d, n) / 10.0 ** exp10
    z = qsgw.from_device(d, v.shape)
    tol = 64 * n * np.finfo(float).eps
    norm = np.linalg.norm(v, 2)
    assert np.abs(lam - np.linalg.eigvalsh(v)[::-1]).max() <= tol * norm
    assert np.abs(v @ z - z * lam).max() <= tol * norm


def test_jacobi_zero_and_non_finite(qsgw):
    d = qsgw.to_device(np.zeros((20, 20), complex, order="F"))
    assert np.array_equal(qsgw.zhegv_d(d, 20), np.zeros(20))
    for bad in (np.nan, np.inf):
        v = np.eye(20, dtype=complex, order="F") * 1e-200
        v[3, 3] = bad
        with pytest.raises(qsgw.QSGWError):
            qsgw.zhegv_d(qsgw.to_device(v), 20)
