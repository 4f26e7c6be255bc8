"""The pivoted inverse at the sizes where its panel kernel changes (one row a thread in registers up to 384
rows) and at ragged last panels; zero diagonals force row exchanges.  Bound: for a matrix of condition c the
inverse's relative error stays below 32 n eps c (a growth factor of a few and n rank-one steps)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 33, 64, 95, 384, 385])
def test_pivoted_inverse_panel_edges(qsgw, n):
    rng = np.random.default_rng(n)
    a = np.zeros((n, n, 3), complex, order="F")
    for b in range(3):
        a[:, :, b] = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
        if n > 1:
            a[np.arange(n), np.arange(n), b] = 0.0
    d = qsgw.to_device(a)
    qsgw.zminv_batched_d(d, n, n, 3)
    qsgw.synchronize()
    got = qsgw.from_device(d, a.shape)
    for b in range(3):
        ref = np.linalg.inv(a[:, :, b])
        cond = np.linalg.norm(a[:, :, b], 2) * np.linalg.norm(ref, 2)
        assert np.linalg.norm(got[:, :, b] - ref) <= 32 * n * np.finfo(float).eps * cond * np.linalg.norm(ref)


@pytest.mark.parametrize("n", [40, 400])
def test_singular_matrix_is_reported(qsgw, n):
    a = np.asfortranarray(np.ones((n, n, 2), complex))
    d = qsgw.to_device(a)
    qsgw.zminv_batched_d(d, n, n, 2)
    with pytest.raises(qsgw.QSGWError) as e:
        qsgw.synchronize()
    assert e.value.code == -5
