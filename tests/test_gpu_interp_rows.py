"""The fused inference kernel at the edges of its 16-row warps and 128-row blocks, rows with linear-only and
invalid heads, rows that are not 16-byte aligned (the layer-by-layer path), and the row sums of the gradient
at the edges of their 64-row blocks, against the float64 statement of the network."""
import numpy as np
import pytest

from oracle import mlp

pytestmark = pytest.mark.gpu


def _net(qsgw, seed):
    rng = np.random.default_rng(seed)
    p = (rng.standard_normal(mlp.NPARAM) * 0.06).astype(np.float32)
    qsgw.wsurr_init(1)
    qsgw.wsurr_params(p)
    return p, rng


@pytest.mark.parametrize("n", [1, 15, 16, 17, 127, 129, 1000])
@pytest.mark.parametrize("shift", [0, 1])
def test_inference_rows(qsgw, n, shift):
    import torch
    p, rng = _net(qsgw, n)
    x = rng.uniform(-1, 1, (n, 16)).astype(np.float32)
    tix = rng.integers(0, mlp.NTMAX, n).astype(np.int32)
    buf = torch.zeros(n * 16 + 4, dtype=torch.float32, device="cuda")
    xd = buf[shift:shift + n * 16]
    xd.copy_(torch.from_numpy(x.ravel()))
    y = torch.full((n,), np.nan, dtype=torch.float32, device="cuda")
    qsgw.wsurr_forward_d(xd, torch.from_numpy(tix).cuda(), y, n)
    qsgw.synchronize()
    ref, _ = mlp.forward(p, x, tix)
    # FP32 sums of 256 terms of order 0.1, and h1 values that round to the other BF16 neighbour (2^-8 of one
    # unit's share, 0.06 |h1|) where the sums before them differ in the last FP32 digit
    assert np.abs(y.cpu().numpy() - ref).max() <= 2e-3 * max(1.0, np.abs(ref).max())
    assert np.linalg.norm(y.cpu().numpy() - ref) <= 1e-4 * max(1.0, np.linalg.norm(ref))


def test_layer_one_against_64_bits(qsgw):
    """W2 the identity and W3 one unit: y is that unit's h1.  It is the BF16 rounding of the 64-bit sum but where the
    sum lies within its own error of a rounding boundary: 17 FP32 roundings of sums of order 0.2 (3e-7 at most)
    against BF16 steps of 5e-4 to 1e-3, one value in a thousand at most."""
    import torch
    p, rng = _net(qsgw, 11)
    p[mlp.OFF_W2:mlp.OFF_B2] = np.eye(mlp.NH, dtype=np.float32).ravel()
    p[mlp.OFF_B2:mlp.OFF_W3] = 0.0
    p[mlp.OFF_B3:] = 0.0
    bf16 = lambda v: torch.from_numpy(np.asarray(v)).to(torch.bfloat16).double().numpy()
    n, units, off = 4096, (0, 7, 8, 15, 16, 100, 255), 0
    x = rng.uniform(-1, 1, (n, 16)).astype(np.float32)
    xd, td = torch.from_numpy(x.ravel()).cuda(), torch.zeros(n, dtype=torch.int32, device="cuda")
    y = torch.zeros(n, dtype=torch.float32, device="cuda")
    w1, b1 = bf16(p[:mlp.OFF_B1]).reshape(16, mlp.NH), bf16(p[mlp.OFF_B1:mlp.OFF_W2])
    for j in units:
        p[mlp.OFF_W3:mlp.OFF_B3] = 0.0
        p[mlp.OFF_W3 + j] = 1.0
        qsgw.wsurr_params(p)
        qsgw.wsurr_forward_d(xd, td, y, n)
        qsgw.synchronize()
        got, ref = y.cpu().numpy().astype(float), bf16(np.maximum(x.astype(float) @ w1[:, j] + b1[j], 0.0))
        off += int((got != ref).sum())
        assert np.all(np.abs(got - ref) <= 2.0 ** -7 * ref + 1e-6)
    assert off <= 1e-3 * n * len(units)


def test_inference_infinite_and_nan_inputs_stay_in_their_rows(qsgw):
    import torch
    p, rng = _net(qsgw, 5)
    x = rng.uniform(-1, 1, (32, 16)).astype(np.float32)
    tix = np.zeros(32, np.int32)
    good, _ = mlp.forward(p, x, tix)
    x[3, 2], x[20, 7] = np.inf, np.nan
    xd = torch.from_numpy(x).cuda()
    y = torch.zeros(32, dtype=torch.float32, device="cuda")
    qsgw.wsurr_forward_d(xd, torch.from_numpy(tix).cuda(), y, 32)
    qsgw.synchronize()
    got = y.cpu().numpy()
    keep = np.setdiff1d(np.arange(32), [3, 20])
    assert np.abs(got[keep] - good[keep]).max() <= 2e-3
    assert not np.isfinite(got[3]) and np.isnan(got[20])      # both reach the linear head


@pytest.mark.parametrize("batch", [1, 63, 64, 65, 500])
def test_gradient_row_blocks(qsgw, batch):
    import torch
    p, rng = _net(qsgw, batch)
    x = rng.uniform(-1, 1, (batch, 16)).astype(np.float32)
    tix = rng.integers(0, mlp.NTMAX, batch).astype(np.int32)
    ys = rng.standard_normal(batch).astype(np.float32)
    w = rng.uniform(0.1, 1.0, batch).astype(np.float32)
    dev = [torch.from_numpy(a).cuda() for a in (x, tix, ys, w)]
    loss, grad = qsgw.wsurr_grad_d(dev[0], dev[1], dev[2], batch, dev[3])
    ref_l, ref = mlp.loss_and_grad(p, x, tix, ys, w)
    assert abs(loss - ref_l) <= 1e-4 * ref_l
    for a, b in ((mlp.OFF_W1, mlp.OFF_B1), (mlp.OFF_B1, mlp.OFF_W2), (mlp.OFF_B2, mlp.OFF_W3)):
        # BF16 neighbours of h1 and g2 (2^-9 of a term, random signs)
        assert np.linalg.norm(grad[a:b] - ref[a:b]) <= 2e-3 * np.linalg.norm(ref[a:b])


def test_loss_does_not_depend_on_the_order_of_its_sums(qsgw):
    """Eight calls on the same rows, and on the rows shuffled: one rounding of FP32 apart at most."""
    import torch
    p, rng = _net(qsgw, 12)
    n = 8191
    x = rng.uniform(-1, 1, (n, 16)).astype(np.float32)
    tix = rng.integers(0, mlp.NTMAX, n).astype(np.int32)
    ys, w = rng.standard_normal(n).astype(np.float32), rng.uniform(0.1, 1.1, n).astype(np.float32)
    loss = []
    for i in range(8):
        o = rng.permutation(n) if i % 2 else np.arange(n)
        dev = [torch.from_numpy(np.ascontiguousarray(a[o])).cuda() for a in (x, tix, ys, w)]
        loss.append(qsgw.wsurr_grad_d(dev[0], dev[1], dev[2], n, dev[3])[0])
    assert max(loss) - min(loss) <= 2.0 ** -23 * max(loss)
