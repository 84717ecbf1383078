"""The pair sums of mse_adc and nll_loss at the edges of their tiles (64 rows,
32 columns, 1024 columns per upper range entry), with one and several column
slices, against the float64 oracle."""

import numpy as np
import pytest

from larndsim_gb300 import consts, losses
from oracle import losses_np as L

# float32 sums of at most ~2000 positive terms carry about 2000 * 2^-25 = 6e-5
# in the worst case and its square root typically; the losses' tolerances here
LOSS_RTOL, GRAD_RTOL = 1e-5, 1e-4

PARAMS = consts.Params()


def _hits(rng, n, n_events, spread):
    ev = np.sort(rng.integers(0, n_events, n)).astype(np.int32)
    xyz = rng.uniform(0, spread, (3, n)).astype(np.float32)
    return [rng.uniform(1, 30, n).astype(np.float32), *xyz, np.zeros(n, np.float32), np.ones(n, np.float32), ev]


def _run(fn, a, b):
    import torch
    dev = [torch.from_numpy(v).cuda() for v in a]
    dev[0].requires_grad_(True)
    dev[3].requires_grad_(True)
    loss, _ = fn(PARAMS, *dev, *[torch.from_numpy(v).cuda() for v in b])
    loss.backward()
    return float(loss.detach()), dev[0].grad.cpu().numpy(), dev[3].grad.cpu().numpy()


def _close(got, want):
    assert np.abs(got - want).max() <= GRAD_RTOL * np.abs(want).max()


@pytest.mark.gpu
@pytest.mark.parametrize("n,m,n_events,spread", [
    (1, 1, 1, 2.0), (31, 33, 1, 4.0), (32, 64, 1, 30.0), (63, 65, 2, 30.0), (64, 32, 3, 30.0), (65, 31, 1, 60.0),
    (127, 129, 4, 8.0), (1023, 1025, 2, 30.0), (1025, 700, 7, 60.0), (2049, 2047, 40, 30.0)])
def test_mse_adc_tile_edges(cuda, n, m, n_events, spread):
    rng = np.random.default_rng(n * 10007 + m)
    a, b = _hits(rng, n, n_events, spread), _hits(rng, m, n_events, spread)
    loss, gq, gz = _run(losses.mse_adc, a, b)
    want = L.mse_adc(a[0], a[1], a[2], a[3], a[5], a[6], b[0], b[1], b[2], b[3], b[5], b[6])[0]
    assert abs(loss - want) <= LOSS_RTOL * max(abs(want), 1e-3)
    wq, wz = L.mse_adc_grad(a[0], a[1], a[2], a[3], a[6], b[0], b[1], b[2], b[3], b[6])[:2]
    _close(gq, wq)
    if np.abs(wz).max() > 1e-8:      # a single pair of hits far apart has no z gradient to speak of
        _close(gz, wz)


def _nll64(a, b):
    """nll_loss and its gradients in Q and z, per event in float64."""
    x9 = lambda h: (h[1] + h[6].astype(np.float32) * np.float32(1e9)).astype(np.float64)   # noqa: E731
    A = np.stack([x9(a), a[2], a[3], a[0] / np.float32(10)], 1).astype(np.float64)
    B = np.stack([x9(b), b[2], b[3], b[0] / np.float32(10)], 1).astype(np.float64)
    d = B[:, None] - A[None]
    K = np.exp(-0.5 * (d ** 2).sum(2)) * (b[6][:, None] == a[6][None])
    lam = K.sum(1) + 1e-10
    c = 1 / lam
    return (a[0].size - np.log(lam).sum(), (K * -d[:, :, 3] * c[:, None]).sum(0) / 10,
            (K * -d[:, :, 2] * c[:, None]).sum(0))


@pytest.mark.gpu
@pytest.mark.parametrize("n,m,n_events,spread", [(1, 1, 1, 2.0), (33, 31, 1, 6.0), (64, 65, 2, 8.0),
                                                (700, 1025, 3, 30.0)])
def test_nll_tile_edges(cuda, n, m, n_events, spread):
    rng = np.random.default_rng(n * 10007 + m)
    a, b = _hits(rng, n, n_events, spread), _hits(rng, m, n_events, spread)
    loss, gq, gz = _run(losses.nll_loss, a, b)
    want, wq, wz = _nll64(a, b)
    assert abs(loss - want) <= LOSS_RTOL * max(abs(want), 1.0)
    _close(gq, wq)
    _close(gz, wz)


@pytest.mark.gpu
def test_mse_adc_one_slice(cuda):
    """Enough rows that no tile's columns are sliced: copies of one event, so
    every sum is the single event's (110 events of 1000 hits: 110000 rows,
    5157 row tiles over the three sums)."""
    rng = np.random.default_rng(3)
    copies, n = 110, 1000
    a1, b1 = _hits(rng, n, 1, 30.0), _hits(rng, n, 1, 30.0)
    for h in (a1, b1):       # x on a grid that x + event * 1e5 keeps exactly
        h[1] = np.round(h[1]).astype(np.float32)
    many = lambda h: [np.tile(v, copies) for v in h[:6]] + [np.repeat(np.arange(copies, dtype=np.int32), n)]   # noqa: E731
    loss, gq, gz = _run(losses.mse_adc, many(a1), many(b1))
    sums = lambda p, q: [(np.exp(-0.5 * sum((p[k][:, None].astype(np.float64) - q[k][None]) ** 2   # noqa: E731
                                             for k in (1, 2, 3))) * w).sum(1)
                         for w in (q[0][None].astype(np.float64),
                                   q[0][None] * (p[3][:, None].astype(np.float64) - q[3][None]))]
    (sa, za), (sb, zb), (sc, _) = sums(a1, a1), sums(a1, b1), sums(b1, b1)
    w, v = a1[0].astype(np.float64), b1[0].astype(np.float64)
    sw, sv = copies * w.sum(), copies * v.sum()
    A, B, C = copies * (w * sa).sum(), copies * (w * sb).sum(), copies * (v * sc).sum()
    rel = (sw - sv) / (sv + 1e-6)
    want = A / sw ** 2 + C / sv ** 2 - 2 * B / (sw * sv) + rel ** 2
    assert abs(loss - want) <= LOSS_RTOL * abs(want)
    wq = 2 * sa / sw ** 2 - 2 * A / sw ** 3 - 2 * sb / (sw * sv) + 2 * B / (sw ** 2 * sv) + 2 * rel / (sv + 1e-6)
    _close(gq, np.tile(wq, copies))
    _close(gz, np.tile(-2 * w * (za / sw ** 2 - zb / (sw * sv)), copies))


@pytest.mark.gpu
def test_pair_sums_keep_nan(cuda):
    """A NaN weight reaches the loss although its hit lies far from all others."""
    rng = np.random.default_rng(5)
    a, b = _hits(rng, 200, 1, 5.0), _hits(rng, 200, 1, 5.0)
    a[1][-1] = 500.0
    a[0][-1] = np.nan
    assert np.isnan(_run(losses.mse_adc, a, b)[0])
