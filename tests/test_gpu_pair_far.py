"""mse_adc and nll_loss where a hit's sums rest on far pairs (kernel values down
to float32's smallest), against float64."""

import numpy as np
import pytest

from larndsim_gb300 import consts, losses

PARAMS = consts.Params()


def _grads(fn, a, b, **kw):
    import torch
    dev = [torch.from_numpy(v).cuda() for v in a]
    dev[0].requires_grad_(True)
    dev[3].requires_grad_(True)
    loss, _ = fn(PARAMS, *dev, *[torch.from_numpy(v).cuda() for v in b], **kw)
    loss.backward()
    return float(loss.detach()), dev[0].grad.cpu().numpy(), dev[3].grad.cpu().numpy()


def _hits(x, z, w, event=None):
    n = len(x)
    f = lambda v: np.array(np.broadcast_to(v, n), np.float32)   # noqa: E731
    ev = np.zeros(n, np.int32) if event is None else event.astype(np.int32)
    return [f(w), f(x), f(0.0), f(z), f(0.0), f(1.0), ev]


def _exact(a, b, sigma):
    """mse_adc's z gradient and the sum of its terms' absolute values."""
    w, v = a[0].astype(np.float64), b[0].astype(np.float64)
    def sums(p, q, m):   # noqa: E306
        same = p[6][:, None] == q[6][None]
        d = sum((p[k][:, None].astype(np.float64) - q[k][None]) ** 2 for k in (1, 2, 3))
        k = np.exp(-d / (2 * sigma ** 2)) * same * m[None]
        dz = p[3][:, None].astype(np.float64) - q[3][None]
        return (k * dz).sum(1), (k * abs(dz)).sum(1)
    (za, ta), (zb, tb) = sums(a, a, w), sums(a, b, v)
    sw, sv = w.sum(), v.sum()
    c = 2 * w / sigma ** 2
    return -c * (za / sw ** 2 - zb / (sw * sv)), c * (ta / sw ** 2 + tb / (sw * sv))


@pytest.mark.gpu
@pytest.mark.parametrize("n_near", [0, 500, 150000])
@pytest.mark.parametrize("sigma", [1.0, 1.3])
@pytest.mark.parametrize("gap", [6.0, 9.2, 9.6, 11.0, 12.5, 13.0, 13.6])
def test_mse_adc_far_hits(cuda, gap, sigma, n_near):
    """Two predicted hits and two reference hits, gap sigma apart in x and half
    of that in z, in a tile with hits of no weight; n_near dense others of small
    weight 200 cm away (150000: no column slices).  The rounding of a squared
    distance (2 for its differences, 2 for its sum, in units of 2^-24) is
    multiplied by the exponent; a kernel value is a multiple of 2^-149."""
    dense = np.sort(np.random.default_rng(1).uniform(200, 200 + 30 * max(1, n_near // 500), n_near))
    def hits(shift):   # noqa: E306
        far = (shift + np.array([0.0, gap] + [0.0] * 62)) * sigma
        return _hits(np.concatenate([far, dense]), np.concatenate([far / 2, 0 * dense]),
                     np.concatenate([[1.0, 1.0], np.zeros(62), np.full(n_near, 1e-5)]))
    a, b = hits(0.0), hits(2 * gap)
    got = _grads(losses.mse_adc, a, b, sigma=sigma)[2][:2].astype(np.float64)
    want, size = _exact([c[:64] for c in a], [c[:64] for c in b], sigma)
    share = (2.0 / a[0].astype(np.float64).sum()) ** 2
    want, size = want[:2] * share, size[:2] * share
    assert np.all(size > 0)
    exponent = 0.625 * gap ** 2
    tiny = 8 * 2.0 ** -149 * gap / sigma
    assert np.all(np.abs(got - want) <= (4 * exponent + 8) * 2.0 ** -24 * size + tiny)


@pytest.mark.gpu
@pytest.mark.parametrize("n_near", [0, 400])
@pytest.mark.parametrize("gap", [9.0, 11.7, 12.0, 13.0])
def test_nll_far_hits(cuda, gap, n_near):
    """One predicted hit gap sigma from the only reference hit near it: its z
    gradient is hp K dz / (lambda + 1e-10) with lambda = K."""
    dense = np.sort(np.random.default_rng(2).uniform(300, 330, n_near))
    def hits(x, z):   # noqa: E306   (the first tile: copies of the hit, far away in y)
        h = _hits(np.concatenate([np.full(64, x), dense]), np.concatenate([np.full(64, z), 0 * dense]), 10.0)
        h[2][:64] = 1000.0 * np.arange(64)
        return h
    a, b = hits(0.0, 0.0), hits(0.6 * gap, 0.8 * gap)
    got = float(_grads(losses.nll_loss, a, b, match_z=True)[2][0])
    dx, dz = (float(np.float64(p[0]) - np.float64(q[0])) for p, q in ((a[1], b[1]), (a[3], b[3])))
    k = np.exp(-0.5 * (dx * dx + dz * dz))
    want = k * dz / (k + 1e-10)
    assert abs(got - want) <= (4 * 0.5 * gap ** 2 + 8) * 2.0 ** -24 * abs(want)


@pytest.mark.gpu
@pytest.mark.parametrize("sigma", [3e-20, 1e-10, 1e10])
def test_mse_adc_extreme_sigma(cuda, sigma):
    """Kernel values 1 at the same place and 0 elsewhere, or 1 everywhere."""
    w = np.array([1.0, 2.0, 4.0, 8.0], np.float32)
    a = _hits(np.arange(4.0), np.arange(4.0), w)
    b = _hits(np.arange(4.0), np.arange(4.0), w[::-1])
    loss = _grads(losses.mse_adc, a, b, sigma=sigma)[0]
    same = sigma < 1
    aa, bb = ((w ** 2).sum(), (w * w[::-1]).sum()) if same else (w.sum() ** 2, w.sum() ** 2)
    want = 2 * (float(aa) - float(bb)) / float(w.sum()) ** 2
    assert abs(loss - want) <= 1e-6


@pytest.mark.gpu
@pytest.mark.parametrize("x0", [3e4, 1.5e5, 1e13, 1e19])
def test_mse_adc_outside_the_detector(cuda, x0):
    """Hits so far out that their event's offset does not keep them apart from
    other events' (a float32 swallows it, or their x makes up for it): every
    pair counts by its distance."""
    rng = np.random.default_rng(6)
    n = 200
    ev = np.repeat([0, 1], n // 2)
    def hits(seed):   # noqa: E306
        h = _hits(rng.uniform(0, 4, n), rng.uniform(0, 4, n), rng.uniform(1, 9, n), ev)
        h[1][[3, n - 4]] = [x0, x0 if x0 > 1e6 else x0 - 1e5]
        h[3][n - 4] = h[3][3] + np.float32(0.5)
        return h
    a, b = hits(0), hits(1)
    got = _grads(losses.mse_adc, a, b, lambda_Q=0)
    X = lambda h: np.stack([(h[1] + h[6].astype(np.float32) * np.float32(1e5)), h[2], h[3]], 1).astype(np.float64)   # noqa: E731
    w, v = a[0].astype(np.float64), b[0].astype(np.float64)
    K = lambda p, q: np.exp(-0.5 * ((X(p)[:, None] - X(q)[None]) ** 2).sum(2))   # noqa: E731
    sw, sv = w.sum(), v.sum()
    aa, bb, cc = K(a, a) @ w, K(a, b) @ v, K(b, b) @ v
    want = (w * aa).sum() / sw ** 2 + (v * cc).sum() / sv ** 2 - 2 * (w * bb).sum() / (sw * sv)
    wq = 2 * aa / sw ** 2 - 2 * (w * aa).sum() / sw ** 3 - 2 * bb / (sw * sv) + 2 * (w * bb).sum() / (sw ** 2 * sv)
    assert abs(got[0] - want) <= 1e-5 * abs(want)
    assert np.abs(got[1] - wq).max() <= 1e-5 * np.abs(wq).max()
