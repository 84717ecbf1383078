"""The front end's threshold path (no sweep of the row) against the sweeps it
replaces, restated in numpy with the kernels' own order of operations: ticks
and integrals bit for bit, on row lengths at the edges of the lanes' chunks,
with and without noise, and on the rows that keep the sweeps (not finite, or
beyond the threshold path's range)."""

import numpy as np
import pytest

from larndsim_gb300 import consts, sim

F = np.float32
TS = 0.125        # a power of two: charge * t_sampling is exact, so a fused multiply-add is an add


def _params(**kw):
    return consts.Params(t_sampling=TS, **kw)


def _cumulative(row):
    """Lane chunks summed in order, chunk totals by the warp's doubling scan."""
    T = row.size
    per = -(-T // 32)
    x = (row * F(TS)).astype(F)
    local = np.zeros(T, F)
    tot = np.zeros(32, F)
    for lane in range(32):
        s = F(0)
        for i in range(min(lane * per, T), min(lane * per + per, T)):
            s = F(s + x[i])
            local[i] = s
        tot[lane] = s
    incl = tot.copy()
    o = 1
    while o < 32:
        sh = incl.copy()
        sh[o:] = (incl[o:] + incl[:-o]).astype(F)
        incl = sh
        o *= 2
    off = (incl - tot).astype(F)
    out = local.copy()
    for lane in range(1, 32):
        b, e = min(lane * per, T), min(lane * per + per, T)
        out[b:e] = (off[lane] + local[b:e]).astype(F)
    return out


def _sweeps(row, params, normals):
    H, thr = params.MAX_ADC_VALUES, F(params.DISCRIMINATION_THRESHOLD)
    gap = consts.fee_interval(params)
    C, T = _cumulative(row), row.size
    on = normals is not None
    rn, un = F(params.RESET_NOISE_CHARGE), F(params.UNCORRELATED_NOISE_CHARGE)
    base = F(normals[0] * rn) if on else F(0)
    integral, ticks = np.zeros(H, F), np.zeros(H, F)
    for h in range(H):
        q = (base + C).astype(F)
        hit = np.flatnonzero((q[:-1] <= thr) & (q[1:] >= thr))
        idx = int(hit[0]) if hit.size else T - 2
        e, e2 = min(idx + 1 + gap, T - 1), min(idx + 2 + gap, T - 1)
        adc = F(F(base + C[e]) + (F(normals[1 + 3 * h] * un) if on else F(0))) if C[e] != 0 else C[e]
        reject = bool(adc < thr) or idx == T - 2
        integral[h], ticks[h] = (F(0), T - 2) if reject else (adc, idx)
        if on:
            base = F(normals[3 + 3 * h] * un) if reject else F(normals[2 + 3 * h] * rn)
        d = (C - C[e2]).astype(F)
        C = np.where(d < 0, F(0), d)
    return integral, ticks


def _rows(rng, n, T, scale):
    """Pulses of both signs on a small drift, some rows empty or flat."""
    w = rng.normal(0, scale * 0.002, (n, T))
    for r in range(n):
        for _ in range(rng.integers(0, 6)):
            t0, width = rng.integers(0, T), rng.integers(1, max(2, T // 8))
            w[r, t0:t0 + width] += rng.uniform(-0.5, 1.5) * scale / width
    w[0] = 0
    if n > 2:
        w[1] = scale / T
        w[2, : T // 2] = 0
    return w.astype(F)


@pytest.mark.gpu
@pytest.mark.parametrize("T", [2, 3, 4, 31, 32, 33, 63, 64, 65, 96, 500, 1999, 2000, 2016, 2047, 2048])
@pytest.mark.parametrize("noise", [False, True])
def test_threshold_path_equals_sweeps(cuda, T, noise):
    import torch
    rng = np.random.default_rng(T)
    p = _params(RESET_NOISE_CHARGE=900 if noise else 0, UNCORRELATED_NOISE_CHARGE=500 if noise else 0)
    n = 24
    w = _rows(rng, n, T, 4e5)
    nrm = rng.normal(size=(n, 1 + 3 * p.MAX_ADC_VALUES)).astype(F) if noise else None
    got_i, got_t = (v.cpu().numpy() for v in sim.get_adc_values(
        p, torch.from_numpy(w).cuda(), normals=None if nrm is None else torch.from_numpy(nrm)))
    for r in range(n):
        want_i, want_t = _sweeps(w[r], p, None if nrm is None else nrm[r])
        assert np.array_equal(got_t[r], want_t), r
        assert np.array_equal(got_i[r], want_i), r


@pytest.mark.gpu
@pytest.mark.parametrize("kw", [dict(DISCRIMINATION_THRESHOLD=0), dict(DISCRIMINATION_THRESHOLD=-100),
                                dict(MAX_ADC_VALUES=1), dict(MAX_ADC_VALUES=16),
                                dict(UNCORRELATED_NOISE_CHARGE=20000, RESET_NOISE_CHARGE=0)])
def test_threshold_path_odd_settings(cuda, kw):
    """Thresholds that the zeroed row meets, hit counts at their limits, and
    noise wider than the threshold (predicates that hold everywhere or nowhere)."""
    import torch
    p = _params(**{**dict(RESET_NOISE_CHARGE=0, UNCORRELATED_NOISE_CHARGE=0), **kw})
    rng = np.random.default_rng(7)
    w = _rows(rng, 24, 700, 4e5)
    nrm = rng.normal(size=(24, 1 + 3 * p.MAX_ADC_VALUES)).astype(F) if p.UNCORRELATED_NOISE_CHARGE else None
    got_i, got_t = (v.cpu().numpy() for v in sim.get_adc_values(
        p, torch.from_numpy(w).cuda(), normals=None if nrm is None else torch.from_numpy(nrm)))
    for r in range(24):
        want_i, want_t = _sweeps(w[r], p, None if nrm is None else nrm[r])
        assert np.array_equal(got_t[r], want_t) and np.array_equal(got_i[r], want_i), r


@pytest.mark.gpu
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, 1e34])
def test_rows_that_keep_the_sweeps(cuda, value):
    import torch
    p = _params(RESET_NOISE_CHARGE=0, UNCORRELATED_NOISE_CHARGE=0)
    rng = np.random.default_rng(9)
    w = _rows(rng, 16, 500, 4e5)
    w[np.arange(16), rng.integers(0, 500, 16)] = value
    got_i, got_t = (v.cpu().numpy() for v in sim.get_adc_values(p, torch.from_numpy(w).cuda()))
    with np.errstate(all="ignore"):
        for r in range(16):
            want_i, want_t = _sweeps(w[r], p, None)
            assert np.array_equal(got_t[r], want_t) and np.array_equal(got_i[r], want_i, equal_nan=True), r


@pytest.mark.gpu
@pytest.mark.parametrize("T", [4, 64, 128, 132, 2000, 2048])
def test_adjoint_on_both_paths(cuda, T):
    """dL/dwfs of the threshold path against the same adjoint in float64 with
    the hits' ticks held: float32 sums of at most 32 entries, so a few 1e-7 of
    the row's largest value."""
    import torch
    p = _params(RESET_NOISE_CHARGE=0, UNCORRELATED_NOISE_CHARGE=0)
    rng = np.random.default_rng(T + 1)
    w = _rows(rng, 16, T, 4e5)
    x = torch.from_numpy(w).cuda().requires_grad_(True)
    adc, ticks = sim.fee_adc(p, x)
    g = torch.from_numpy(rng.normal(size=tuple(adc.shape)).astype(F)).cuda()
    adc.backward(g)
    got, gap, H = x.grad.cpu().numpy(), consts.fee_interval(p), p.MAX_ADC_VALUES
    integral, _ = sim.get_adc_values(p, x.detach())
    integral, ticks, g = integral.cpu().numpy(), ticks.cpu().numpy(), g.cpu().numpy()
    for r in range(16):
        C = _cumulative(w[r])
        keeps, es, e2s, conds = [], [], [], []
        for h in range(H):
            cond = ticks[r, h] == T - 2
            q = C
            hit = np.flatnonzero((q[:-1] <= F(p.DISCRIMINATION_THRESHOLD)) & (q[1:] >= F(p.DISCRIMINATION_THRESHOLD)))
            idx = int(hit[0]) if hit.size else T - 2
            es.append(min(idx + 1 + gap, T - 1))
            e2s.append(min(idx + 2 + gap, T - 1))
            d = (C - C[e2s[-1]]).astype(F)
            keeps.append(~(d < 0))
            conds.append(cond)
            C = np.where(d < 0, F(0), d)
        G = np.zeros(T)
        for h in reversed(range(H)):
            G = np.where(keeps[h], G, 0.0)
            G[e2s[h]] -= G.sum()
            if not conds[h]:
                pre = integral[r, h] * p.GAIN + p.V_PEDESTAL - p.V_CM
                y = max(pre, 0) * p.ADC_COUNTS / (p.V_REF - p.V_CM)
                if pre > 0 and y < p.ADC_COUNTS:
                    G[es[h]] += g[r, h] * p.ADC_COUNTS / (p.V_REF - p.V_CM) * p.GAIN
        want = np.cumsum(G[::-1])[::-1] * TS
        assert np.abs(got[r] - want).max() <= 2e-6 * max(np.abs(want).max(), 1e-6), r
