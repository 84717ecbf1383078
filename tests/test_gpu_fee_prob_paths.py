"""The probabilistic front end's values-only evaluation (ticks of no weight
left out, improbable pixels stopped, path values kept between steps) against
the evaluation that forms the full distributions: the same reductions bit for
bit, on the waveforms where the two could part; and the adjoint on a forward's
record against the adjoint that re-runs the forward, bit for bit."""

import numpy as np
import pytest
import torch

from larndsim_gb300 import _abi, consts, sim

pytestmark = pytest.mark.gpu


def _rows(T, seed):
    rng = np.random.default_rng(seed)
    t = np.arange(T)
    rows = [np.zeros(T), np.full(T, 0.5), np.full(T, 2.0), np.full(T, 30.0)]
    # rises around the line below which a tick is left out (1.4e-3 noise widths of 900 e- per tick of 0.1 us)
    rows += [np.full(T, r) for r in (12.5, 12.6, 12.7, 13.0)]
    for amp in (2e4, 8e4, 3e5, 5e6):
        for width in (1, 3, 20, 150):
            w = np.zeros(T)
            for t0 in rng.integers(0, max(1, T - 1), 3):
                w[t0:t0 + width] += amp / width / 0.1 * rng.uniform(0.3, 1.2)
            rows.append(w)
            rows.append(w + rng.uniform(0, 3, T))                     # on a pedestal: no tick without a rise
            rows.append(w * np.where(rng.random(T) < 0.2, -0.7, 1))    # both signs
    # a hit whose future falls far below threshold: its selection value is as low as a left-out tick's may be
    for fall in (1.5e5, 1.9e5, 2.5e5, 1e6):
        w = 3e4 / 10 / 0.1 * ((t >= T // 4) & (t < T // 4 + 10))
        rows.append(w - fall / 0.1 / 40 * ((t >= T // 2) & (t < T // 2 + 40)))
    bad = np.full(T, 20.0)
    bad[T // 2] = np.nan
    rows.append(bad)
    return np.array(rows, np.float32)


def _both(p, w):
    x = torch.from_numpy(w).cuda()
    _, _, full, _ = sim._fee_prob(p, x, 1e-9, True, True)
    _, _, only, _ = sim._fee_prob(p, x, 1e-9, False, True)
    return [[v.cpu().numpy() for v in g] for g in (full, only)]


@pytest.mark.parametrize("T", [40, 97, 600, 2000, 2048])
@pytest.mark.parametrize("K", [1, 8, 20, 32])
def test_values_only_equals_full(cuda, T, K):
    p = consts.Params(RESET_NOISE_CHARGE=900, fee_paths_scaling=K)
    full, only = _both(p, _rows(T, T + K))
    for a, b in zip(full, only):
        assert np.array_equal(a, b, equal_nan=True), np.argwhere(~((a == b) | (np.isnan(a) & np.isnan(b))))[:5]


@pytest.mark.parametrize("T,K", [(3, 2), (4, 3), (33, 20)])
def test_shortest_rows(cuda, T, K):
    p = consts.Params(RESET_NOISE_CHARGE=900, fee_paths_scaling=K)
    rng = np.random.default_rng(T)
    full, only = _both(p, (rng.normal(size=(16, T)) * 1e5).astype(np.float32))
    for a, b in zip(full, only):
        assert np.array_equal(a, b, equal_nan=True)


def test_more_pixels_than_blocks(cuda):
    """Pixels handed out by the counter: the rows of a large batch are those of a small one."""
    p = consts.Params(RESET_NOISE_CHARGE=900)
    w = _rows(500, 4)[:-1]
    _, small = _both(p, w)
    _, large = _both(p, np.tile(w, (20, 1)))
    for a, b in zip(small, large):
        assert np.array_equal(np.tile(a, (20, 1)), b)


@pytest.mark.parametrize("kind", ["values", "distributions"])
def test_recorded_adjoint_equals_rerun(cuda, kind):
    p = consts.Params(RESET_NOISE_CHARGE=900)
    w = torch.from_numpy(_rows(500, 5)[:-1]).cuda().requires_grad_(True)
    P, T = w.shape
    H, K = int(p.MAX_ADC_VALUES), int(p.fee_paths_scaling)
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    lib, lp = _abi.load(), _abi.make_params(p)
    ws = torch.empty(lib.lsim_fee_prob_vjp_workspace_bytes(lp, P, K), dtype=torch.uint8, device="cuda")
    rerun = torch.empty(P, T, device="cuda")
    if kind == "values":
        out = sim.average_hit_values(p, w)
        cot = [torch.randn(P, H, generator=g, device="cuda") for _ in range(3)]
        args = (None, None, *(c.data_ptr() for c in cot))
    else:
        out = sim.get_adc_values_average_noise_vmap(p, w)
        cot = [torch.randn(P, H, T - 1, generator=g, device="cuda") for _ in range(2)]
        args = (*(c.data_ptr() for c in cot), None, None, None)
    torch.autograd.backward(out, cot)
    _abi.check(lib, lib.lsim_fee_prob_vjp(lp, w.data_ptr(), P, T, K, 1e-9, *args, rerun.data_ptr(), ws.data_ptr(),
                                          ws.numel(), sim._stream()))
    torch.cuda.synchronize()
    assert torch.equal(w.grad, rerun) and bool((w.grad != 0).any())
