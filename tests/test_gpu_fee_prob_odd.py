"""Adjoint of the probabilistic front end with cotangents and rows that are not
finite: a NaN or an infinity on any hit of a row makes the row's gradient NaN
(0 probability times infinity included) and touches no other row."""

import numpy as np
import pytest

from larndsim_gb300 import consts, sim

pytestmark = pytest.mark.gpu


def _rows(n, T):
    import torch
    rng = np.random.default_rng(T)
    w = np.zeros((n, T), np.float32)
    for r in range(n):
        t = rng.integers(T // 8, T // 2)
        w[r, t:t + T // 8] = rng.uniform(500, 3000)
    w[0, T // 16:-T // 16] = 3000      # hits on every step, so that no step is left out for the batch
    return torch.from_numpy(w).cuda()


def _grad(w, cot):
    import torch
    w = w.detach().requires_grad_(True)
    out = sim.average_hit_values(consts.Params(), w)
    torch.autograd.backward(out, cot)
    return w.grad, out


@pytest.mark.parametrize("hit,which,value", [(h, w, v) for h in (0, 1, 9) for w in (0, 1, 2)
                                             for v in (np.nan, np.inf, -np.inf)] + [(9, 0, 3e38), (9, 1, 3e38)])
def test_odd_cotangent(cuda, hit, which, value):
    """On the first hit, on one without probability and on the last step; 3e38
    overflows over the smallest denominator, 1e-10, of a hit without probability."""
    import torch
    n, T, H = 6, 700, 10
    w = _rows(n, T)
    g = torch.Generator(device="cuda").manual_seed(1)
    cot = [torch.randn((n, H), generator=g, device="cuda") for _ in range(3)]
    clean, out = _grad(w, cot)
    lam = out[2].detach()
    assert float(lam[0].min()) > 0.5 and float(lam[2, 9]) == 0
    cot[which][2, hit] = value
    got, _ = _grad(w, cot)
    keep = [r for r in range(n) if r != 2]
    assert torch.equal(got[keep], clean[keep])
    assert bool(torch.isnan(got[2]).all())


@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_odd_row(cuda, value):
    import torch
    n, T, H = 6, 700, 10
    w = _rows(n, T)
    g = torch.Generator(device="cuda").manual_seed(1)
    cot = [torch.randn((n, H), generator=g, device="cuda") for _ in range(3)]
    clean, _ = _grad(w, cot)
    odd = w.clone()
    odd[3, 400] = value
    got, out = _grad(odd, cot)
    keep = [r for r in range(n) if r != 3]
    assert torch.equal(got[keep], clean[keep])
    assert bool(torch.isnan(out[1][3].detach()).any()) and bool(torch.isnan(got[3]).all())


@pytest.mark.parametrize("hit", [0, 1])
def test_hit_without_cotangent(cuda, hit):
    """A row whose second hit has infinite arguments (and NaN partials): the
    gradient is NaN where that hit has a cotangent, and is not where it has none."""
    import torch
    w = torch.tensor([[1281.4675, 3e38, -2556.0]], device="cuda").requires_grad_(True)
    lam = sim.average_hit_values(consts.Params(fee_paths_scaling=2, MAX_ADC_VALUES=2), w)[2]
    assert lam[0, 0] == 1 and 1e-8 < lam[0, 1] < 2e-8
    lam[0, hit].backward()
    assert bool(torch.isnan(w.grad).all()) if hit else bool(torch.isfinite(w.grad).all())


def test_partials_without_weight(cuda):
    """A row that falls and rises by 1e31: where the minimum of a hit's two
    terms gives the one with a NaN partial no weight, 0 times it is NaN."""
    import torch
    w = np.random.default_rng(3).normal(300, 2000, (4, 65)).astype(np.float32)
    w[1, 1], w[1, 26] = -1e31, 1e31
    params = consts.Params(fee_paths_scaling=20, RESET_NOISE_CHARGE=50, DISCRIMINATION_THRESHOLD=-200)
    x = torch.from_numpy(w).cuda().requires_grad_(True)
    out = sim.average_hit_values(params, x)
    assert all(bool(torch.isfinite(o).all()) for o in out)
    torch.autograd.backward(out, [torch.ones_like(o) for o in out])
    odd = torch.isnan(x.grad).any(1).tolist()
    assert odd == [False, True, False, False]
