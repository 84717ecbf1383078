"""lsim_fee_prob_vjp_recorded takes a record for what it was made from only."""

import numpy as np
import pytest

from larndsim_gb300 import _abi, consts, sim

pytestmark = pytest.mark.gpu

PARAMS = consts.Params()


def _record(w, K, dist):
    """The record of a forward of the rows' values (or distributions)."""
    import torch
    lib, lp = _abi.load(), _abi.make_params(PARAMS)
    P, T = w.shape
    H = int(lp.max_adc_values)
    ws = torch.empty(lib.lsim_fee_prob_scratch_bytes(lp, P, T, K), dtype=torch.uint8, device="cuda")
    rec = torch.empty(max(lib.lsim_fee_prob_record_bytes(lp, 64, 32), 1), dtype=torch.uint8, device="cuda")
    d = [torch.empty((P, H, T - 1), device="cuda") if dist else None for _ in range(2)]
    red = [torch.empty((P, H), device="cuda") for _ in range(3)]
    _abi.check(lib, lib.lsim_fee_prob_record(lp, sim._ptr(w), P, T, K, 1e-9, *(sim._ptr(t) for t in d + red),
                                             sim._ptr(rec), rec.numel(), sim._ptr(ws), ws.numel(), sim._stream()))
    return rec


def _vjp(w, K, rec, kind):
    import torch
    lib, lp = _abi.load(), _abi.make_params(PARAMS)
    P, T = w.shape
    H = int(lp.max_adc_values)
    g = torch.zeros_like(w)
    rng = np.random.default_rng(3)
    cot = lambda *s: torch.from_numpy(rng.normal(size=s).astype(np.float32)).cuda()   # noqa: E731
    args = [None] * 5
    if kind in ("log_prob", "charge"):
        args[("log_prob", "charge").index(kind)] = cot(P, H, T - 1)
    else:
        args[2:] = [cot(P, H) for _ in range(3)]
    _abi.check(lib, lib.lsim_fee_prob_vjp_recorded(lp, sim._ptr(w), P, T, K, sim._ptr(rec), rec.numel(),
                                                   *(sim._ptr(t) for t in args), sim._ptr(g), sim._stream()))
    return g


def _rows(n, T):
    import torch
    rng = np.random.default_rng(T)
    w = np.zeros((n, T), np.float32)
    for r in range(n):
        t = rng.integers(T // 8, T // 2)
        w[r, t:t + T // 8] = rng.uniform(500, 3000)
    return torch.from_numpy(w).cuda()


@pytest.mark.parametrize("kind", ["values", "log_prob", "charge"])
@pytest.mark.parametrize("dist", [False, True])
def test_kind_of_record(cuda, dist, kind):
    import torch
    w = _rows(5, 400)
    g = _vjp(w, 20, _record(w, 20, dist), kind)
    if dist or kind == "values":
        assert bool(torch.isfinite(g).all()) and float(g.abs().max()) > 0
    else:
        assert bool(torch.isnan(g).all())


def test_record_of_another_call(cuda):
    import torch
    w = _rows(5, 400)
    rec = _record(w, 20, True)
    for other, K in ((_rows(4, 400), 20), (_rows(5, 200), 20), (w, 19), (_rows(6, 2000), 32)):
        assert bool(torch.isnan(_vjp(other, K, rec, "values")).all())
    assert bool(torch.isfinite(_vjp(w, 20, rec, "values")).all())
