"""Scratch of the probabilistic front end: it follows the rows, ticks and paths
of the call, and nothing is written past it."""

import numpy as np
import pytest

from larndsim_gb300 import _abi, consts, sim

# 3 arrays of T (rounded up to 32) floats per path, rows at a time: two per SM, of at most 200 SMs
LIMIT = lambda rows, T, K: 4 * 3 * (T + 31) * K * min(rows, 400)   # noqa: E731


def _rows(n, T, seed=0):
    rng = np.random.default_rng(seed)
    w = np.zeros((n, T), np.float32)
    for r in range(n):
        t = rng.integers(T // 8, T // 2)
        w[r, t:t + T // 8] = rng.uniform(500, 3000)
    return w


@pytest.mark.parametrize("rows,T,K", [(0, 2000, 20), (1, 2000, 1), (1, 2000, 20), (3, 64, 4), (300, 100, 20),
                                      (100000, 2000, 20)])
def test_scratch_bytes(rows, T, K):
    lib = _abi.load()
    p = _abi.make_params(consts.Params())
    small = lib.lsim_fee_prob_scratch_bytes(p, rows, T, K)
    assert 256 <= small <= LIMIT(rows, T, K) + 1024
    assert small <= lib.lsim_fee_prob_workspace_bytes(p)
    record = lib.lsim_fee_prob_record_bytes(p, rows, K)
    assert lib.lsim_fee_prob_vjp_workspace_bytes(p, rows, K) <= record + LIMIT(rows, 2048, K) + 1024


@pytest.mark.gpu
@pytest.mark.parametrize("rows,T,K", [(1, 2000, 20), (3, 65, 4), (700, 200, 5)])
def test_scratch_is_enough(cuda, rows, T, K):
    """Exactly the scratch asked for, poisoned and with a guard behind it: the
    same outputs as with the largest workspace."""
    import torch
    lib = _abi.load()
    lp = _abi.make_params(consts.Params(fee_paths_scaling=K))
    w = torch.from_numpy(_rows(rows, T)).cuda()
    H = int(lp.max_adc_values)
    need = lib.lsim_fee_prob_scratch_bytes(lp, rows, T, K)
    outs = []
    for size, fill in ((need, 255), (lib.lsim_fee_prob_workspace_bytes(lp), 0)):
        ws = torch.full((size + 4096,), fill, dtype=torch.uint8, device="cuda")
        ws[size:] = 17
        for dist in (True, False):
            d = [torch.empty((rows, H, T - 1), device="cuda") for _ in range(2)] if dist else [None, None]
            red = [torch.empty((rows, H), device="cuda") for _ in range(3)]
            _abi.check(lib, lib.lsim_fee_prob(lp, sim._ptr(w), rows, T, K, 1e-9, *(sim._ptr(t) for t in d + red),
                                              sim._ptr(ws), size, sim._stream()))
            outs.append([t for t in d + red if t is not None])
        assert bool((ws[size:] == 17).all())
    for a, b in zip(outs[:2], outs[2:]):
        for x, y in zip(a, b):
            assert torch.equal(x, y)
    assert lib.lsim_fee_prob(lp, sim._ptr(w), rows, T, K, 1e-9, *(sim._ptr(t) for t in [None] * 2 + red),
                             sim._ptr(ws), need - 256, sim._stream()) == _abi.LSIM_ERR_CAPACITY


@pytest.mark.gpu
def test_one_row_allocates_little(cuda):
    import torch
    w = torch.from_numpy(_rows(1, 2000)).cuda()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    sim.average_hit_values(consts.Params(), w)
    assert torch.cuda.max_memory_allocated() - before < 4 << 20
