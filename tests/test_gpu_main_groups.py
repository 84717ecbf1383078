"""The main-bin kernels' split (two segments with one template a warp at a
time, 24 warps a block): segment counts at the edges of the groups, blocks and
template runs give the waveforms of the CPU oracle, and every launch shape
the same bits."""

from __future__ import annotations

import numpy as np
import pytest

from gpu_common import WFS_RTOL, compare_wfs, small_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 47, 48, 49, 97, 640])
@pytest.mark.parametrize("spread", [0.0, 25.0])
def test_group_edges(cuda, n, spread):
    """``spread`` 0: all segments at one drift distance (one template)."""
    import torch
    from larndsim_gb300 import grad, sim, tune, workloads
    from oracle import reference_np as R
    p = small_params(n_neighbors=1, n_templates=20)
    tmpl = R.load_lut_templates(workloads.synthetic_response(seed=0, nx=15, ny=15), p)
    tracks, fields = workloads.shower_event(seed=n, n_segments=n)
    z = (15.0 + spread * (np.random.default_rng(n).random(n) - 0.5)).astype(np.float32)
    for k in ("z", "z_start", "z_end"):
        tracks[:, fields.index(k)] = z
    bank = torch.from_numpy(tmpl).cuda()
    sim.reset_size_history()
    wfs, unique = sim.simulate_wfs(p, bank, tracks, fields)
    ref, uref = R.simulate_wfs(p, tmpl, tracks, fields, history={})
    assert compare_wfs(wfs.cpu().numpy(), unique.cpu().numpy(), ref, uref) < WFS_RTOL
    chain = grad.LUTChain(p, bank, tracks, fields, n_events=1)
    # through the adjoint of the waveforms: a few segments make no hits
    cot = torch.randn(wfs.shape, generator=torch.Generator().manual_seed(n)).cuda()
    base = chain.wfs_vjp(p, cot).cpu().numpy()
    assert np.isfinite(base).all() and (base[[0, 2, 5, 6]] != 0).all()
    try:
        for cfg in ({"main_block_warps": 8}, {"main_block_warps": 4, "main_blocks": 3}, {"main_blocks": 1}):
            tune.set_tuning(cfg)
            assert np.array_equal(base, chain.wfs_vjp(p, cot).cpu().numpy()), cfg
            assert np.array_equal(wfs.cpu().numpy(), sim.simulate_wfs(p, bank, tracks, fields)[0].cpu().numpy()), cfg
    finally:
        tune.set_tuning(None)
