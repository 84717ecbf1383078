"""The slot lists' order (a thread per segment counts the segments before it):
list lengths at the edges of its unrolled loop, of warps and beyond a block's
worth give the CPU oracle's waveforms, and the same bits on every run although
segments arrive at their lists in any order."""

from __future__ import annotations

import numpy as np
import pytest

from gpu_common import WFS_RTOL, compare_wfs, small_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 31, 33, 65, 300, 9000])
def test_segments_of_one_pixel(cuda, n):
    import torch
    from larndsim_gb300 import grad, sim, workloads
    from oracle import reference_np as R
    p = small_params(n_neighbors=1)
    tmpl = R.load_lut_templates(workloads.synthetic_response(seed=0, nx=15, ny=15), p)
    tracks, fields = workloads.shower_event(seed=1, n_segments=n)
    rng = np.random.default_rng(n)
    col = fields.index
    for k in "xy":         # all in the first segment's pixel, or one beside it
        at = tracks[0, col(k)] + 0.02 * rng.random(n)
        tracks[:, col(k)] = tracks[:, col(k + "_start")] = tracks[:, col(k + "_end")] = at
    bank = torch.from_numpy(tmpl).cuda()
    sim.reset_size_history()
    wfs, unique = sim.simulate_wfs(p, bank, tracks, fields)
    if n <= 300:
        ref, uref = R.simulate_wfs(p, tmpl, tracks, fields, history={})
        assert compare_wfs(wfs.cpu().numpy(), unique.cpu().numpy(), ref, uref) < WFS_RTOL
    chain = grad.LUTChain(p, bank, tracks, fields, n_events=1)
    cot = torch.randn(wfs.shape, generator=torch.Generator().manual_seed(n)).cuda()
    g = chain.wfs_vjp(p, cot)
    for _ in range(3):
        sim.reset_size_history()
        again, _ = sim.simulate_wfs(p, bank, tracks, fields)
        assert torch.equal(again, wfs) and torch.equal(chain.wfs_vjp(p, cot), g)
