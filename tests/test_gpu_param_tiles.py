"""Parametrised mode's per-segment kernels at the edges of their split: odd
segment counts (two segments per warp), pairs with a segment that does not
contribute (no charge, outside the pixel plane, event -1), pixels with more
segments than a warp has lanes, and windows that cross either end of the
waveform, against the CPU oracle; and the adjoint on the same splits."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from gpu_common import WFS_RTOL, compare_wfs, small_params

pytestmark = pytest.mark.gpu


def _segments(n, spot, kill):
    """n segments within ``spot`` cm of one point; every ``kill``-th without charge."""
    from larndsim_gb300 import workloads
    tracks, fields = workloads.shower_event(seed=n, n_segments=n)
    c = {f: i for i, f in enumerate(fields)}
    rng = np.random.default_rng(n)
    for ax, at in (("x", 3.1), ("y", 5.2)):
        d = at + rng.uniform(-spot, spot, n).astype(np.float32) - tracks[:, c[ax]]
        for k in ("", "_start", "_end"):
            tracks[:, c[ax + k]] += d
    if kill:
        tracks[::kill, c["dE"]] = 0
        tracks[1::kill, c["x"]] = 40.0          # outside the pixel plane
        tracks[2::kill, c["eventID"]] = -1
    return tracks, fields


@pytest.mark.parametrize("n,spot,kill", [(1, 0.1, 0), (2, 0.1, 0), (3, 0.1, 3), (33, 0.02, 0), (64, 0.02, 5),
                                         (129, 0.1, 2), (1001, 3.0, 7)])
def test_param_tiles(cuda, n, spot, kill):
    from larndsim_gb300 import sim
    from oracle import reference_np as R
    p = small_params(n_neighbors=0, mc_diff=True)
    tracks, fields = _segments(n, spot, kill)
    nrm = np.random.default_rng(n + 1).standard_normal((n, 3)).astype(np.float32)
    sim.reset_size_history()
    wfs, unique = sim.simulate_parametrized_wfs(p, tracks, fields, offsets=torch.from_numpy(nrm).cuda())
    ref = R.simulate_parametrized(p, tracks, fields, nrm, history={})
    assert compare_wfs(wfs.cpu().numpy(), unique.cpu().numpy(), ref["wfs"], ref["unique_pixels"]) < WFS_RTOL


@pytest.mark.parametrize("n,spot", [(1, 0.1), (2, 0.1), (33, 0.02), (64, 0.02), (129, 0.1), (1001, 3.0)])
@pytest.mark.parametrize("every", [1, 2, 3])
def test_inert_segments_change_nothing(cuda, n, spot, every):
    """Chargeless copies of segments put between them move every segment to
    another place in its warp's pair and in its pixel's batch of 32, and leave
    waveforms and gradient as they are, bit for bit."""
    from larndsim_gb300 import grad, sim
    p = small_params(n_neighbors=0, mc_diff=True)
    tracks, fields = _segments(n, spot, 0)
    nrm = np.random.default_rng(n + 1).standard_normal((n, 3)).astype(np.float32)
    at = np.sort(np.concatenate([np.arange(n), np.arange(0, n, every)]))
    inert = np.concatenate([[False], at[1:] == at[:-1]])
    more = tracks[at].copy()
    more[inert, fields.index("dE")] = 0
    got = []
    for t, z in ((tracks, nrm), (more, nrm[at])):
        sim.reset_size_history()
        theta = grad.theta_of(p).requires_grad_(True)
        wfs, unique = sim.param_wfs_fn(theta, p, t, fields, z)
        c = np.random.default_rng(n + 2).standard_normal(tuple(wfs.shape)).astype(np.float32)
        wfs.backward(torch.from_numpy(c).cuda())
        got.append((unique.cpu().numpy(), wfs.detach().cpu().numpy(), theta.grad.cpu().numpy()))
    for a, b in zip(*got):
        assert np.array_equal(a, b)
    assert np.abs(got[0][2]).max() > 0


@pytest.mark.parametrize("interval", [(0, 20.0), (0, 12.8)])
def test_param_window_at_the_ends(cuda, interval):
    """Drift times from 0 to beyond a short waveform: windows cut at both ends."""
    from larndsim_gb300 import sim
    from oracle import reference_np as R
    p = small_params(n_neighbors=0, mc_diff=True, time_interval=interval)
    tracks, fields = _segments(150, 0.3, 0)
    z = np.linspace(30.58, 26.0, 150).astype(np.float32)     # the anode of TPC 0 is at z = 30.58975
    for k in ("z", "z_start", "z_end"):
        tracks[:, fields.index(k)] = z
    nrm = np.zeros((150, 3), np.float32)
    sim.reset_size_history()
    wfs, unique = sim.simulate_parametrized_wfs(p, tracks, fields, offsets=torch.from_numpy(nrm).cuda())
    ref = R.simulate_parametrized(p, tracks, fields, nrm, history={})
    assert compare_wfs(wfs.cpu().numpy(), unique.cpu().numpy(), ref["wfs"], ref["unique_pixels"]) < WFS_RTOL
