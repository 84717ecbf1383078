"""The pixel kernels' two compilations, with and without noise draws: draws
that are all zero change nothing, and with draws the fused front end gives the
hits and the loss of the front end run on the stored waveforms."""

from __future__ import annotations

import numpy as np
import pytest

from gpu_common import small_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_segments", [40, 1500])
def test_noise_and_no_noise(cuda, n_segments):
    import torch
    from larndsim_gb300 import grad, sim, workloads
    p = small_params(n_neighbors=1)
    lut, p = sim.load_lut(workloads.synthetic_response(seed=0, nx=15, ny=15), p)
    tracks, fields = workloads.muon_event(seed=3, n_tracks=2)
    if n_segments > 100:
        tracks = np.concatenate([tracks, workloads.shower_event(seed=4, n_segments=n_segments)[0]])
    chain = grad.LUTChain(p, lut, tracks, fields)
    target = chain.target(p.replace(lifetime=2000.0))
    plain, ticks, _ = chain.adc(p)
    P, H = plain.shape
    zeros = torch.zeros((P, 1 + 3 * H), device="cuda")
    a, t, _ = chain.adc(p, zeros)
    assert torch.equal(a, plain) and torch.equal(t, ticks)
    assert torch.equal(chain.loss_and_grad_device(p, target, normals=zeros), chain.loss_and_grad_device(p, target))
    draws = torch.randn((P, 1 + 3 * H), generator=torch.Generator().manual_seed(1)).cuda()
    a, t, _ = chain.adc(p, draws)
    loss, g, wfs = chain.loss_and_grad_stored(p, target, normals=draws)
    adc, t2 = sim.fee_adc(p, wfs, normals=draws)
    assert torch.equal(t, t2) and torch.equal(a, adc)
    fused = chain.loss_and_grad_device(p, target, normals=draws).cpu().numpy()
    assert loss == fused[0] and np.array_equal(fused[1:], np.array(list(g.values()), np.float32)) and loss > 0
