"""The probabilistic front end makes the adjoint's record only where a backward
pass can follow (the kernels replaced by a stand-in)."""

import pytest
import torch

from larndsim_gb300 import consts, sim


@pytest.mark.parametrize("fn", [sim.average_hit_values, sim.get_adc_values_average_noise_vmap])
@pytest.mark.parametrize("requires,mode,want", [(True, torch.enable_grad, True), (True, torch.no_grad, False),
                                                (False, torch.enable_grad, False),
                                                (True, torch.inference_mode, False)])
def test_record_follows_grad_mode(monkeypatch, fn, requires, mode, want):
    made = []

    def stand_in(params, wfs, stop_threshold, distributions, reductions, record=False):
        made.append(bool(record))
        P, H = wfs.shape[0], int(params.MAX_ADC_VALUES)
        d = [torch.zeros(P, H, wfs.shape[1] - 1) if distributions else None for _ in range(2)]
        return (*d, [torch.zeros(P, H) for _ in range(3)], torch.zeros(1, dtype=torch.uint8) if record else None)

    monkeypatch.setattr(sim, "_fee_prob", stand_in)
    monkeypatch.setattr(sim, "_as_wfs", lambda w: w)
    w = torch.zeros(2, 50, requires_grad=requires)
    with mode():
        out = fn(consts.Params(), w)
    assert made == [want]
    assert all(o.requires_grad == want for o in out)
