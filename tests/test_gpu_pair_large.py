"""mse_adc's charge gradient on large events, without column slices, against float64."""

import numpy as np
import pytest

from larndsim_gb300 import consts, losses


@pytest.mark.gpu
def test_mse_adc_large_events(cuda):
    """12 events of 9000 hits in 4 cm, the reference hits 200 cm away, charge
    term off: dL/dQ = 2 a / sw^2 - 2 A / sw^3 with a a sum of 9000 terms.  Added
    one by one in float32 they carry 2^-25 sqrt(9000 / 3) = 1.6e-6 of a, in
    groups of 1024 and then by group 2^-25 (sqrt(1024 / 3) / 3 + sqrt(9 / 3)) =
    2.3e-7, besides a kernel value's own errors (1.2e-7 in common)."""
    import torch
    rng = np.random.default_rng(4)
    E, n = 12, 9000
    ev = torch.arange(E, device="cuda").repeat_interleave(n).int()
    hit = lambda lo, hi: torch.from_numpy(rng.uniform(lo, hi, E * n).astype(np.float32)).cuda()   # noqa: E731
    q, x, y, z = hit(1, 30), (hit(0, 4) * 2).round() / 2, hit(0, 4), hit(0, 4)
    zero, one = torch.zeros(E * n, device="cuda"), torch.ones(E * n, device="cuda")
    qg = q.clone().requires_grad_(True)
    loss, _ = losses.mse_adc(consts.Params(), qg, x, y, z, zero, one, ev, q, x + 200, y, z, zero, one, ev, lambda_Q=0)
    loss.backward()
    w = q.double()
    a = torch.cat([torch.exp(-0.5 * sum((c[s][:, None].double() - c[s][None].double()) ** 2 for c in (x, y, z))) @ w[s]
                   for s in (slice(e * n, (e + 1) * n) for e in range(E))])
    sw = w.sum()
    want = 2 * a / sw ** 2 - 2 * (w * a).sum() / sw ** 3
    err, size = (qg.grad.double() - want).square().mean().sqrt(), (2 * a / sw ** 2).square().mean().sqrt()
    assert float(err) <= 6e-7 * float(size)
