"""Adjoint of the probabilistic front end over path counts that do and do not
divide a block's threads (a round of the kernel holds 512 / paths classes),
against float64 central differences with the GPU's own choices held, and over
a batch of more rows than blocks fit on the device.

Tolerance: 5e-3 relative on each directional derivative, the bound that
float32 log-probabilities (log(Phi(a) - Phi(b))) leave at 20 paths; it does
not depend on the number of paths."""

from __future__ import annotations

import numpy as np
import pytest

from test_gpu_fee_prob_grad import RTOL, _functional, _run, case  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [1, 3, 7, 16, 17, 32])
def test_path_counts(cuda, case, K):  # noqa: F811
    p, w = case
    p = p.replace(fee_paths_scaling=K)
    w = w[:4]
    rng = np.random.default_rng(K)
    P, T = w.shape
    H = int(p.MAX_ADC_VALUES)
    red = [rng.standard_normal((P, H)) * 1e-2, rng.standard_normal((P, H)), rng.standard_normal((P, H))]
    g, top, n_exec = _run(p, w, red=red)
    assert top.shape[2] == K and np.all(np.isfinite(g))
    for _ in range(2):
        delta = rng.standard_normal(w.shape)
        eps = 1e-2
        w64 = w.astype(np.float64)
        fd = (_functional(p, w64 + eps * delta, top, n_exec, None, None, red)
              - _functional(p, w64 - eps * delta, top, n_exec, None, None, red)) / (2 * eps)
        an = float((g * delta).sum())
        assert abs(an - fd) <= RTOL * abs(fd) + 1e-9, (K, an, fd)


def test_rows_do_not_depend_on_the_batch(cuda, case):  # noqa: F811
    p, w = case
    rng = np.random.default_rng(5)
    H = int(p.MAX_ADC_VALUES)
    red = [rng.standard_normal((w.shape[0], H)) for _ in range(3)]
    g, _, _ = _run(p, w, red=red)
    n = 40
    many, _, _ = _run(p, np.tile(w, (n, 1)), red=[np.tile(r, (n, 1)) for r in red])
    assert np.array_equal(many, np.tile(g, (n, 1)))
