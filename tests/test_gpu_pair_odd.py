"""nll_loss and mse_adc with hits that are not finite, and with events in no order."""

import numpy as np
import pytest

from larndsim_gb300 import losses
from test_gpu_pair_tiles import _close, _hits, _nll64, _run

pytestmark = pytest.mark.gpu


def _events(n, m, seed, n_events=4, spread=8.0):
    rng = np.random.default_rng(seed)
    return _hits(rng, n, n_events, spread), _hits(rng, m, n_events, spread)


@pytest.mark.parametrize("column", [0, 1, 2, 3])
def test_nll_nan_reference_hit(cuda, column):
    """Its lambda is NaN, and so are the loss and the gradients of its event's hits."""
    a, b = _events(500, 700, 11)
    b[column][int(np.nonzero(b[6] == 2)[0][5])] = np.nan
    loss, gq, gz = _run(losses.nll_loss, a, b)
    assert np.isnan(loss) and np.isnan(gz[a[6] == 2]).all() and np.isnan(gq[a[6] == 2]).all()


@pytest.mark.parametrize("column", [1, 2])
def test_nll_reference_hit_at_infinity(cuda, column):
    """Its lambda is 0 and its kernel values are 0: the rest is as without it."""
    a, b = _events(500, 700, 11)
    j = int(np.nonzero(b[6] == 2)[0][5])
    b[column][j] = np.inf
    loss, gq, gz = _run(losses.nll_loss, a, b)
    loss0, gq0, gz0 = _run(losses.nll_loss, a, [np.delete(c, j) for c in b])
    assert abs(loss - (loss0 - np.log(1e-10))) <= 1e-5 * abs(loss)
    _close(gq, gq0)
    _close(gz, gz0)


@pytest.mark.parametrize("column", [1, 2])
def test_nll_predicted_hit_at_infinity(cuda, column):
    a, b = _events(300, 400, 12)
    loss0 = _run(losses.nll_loss, [c[:-1] for c in a], b)[0]
    a[column][-1] = np.inf
    loss = _run(losses.nll_loss, a, b)[0]
    assert abs(loss - (loss0 + 1.0)) <= 1e-5 * abs(loss0)


@pytest.mark.parametrize("column", [1, 2, 3])
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_mse_adc_odd_coordinate(cuda, column, value):
    """A distance to itself that is NaN reaches the loss, however far its chunk."""
    a, b = _events(900, 800, 13, n_events=2, spread=60.0)
    a[column][3] = value
    assert np.isnan(_run(losses.mse_adc, a, b)[0])


def test_nll_shuffled_events(cuda):
    a, b = _events(600, 900, 14)
    rng = np.random.default_rng(15)
    a, b = ([c[p] for c in h] for h, p in ((a, rng.permutation(600)), (b, rng.permutation(900))))
    loss, gq, gz = _run(losses.nll_loss, a, b)
    want, wq, wz = _nll64(a, b)
    assert abs(loss - want) <= 1e-5 * max(abs(want), 1.0)
    _close(gq, wq)
    _close(gz, wz)
