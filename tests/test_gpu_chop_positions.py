"""chop_tracks' float-pair positions against the oracle's float64 ones, bit for
bit, where their rounding is in doubt or leaves the pair's range: positions
half way between floats, cancellation across zero, tiny and large steps, more
than 2^24 steps; and at the edges of the 128-row tiles."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _tracks(starts, ends):
    from larndsim_gb300 import workloads
    s, e = np.asarray(starts, np.float32), np.asarray(ends, np.float32)
    n = s.shape[0]
    return workloads._rows(s, e, np.linspace(0.1, 3.0, n), 0, np.arange(n), 13), workloads.SEGMENT_FIELDS


def _check(tracks, fields, precision):
    from larndsim_gb300 import dataio
    from oracle import reference_np as R
    got = dataio.chop_tracks(tracks, fields, precision).cpu().numpy()
    want = R.chop_tracks(tracks, fields, precision)
    assert got.shape == want.shape and np.array_equal(got.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("exp", [-22, -24, -25, -26])
def test_ties(cuda, exp):
    """Axis-aligned tracks with a power-of-two step: every other position is a tie."""
    step = 2.0 ** exp
    n = 700
    s = [[1.0, 0.25, -1.0], [3.0, -2.0, 0.5], [-1.0, 1.0, 1.0]]
    e = [[1.0 + n * step * 8, 0.25, -1.0], [3.0, -2.0 - n * step * 16, 0.5], [-1.0, 1.0, 1.0 + n * step * 8]]
    _check(*_tracks(s, e), step)


@pytest.mark.parametrize("precision", [1e-6, 1e-3, 0.04, 0.3, 7.0])
@pytest.mark.parametrize("scale", [1e-12, 1e-3, 1.0, 1e6])
def test_positions(cuda, precision, scale):
    rng = np.random.default_rng(int(1e6 * precision))
    n, steps = 40, 300
    s = rng.uniform(-1, 1, (n, 3)) * scale
    d = rng.normal(size=(n, 3))
    d *= precision * rng.uniform(0, steps, (n, 1)) / np.linalg.norm(d, axis=1, keepdims=True)
    s[:5] = 0.0
    s[5:10] = -0.5 * d[5:10]          # through zero
    e = s + d
    _check(*_tracks(s, e), precision)


@pytest.mark.parametrize("rows", [1, 127, 128, 129, 255, 256, 257])
@pytest.mark.parametrize("tracks", [1, 3, 0])
def test_tile_edges(cuda, rows, tracks):
    """``rows`` steps in one track, in three, and one each."""
    t = rows if tracks == 0 else min(tracks, rows)
    n = np.full(t, rows // t)
    n[: rows % t] += 1
    s = np.random.default_rng(rows).uniform(-20, 20, (t, 3))
    e = s.copy()
    e[:, 1] += (n - 0.5) * 0.25
    _check(*_tracks(s, e), 0.25)


def test_more_than_2_to_24_steps(cuda):
    from larndsim_gb300 import dataio
    tracks, fields = _tracks([[0.3, 0.1, -0.2]], [[0.3, 17.0, 3.0]])
    prec = 1e-6
    out = dataio.chop_tracks(tracks, fields, prec)
    n = out.shape[0]
    assert n > (1 << 24) + 1000
    f = np.float32
    s = tracks[0, [fields.index(k) for k in ("x_start", "y_start", "z_start")]]
    e = tracks[0, [fields.index(k) for k in ("x_end", "y_end", "z_end")]]
    seg = (e - s).astype(f)
    length = np.sqrt(((seg[0] * seg[0] + seg[1] * seg[1]).astype(f) + seg[2] * seg[2]).astype(f)).astype(f)
    d = (seg / f(length + f(1e-10))).astype(f)
    for k in (0, 1, (1 << 24) - 1, 1 << 24, (1 << 24) + 1, n - 2):
        want = (s.astype(np.float64) + (k * prec) * d.astype(np.float64)).astype(f)
        got = out[k, [fields.index(q) for q in ("x_start", "y_start", "z_start")]].cpu().numpy()
        assert np.array_equal(got, want), k
