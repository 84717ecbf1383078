"""chop_tracks on many tracks of one to three steps: up to 32 starts in a tile
of 32 rows, with a warp filling several tiles one after the other."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("most", [1, 2, 3, 40])
@pytest.mark.parametrize("tracks", [300001, 700000])
def test_short_tracks(cuda, tracks, most):
    from larndsim_gb300 import dataio, workloads
    from oracle import reference_np as R
    rng = np.random.default_rng(tracks + most)
    s = rng.uniform(-20, 20, (tracks, 3)).astype(np.float32)
    n = rng.integers(1, most + 1, tracks)
    if most == 40:                     # runs of one-step tracks between longer ones
        n[rng.uniform(size=tracks) < 0.9] = 1
    e = s.copy()
    e[:, 1] += ((n - 0.5) * 0.25).astype(np.float32)
    t = workloads._rows(s, e, rng.uniform(0.1, 3.0, tracks), 0, np.arange(tracks), 13)
    got = dataio.chop_tracks(t, workloads.SEGMENT_FIELDS, 0.25).cpu().numpy()
    want = R.chop_tracks(t, workloads.SEGMENT_FIELDS, 0.25)
    assert got.shape == want.shape and np.array_equal(got.view(np.uint32), want.view(np.uint32))
