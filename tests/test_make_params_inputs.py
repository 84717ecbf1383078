"""make_params on parameter values that are not plain numbers."""

import math

import numpy as np
import pytest

from larndsim_gb300 import _abi, consts


@pytest.mark.parametrize("field", ["Ab", "kb", "alpha", "beta", "shift_x", "UNCORRELATED_NOISE_CHARGE"])
def test_unset_parameter_is_nan(field):
    """A parameter that the recombination mode or the path does not use may be None."""
    lp = _abi.make_params(consts.Params(**{field: None}))
    name = {"UNCORRELATED_NOISE_CHARGE": "uncorr_noise"}.get(field, field)
    assert math.isnan(getattr(lp, name))


@pytest.mark.parametrize("pitch", [np.float32(0.38), np.float32(0.4434), np.float64(0.38), np.array(0.38, np.float32)])
@pytest.mark.parametrize("bins", [10, np.int64(10), np.float32(10)])
def test_edges_in_the_parameters_own_arithmetic(pitch, bins):
    """The bin edges are the expression on the values as they are given; plain
    numbers of the same value before and after change nothing."""
    for p in (float(pitch), pitch, float(pitch)):
        params = consts.Params(pixel_pitch=p, nb_sampling_bins_per_pixel=bins)
        sym = (params.nb_tran_diff_bins - 1) // 2
        width = p / bins
        want = consts.jax_linspace_f32(-sym * width, (sym + 1) * width, params.nb_tran_diff_bins + 1)
        got = np.array(_abi.make_params(params).tran_edges[:len(want)], np.float32)
        assert np.array_equal(got, np.asarray(want, np.float32))
