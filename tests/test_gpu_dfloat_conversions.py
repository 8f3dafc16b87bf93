"""The integer conversions between double and float inside the double-float exp and log
(xreac_gb300/csrc/xr_dfloat.cuh), at the arguments where their two routes meet: reduced arguments that are zero,
below float's normal range, halves of a float's last place, and both ends of log's domain. Bounds as for the functions
themselves: 2e-14 relative for exp, 2e-14 absolute or relative for log."""

import numpy as np
import pytest
from test_gpu_dfloat import _apply

pytestmark = pytest.mark.gpu


def edges():
    step = np.log(2.0) / 64
    k = np.arange(-640, 641)
    tiny = np.concatenate([s * 2.0 ** np.arange(-1074, -20, 3.0) for s in (1.0, -1.0)])
    half = np.float64(np.float32(1.0)) * (1.0 + 2.0**-24 * np.arange(-9, 10)) + 2.0**-52 * np.arange(-9, 10)
    return tiny, (k * step), half


def test_exp_where_the_reduced_argument_is_tiny_or_a_tie():
    tiny, multiples, half = edges()
    x = np.concatenate([tiny, multiples, multiples + 2.0**-40, half, -half, half * 2.0**-8, [0.0, -0.0]])
    got, want = _apply(0, x), _apply(1, x)
    assert (np.abs(got - want) / want).max() < 2e-14


@pytest.mark.parametrize("scale", [2.0**-99, 2.0**-97, 2.0**-96, 2.0**-95, 1.0, 2.0**60, 2.0**99])
def test_log_at_both_ends_and_at_ties(scale):
    _, _, half = edges()
    a = np.concatenate([half, half * 1.99, half * 1.41]) * scale
    got, want = _apply(2, a), _apply(3, a)
    assert (np.abs(got - want) / np.maximum(1.0, np.abs(want))).max() < 2e-14
