"""Quotients through a kept reciprocal are NumPy's, for every kind of dividend
and divisor (two quotients per point: the rule that keeps one)."""

import numpy as np
import pytest

from test_gpu_division import _bits, _run, _same

pytestmark = pytest.mark.gpu


def either(u, s, i):
    return where(u[i - 1] > 0.0, u[i] / s, (0.75 * u[i]) / s)  # noqa: F821


def test_every_dividend_and_divisor():
    one = float(np.nextafter(2.0, 0.0))      # all-ones significand
    rng = np.random.default_rng(1)
    values = [3.0, 0.1, -7.0, 1.0 / 1536, one, float(np.nextafter(1.0, 2.0)), 2.0, 0.0, -0.0,
              np.inf, -np.inf, np.nan, 5e-324, 1e-308, 1.7e308, 2.0 ** -480, 2.0 ** 480,
              float(np.nextafter(2.0 ** -480, 0.0))]
    values += [float(x) for x in rng.random(8) + 1.0]
    for k, s in enumerate(values):
        u = _bits(np.float64, 100 + k)
        got, inner = _run(either, np.float64, u, s=s)
        with np.errstate(all="ignore"):
            c = u[inner]
            want = np.where(u[inner.start - 1:inner.stop - 1] > 0.0, c / s, (0.75 * c) / s)
            _same(got, want)
