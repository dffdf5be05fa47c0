"""Bins of the pair histogram around the number whose thresholds are formed on the
device: exact counts with edges at distances that occur, at zero, tiny and huge."""

from __future__ import annotations

import numpy as np
import pytest

from xla_cco.analysis.pairs import pair_distance_histogram
from xla_cco.box import Box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bins", [1022, 1023, 1024, 1025, 8192, 8193, 12000])
@pytest.mark.parametrize("side", [1.0, 37.5, 1e-150, 1e150])
def test_counts_with_many_edges(bins, side):
    rng = np.random.default_rng(bins)
    n = 180
    s = np.floor(64.0 * rng.uniform(size=(1, n, 2))) / 64.0   # many equal distances
    s[0, ::3] = rng.uniform(size=s[0, ::3].shape)
    v = s[0][None] - s[0][:, None]
    v = (v - np.rint(v)) * side
    r2 = v[..., 0] * v[..., 0]
    r2 = r2 + v[..., 1] * v[..., 1]
    off = np.sqrt(r2)[np.triu_indices(n, 1)]
    at = np.unique(off[off > 0.0])
    grid = np.linspace(0.0, 0.7 * side, bins + 1)
    e = np.unique(np.r_[0.0, at[: bins // 2], np.nextafter(at[: bins // 4], np.inf), grid[1:]])
    e = np.sort(rng.permutation(e)[: bins + 1])
    assert len(e) == bins + 1
    got = pair_distance_histogram(s, Box(side * np.eye(2)), e)
    np.testing.assert_array_equal(got, np.histogram(off, bins=e)[0])
