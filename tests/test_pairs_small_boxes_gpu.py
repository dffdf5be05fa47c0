"""Pair histogram on cell grids of very small and very large boxes with fine even
bins: the single-precision bins must keep their distance from every length that
does not scale with the box. Exact counts, among them pairs at and near zero."""

from __future__ import annotations

import numpy as np
import pytest

from xla_cco.analysis.pairs import pair_distance_histogram
from xla_cco.box import Box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side", [1.05e-12, 3e-12, 1e-11, 3e-11, 1e-6, 1e3, 9e11])
@pytest.mark.parametrize("d,n,bins", [(2, 200, 8000), (2, 1000, 1000), (3, 700, 4001), (1, 128, 8000)])
def test_counts_do_not_depend_on_the_unit_of_length(side, d, n, bins):
    rng = np.random.default_rng(n + bins)
    s = rng.uniform(size=(1, n, d))
    s[0, 1::4] = s[0, ::4][: len(s[0, 1::4])]   # coincident pairs
    # pairs from 1e-9 to 1e-2 of the box apart
    k = len(s[0, 3::4])
    s[0, 3::4] = s[0, 2::4][:k] + 10.0 ** rng.uniform(-9, -2, size=(k, 1)) / np.sqrt(d)
    box = side * np.array([1.0, 0.9, 1.1])[:d]
    e = np.linspace(0.0, 0.25 * side, bins + 1)
    ds = s[0][None] - s[0][:, None]
    v = (ds - np.rint(ds)) * box
    r2 = np.zeros((n, n))
    for c in range(d):
        r2 = r2 + v[..., c] * v[..., c]
    off = np.sqrt(r2)[np.triu_indices(n, 1)]
    got = pair_distance_histogram(s, Box(np.diag(box)), e)
    np.testing.assert_array_equal(got, np.histogram(off, bins=e)[0])
