"""Pair histogram and nearest neighbours on cell grids (diagonal bases, edges well
inside the box) against all pairs in double precision: exact counts and bit-equal
distances. Even edges (bins decided in single precision away from the edges),
edges at distances that occur, uneven and very narrow bins (every pair measured),
a first edge above zero; uniform, lattice, unwrapped and far-away positions, a
crowded cell, coincident and non-finite particles; sizes around a warp's rows, a
CTA's share and several CTAs."""

from __future__ import annotations

import numpy as np
import pytest

from xla_cco.analysis.pairs import nearest_neighbor_distances_batch, pair_distance_histogram
from xla_cco.box import Box

pytestmark = pytest.mark.gpu


def _r(s, side):
    """(N, N) distances of the nearest image on a diagonal basis."""
    ds = s[None] - s[:, None]
    v = (ds - np.rint(ds)) * side
    r2 = np.zeros(v.shape[:2])
    for c in range(v.shape[2]):
        r2 = r2 + v[..., c] * v[..., c]
    return np.sqrt(r2)


def _positions(kind, rng, b, n, d):
    s = rng.uniform(size=(b, n, d))
    if kind == "lattice":       # many equal distances, coincident particles, cell boundaries
        s = np.floor(20.0 * s) / 20.0
    elif kind == "unwrapped":
        s = s + rng.integers(-3, 4, size=s.shape)
    elif kind == "far":         # beyond the reach of the grid: all pairs
        s[0] += 1.0e6
    elif kind == "crowded":     # most of one configuration in a hundredth of the box
        s[-1, : 3 * n // 4] *= 0.01
    elif kind == "edge":        # just below and at the box's faces
        s[:, ::5] = np.where(rng.uniform(size=s[:, ::5].shape) < 0.5, -1e-18, 1.0 - 2.0**-53)
    elif kind == "nan":
        s[0, n // 2] = np.nan
    return s


CASES = [(2, 64, 3, "uniform"), (2, 1000, 2, "uniform"), (2, 1500, 1, "lattice"), (2, 333, 2, "unwrapped"),
         (2, 200, 2, "far"), (2, 600, 2, "crowded"), (2, 500, 2, "edge"), (2, 129, 2, "nan"),
         (1, 97, 2, "uniform"), (1, 700, 1, "lattice"), (3, 1100, 1, "uniform"), (3, 512, 2, "lattice"),
         (3, 900, 1, "edge"), (1, 400, 2, "crowded")]  # fmt: skip


@pytest.mark.parametrize("d,n,b,pos", CASES)
@pytest.mark.parametrize("edges", ["even", "from", "narrow", "uneven", "at_distances"])
def test_cell_grids_vs_all_pairs(d, n, b, pos, edges):
    rng = np.random.default_rng(31 * n + d)
    side = n ** (1.0 / d) * np.array([1.0, 0.8, 1.3])[:d]
    s = _positions(pos, rng, b, n, d)
    dist = [_r(x, side) for x in s]
    off = np.concatenate([r[np.triu_indices(n, 1)] for r in dist])
    off = off[np.isfinite(off)]
    top = 0.18 * side.min()
    near = np.sort(off[off < top])
    e = {"even": np.linspace(0.0, top, 201), "from": np.linspace(0.3 * top, top, 51),
         "narrow": np.linspace(0.5 * top, 0.5 * top * (1.0 + 1e-4), 101),
         "uneven": np.r_[0.0, np.geomspace(1e-3 * top, top, 30)],
         "at_distances": np.unique(np.r_[0.0, near[:: max(1, near.size // 50)]])}[edges]
    if len(e) < 2:
        e = np.array([0.0, top])
    got = pair_distance_histogram(s, Box(np.diag(side)), e)
    np.testing.assert_array_equal(got, np.histogram(off, bins=e)[0])
    if edges == "even":
        nn = nearest_neighbor_distances_batch(s, Box(np.diag(side)))
        for i, r in enumerate(dist):
            np.fill_diagonal(r, np.inf)
            lone = np.where(np.isfinite(s[i]).all(1), side.min(), np.inf)   # its own nearest image
            np.testing.assert_array_equal(nn[i], np.fmin(np.fmin.reduce(r, axis=1), lone))
