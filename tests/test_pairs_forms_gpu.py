"""Pair statistics on a diagonal basis (one image, r2 thresholds) against the
minimum over all 3^d shifts, and on a sheared basis (all shifts): exact counts
and bit-equal nearest distances. Edges at distances that occur, uneven edges,
more bins than shared memory holds, ragged tiles, ties at half a box, coincident
and non-finite particles, unwrapped positions."""

from __future__ import annotations

import itertools

import numpy as np
import pytest

from xla_cco.analysis.pairs import nearest_neighbor_distances_batch, pair_distance_histogram
from xla_cco.box import Box

pytestmark = pytest.mark.gpu


def _basis(kind, d, n):
    side = n ** (1.0 / d)
    b = np.diag(side * np.array([1.0, 0.8, 1.3])[:d])
    if kind == "sheared" and d > 1:
        b[1, 0] = 0.3 * side
    return b


def _positions(n, d, b, kind):
    s = np.random.default_rng(17 * n + d).uniform(size=(b, n, d))
    if kind == "lattice":      # multiples of 1/8: many equal distances, |ds| = 1/2, coincident particles
        s = np.floor(8.0 * s) / 8.0
    if kind == "unwrapped":    # periodic copies
        s = s + np.random.default_rng(5).integers(-3, 4, size=s.shape)
    return s


@pytest.mark.parametrize("n,d,b,box,pos", [(127, 2, 3, "diagonal", "uniform"), (129, 3, 2, "diagonal", "lattice"),
                                           (257, 1, 2, "diagonal", "lattice"), (130, 2, 2, "sheared", "lattice"),
                                           (100, 3, 1, "sheared", "uniform"), (385, 2, 1, "diagonal", "unwrapped"),
                                           (2, 2, 1, "diagonal", "uniform")])  # fmt: skip
@pytest.mark.parametrize("edges", ["even", "at_distances", "uneven", "many"])
def test_histogram_and_nearest_vs_all_shifts(n, d, b, box, pos, edges):
    basis = _basis(box, d, n)
    s = _positions(n, d, b, pos)
    dist = [_distances(x, basis) for x in s]
    off = np.concatenate([r[np.triu_indices(n, 1)] for r in dist])
    top = off.max()
    e = {"even": np.linspace(0.0, 0.6 * top, 201), "uneven": np.unique(np.r_[0.0, np.geomspace(1e-3 * top, top, 40)]),
         "at_distances": np.unique(np.r_[0.0, off[:: max(1, off.size // 60)]]),
         "many": np.linspace(0.1 * top, top, 9002)}[edges]
    got = pair_distance_histogram(s, Box(basis), e)
    np.testing.assert_array_equal(got, np.histogram(off, bins=e)[0])
    nn = nearest_neighbor_distances_batch(s, Box(basis))
    for i, r in enumerate(dist):
        np.testing.assert_array_equal(nn[i], r.min(1))


def _distances(s, basis):
    """(N, N) minimum-image distances over the 3^d shifts, every operation
    rounded by itself; the diagonal holds a particle's own nearest image."""
    n, d = s.shape
    ds = s[None, :, :] - s[:, None, :]
    ds = ds - np.rint(ds)
    best = np.full((n, n), np.inf)
    for sh in itertools.product((-1.0, 0.0, 1.0), repeat=d):
        r2 = np.zeros((n, n))
        for a in range(d):
            v = np.zeros((n, n))
            for c in range(d):
                v = v + (ds[..., c] + sh[c]) * basis[c, a]
            r2 = r2 + v * v
        if not any(sh):
            r2[np.eye(n, dtype=bool)] = np.inf
        best = np.fmin(best, r2)
    return np.sqrt(best)


def test_non_finite_particles_are_not_counted():
    basis = np.diag([3.0, 4.0])
    s = np.random.default_rng(2).uniform(size=(1, 50, 2))
    s[0, 7, 1] = np.nan
    s[0, 9, 0] = np.inf
    keep = np.delete(s, [7, 9], axis=1)
    e = np.linspace(0.0, 3.0, 31)
    np.testing.assert_array_equal(pair_distance_histogram(s, Box(basis), e), pair_distance_histogram(keep, Box(basis), e))
    assert np.isinf(nearest_neighbor_distances_batch(s, Box(basis))[0, [7, 9]]).all()
