"""Densities of the unconstrained tracked waves at the start of an MD segment
against extended-precision sums, for both kernels (axis tables; a sincos per
pair for components of 200 and more) at the edges of their tiles: one particle,
fewer than a tile, more than a cluster's tiles, waves around the 512 of a CTA,
components of both signs, tiles of 64 and 32 particles. The box edge is a power
of two, so the fractional positions are exact. Bound: a table entry is at most
7 products from its anchor (22 roundings), a wave multiplies d of them, the sum
adds n terms - 80 roundings a term cover d = 3."""

from __future__ import annotations

import numpy as np
import pytest

from xla_cco.dynamics import MDSettings, Waves, init_state, make_key
from xla_cco.energy import StealthyEnergy

pytestmark = pytest.mark.gpu


CASES = [(1, 60, 5, 3), (1, 150, 40, 700), (1, 300, 33, 65), (2, 5, 1, 1), (2, 16, 511, 31), (2, 18, 512, 64),
         (2, 20, 700, 530), (2, 70, 90, 33), (3, 4, 200, 63), (3, 30, 65, 129), (3, 45, 17, 1100)]  # fmt: skip


@pytest.mark.parametrize("d,r,extra,n", CASES)
def test_fresh_wave_densities(d, r, extra, n):
    rng = np.random.default_rng(10 * d + r)
    inner = np.eye(d)
    rows = np.unique(rng.integers(-r, r + 1, size=(4 * extra + 40, d)), axis=0)
    rows = rows[(np.abs(rows) > 1).any(axis=1)]
    rows = rng.permutation(rows)[:extra].astype(np.float64)
    rows[-1, 0] = r
    edge, b = 16.0, 3
    basis = edge * np.eye(d)
    nv = np.concatenate([inner, rows])
    waves = Waves(n_vectors=nv, kvec=nv @ (2.0 * np.pi * np.linalg.inv(basis).T),
                  constrained=np.arange(len(nv)) < d, n_constrained=d)  # fmt: skip
    en = StealthyEnergy(inner, np.ones(d), np.float64(edge**d))
    r0 = rng.uniform(-1.0, 2.0, size=(b, n, d)) * edge       # unwrapped positions
    keys = np.stack([make_key(i) for i in range(b)])
    st = MDSettings(dt=0.01, scheme="verlet", chunk_steps=1, drift_tol=np.inf)
    out = init_state(en, waves, basis, r0, np.zeros_like(r0), np.full(b, 0.1), keys, st)
    s = (r0 / edge).astype(np.longdouble)
    for i in range(b):
        x = s[i] @ nv.T.astype(np.longdouble)
        x = 2 * np.longdouble("3.14159265358979323846") * (x - np.rint(x))
        ref = np.stack([np.cos(x).sum(0), np.sin(x).sum(0)], axis=-1)
        np.testing.assert_allclose(out.rho_prev[i], ref.astype(np.float64), rtol=0, atol=n * 80 * 2.0**-53)
