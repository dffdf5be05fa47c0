"""The Hessian's matrix-pipe tiles against the closed form in NumPy at the edges
of their tiling: particle counts around 32, k counts off 16, batches, and phases
that come in several k-chunks. 1e-11 of max |H| (the package's own tolerance) and
exact symmetry."""

from __future__ import annotations

import numpy as np
import pytest

from xla_cco.workloads import energy_for

pytestmark = pytest.mark.gpu


def _phase(nv, s):
    hi = np.round(s * 2.0**26) / 2.0**26   # n hi is exact: its whole part leaves before rounding
    t = nv @ hi.T
    return 2.0 * np.pi * ((t - np.round(t)) + nv @ (s - hi).T)


def _rows(en, s, js):
    """Rows (j, a) of the Hessian for the particles js: (len(js) d, N d)."""
    n, d = s.shape
    nv, w = en.n_vectors[en._rows], en.weights[en._rows]
    th = _phase(nv, s)
    c, sn = np.cos(th), np.sin(th)
    re, im = c.sum(1), sn.sum(1)
    out = np.zeros((len(js), d, n, d))
    for a in range(d):
        for b in range(d):
            q = w * nv[:, a] * nv[:, b]
            blk = (q[:, None] * c[:, js]).T @ c + (q[:, None] * sn[:, js]).T @ sn
            dg = (q[:, None] * (re[:, None] * c[:, js] + im[:, None] * sn[:, js])).sum(0)
            blk[np.arange(len(js)), js] -= dg
            out[:, a, :, b] = blk
    return 2.0 * (2.0 * np.pi) ** 2 / float(en.volume) * out.reshape(len(js) * d, n * d)


@pytest.mark.parametrize("d,n,chi,b", [(1, 31, 0.4, 2), (1, 96, 0.3, 1), (2, 33, 0.4, 3), (2, 64, 0.2, 1),
                                       (2, 129, 0.45, 2), (3, 65, 0.3, 2), (3, 32, 0.4, 1), (2, 3, 0.9, 1)])  # fmt: skip
def test_hessian_vs_closed_form(d, n, chi, b):
    en = energy_for(n, d, chi)
    s = np.random.default_rng(n).uniform(size=(b, n, d))
    h = en.hessian(s)
    for i in range(b):
        ref = _rows(en, s[i], np.arange(n))
        np.testing.assert_allclose(h[i], ref, rtol=0, atol=1e-11 * np.abs(ref).max())
        assert np.array_equal(h[i], h[i].T)
    assert np.array_equal(en.hessian(s[0]), h[0])


def test_hessian_in_several_k_chunks():
    n = 6000   # 2940 rows x 6000 particles x 16 bytes: more phases than are held at a time
    en = energy_for(n, 1, 0.49)
    s = np.random.default_rng(8).uniform(size=(n, 1))
    h = en.hessian(s)
    js = np.array([0, 31, 32, 2999, 5999])
    ref = _rows(en, s, js)
    np.testing.assert_allclose(h[js], ref, rtol=0, atol=1e-11 * np.abs(ref).max())
    assert np.array_equal(h, h.T)
