"""A particle with a non-finite coordinate makes its lane's energy, gradient and every
density row NaN, also rows whose component along that coordinate is zero (n . s is
NaN), in every form of the evaluation; the other lanes keep their bits."""

from __future__ import annotations

import numpy as np
import pytest

from xla_cco.energy import StealthyEnergy
from xla_cco.minimize import DescentSettings, relax

pytestmark = pytest.mark.gpu


def _ball(d, r):
    g = np.stack(np.meshgrid(*([np.arange(-r, r + 1)] * d), indexing="ij"), axis=-1).reshape(-1, d)
    first = np.array([x[np.flatnonzero(x)[0]] if x.any() else 0 for x in g])
    return g[(first > 0) & ((g * g).sum(1) < r * r)].astype(np.float64)


def _lines(d, r, top):
    v = [x for x in _ball(d, r).astype(int) if np.gcd.reduce(np.abs(x)) == 1]
    return np.array([i * x for x in v for i in range(1, int(top / np.sqrt(x @ x)) + 1)], dtype=np.float64)


def _axis(d, m):
    n = np.zeros((m, d))
    n[:, 0] = np.arange(1, m + 1)
    return n


KSETS = {
    "grid": lambda d: _ball(d, 14 if d == 2 else 6),            # roots formed in the passes
    "grid roots": lambda d: _ball(d, 60 if d == 2 else 13),     # many blocks: from the roots kernel
    "lines": lambda d: _lines(d, 4 if d == 2 else 3, 150.0),
    "few rows": lambda d: _ball(d, 2),                          # recurrences
    "one axis": lambda d: _axis(d, 400),
}


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("d", [2, 3])
@pytest.mark.parametrize("form", list(KSETS))
def test_every_row_is_nan(form, d, value):
    nv = KSETS[form](d)
    n = 70
    en = StealthyEnergy(nv, np.ones(len(nv)), np.float64(n))
    good = np.random.default_rng(len(nv)).uniform(size=(d + 1, n, d))
    s = good.copy()
    for a in range(d):
        s[a, 11 * a + 3, a] = value   # lane a: coordinate a of one particle
    phi, grad, re, im = en.evaluate(s, want_rho=True)
    ref = en.evaluate(good, want_rho=True)
    assert np.isnan(phi[:d]).all() and np.isnan(grad[:d]).all()
    assert np.isnan(re[:d]).all() and np.isnan(im[:d]).all()
    for x, y in zip((phi, grad, re, im), ref):
        assert np.array_equal(x[d], y[d])
    assert np.isnan(en.evaluate(s, want_grad=False)[0][:d]).all()


@pytest.mark.parametrize("d", [2, 3])
def test_small_descents_see_it(d):
    nv = _axis(d, 6)
    en = StealthyEnergy(nv, np.ones(6), np.float64(30.0))
    s = np.random.default_rng(d).uniform(size=(2, 30, d))
    s[0, 5, d - 1] = np.nan
    res = relax(en, s, DescentSettings(max_evals=20))
    assert np.isnan(res.energy[0]) and np.isfinite(res.energy[1])
