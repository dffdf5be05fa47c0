"""Descent lanes that run altogether in shared memory (k_persist_compact) against
the oracle's descent, at the sizes where its loops have edges: one and many
particles (below and above its threads, not multiples of a warp), one row and
more rows than four per warp, rows of both signs, and a problem whose phases no
longer fit beside its tables. Iterates 1e-14 on the torus per iteration that both
take (the package's own descent tolerance, times the few iterations run)."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from conftest import ATOL_DESCENT_ITERATE, RTOL_VMAP_E
from xla_cco.energy import StealthyEnergy
from xla_cco.minimize import relax, relax_device
from xla_cco.minimize.descent import DescentSettings

pytestmark = pytest.mark.gpu


def _rows(d, m, r):
    """m distinct integer rows of one half space, components within +-r."""
    g = np.stack(np.meshgrid(*([np.arange(-r, r + 1)] * d), indexing="ij"), axis=-1).reshape(-1, d)
    first = np.zeros(len(g), dtype=np.int64)
    for a in range(d):
        first = np.where(first == 0, np.sign(g[:, a]), first)
    g = g[first > 0]
    g = g[np.argsort((g * g).sum(1), kind="stable")][:m]
    assert len(g) == m
    sign = np.where(np.arange(m) % 3 == 1, -1, 1)      # any one of k, -k
    return g * sign[:, None]


CASES = [(1, 2, 1, 3), (1, 33, 20, 4), (1, 300, 30, 2), (1, 700, 3, 2), (2, 31, 5, 3), (2, 64, 70, 2),
         (2, 130, 13, 3), (2, 600, 19, 2),
         (3, 2, 4, 2), (3, 97, 65, 2), (3, 257, 14, 2)]  # fmt: skip


@pytest.mark.parametrize("d,n,m,b", CASES)
def test_compact_descent_vs_oracle(d, n, m, b):
    nv = _rows(d, m, {1: 40, 2: 9, 3: 4}[d])
    rng = np.random.default_rng(100 * d + n)
    w = rng.uniform(0.5, 1.5, size=m)
    s0 = rng.uniform(size=(b, n, d))
    vol = 2.0 * n
    en = StealthyEnergy(nv.astype(np.float64), w, np.float64(vol))
    cfg = DescentSettings(max_evals=21, step_init=1e-3 / np.sqrt(n), record_every=2, max_records=4)
    out = relax(en, s0, cfg)
    assert relax_device(en, _cuda(s0), cfg)["ticks"] == 0
    ref = oracle.relax_batch("descent", s0, nv, w, vol, cfg)
    for f in ("n_iters", "n_evals", "status"):
        np.testing.assert_array_equal(getattr(out, f), ref[f], err_msg=f)
    np.testing.assert_allclose(out.energy, ref["energy"], rtol=RTOL_VMAP_E)
    dev = out.s - ref["s"]
    assert np.max(np.abs(dev - np.round(dev))) <= ATOL_DESCENT_ITERATE * max(1, int(np.max(ref["n_iters"])))
    one = relax(en, s0[:1], cfg)                        # alone and in a batch: the same bits
    np.testing.assert_array_equal(one.s[0], out.s[0])


def _cuda(x):
    import torch

    return torch.from_numpy(x).cuda()
