"""Small descents of more lanes than SMs run with fewer threads a lane: the same bits as
each lane alone, at sizes where a CTA's 512, 256 and 128 threads are chosen, lanes of
one and of several particles a thread, and faster than in rounds of one lane per SM."""

from __future__ import annotations

import time

import numpy as np
import pytest

from xla_cco.minimize import DescentSettings, relax_device
from xla_cco.workloads import energy_for

pytestmark = pytest.mark.gpu


def _lanes(n, d, chi, b):
    import torch

    return energy_for(n, d, chi), torch.from_numpy(np.random.default_rng(n + b).uniform(size=(b, n, d))).cuda()


@pytest.mark.parametrize("n,d,chi", [(20, 1, 0.3), (60, 1, 0.3), (150, 1, 0.3), (20, 2, 0.4), (120, 2, 0.1),
                                     (300, 2, 0.05), (60, 3, 0.05), (200, 3, 0.05)])  # fmt: skip
@pytest.mark.parametrize("lanes", [149, 300, 700])
def test_lanes_keep_their_bits(n, d, chi, lanes):
    import torch

    en, s = _lanes(n, d, chi, lanes)
    st = DescentSettings(max_evals=40)
    out = relax_device(en, s, st)
    for i in (0, lanes // 2, lanes - 1):
        one = relax_device(en, s[i:i + 1].contiguous(), st)
        for k in ("s", "energy", "grad_norm", "n_evals", "n_iters", "status"):
            assert torch.equal(out[k][i], one[k][0]), (i, k)


def test_many_lanes_share_the_sms():
    import torch

    st = DescentSettings(max_evals=100)
    best = {}
    for lanes in (148, 1480):
        en, s = _lanes(60, 1, 0.3, lanes)
        for _ in range(10):
            torch.cuda.synchronize()
            t = time.perf_counter()
            relax_device(en, s, st)
            torch.cuda.synchronize()
            best[lanes] = min(best.get(lanes, 1e9), time.perf_counter() - t)
    assert best[1480] < 5.0 * best[148], best   # ten rounds of one lane per SM took 7 times as long
