"""The serving pool counts the ticks that ran, not those its launches may run: a
launch is a loop that ends with the last running lane, and those queued behind it
run none."""

from __future__ import annotations

import numpy as np
import pytest

from xla_cco.box import cubic_box
from xla_cco.energy import make_stealthy_energy
from xla_cco.kvectors import enumerate_kvectors, k_outer_from_ka, ka_from_chi
from xla_cco.minimize.lbfgs import LBFGSSettings
from xla_cco.serve import RelaxServer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph_ticks", [8, 64, 256])
def test_ticks_are_those_that_ran(graph_ticks):
    n, d = 200, 2
    box = cubic_box(n, d)
    ks = enumerate_kvectors(box.basis, 0.0, k_outer_from_ka(ka_from_chi(0.3, 0.05, d), 0.05, d))
    en = make_stealthy_energy(box, ks)
    rng = np.random.default_rng(6)
    total = 0
    st = LBFGSSettings(energy_tol=1e-30, rescales=(1e4,), max_evals_per_pass=20)
    with RelaxServer(st, graph_ticks=graph_ticks) as srv:
        for _ in range(3):   # one after the other: a plan each
            res = srv.result(srv.submit(en, rng.uniform(size=(n, d))))
            total += res.n_evals
        ticks = srv.stats().ticks
    # a loop body holds at most 64 ticks of so small a lane (0.6 ms of kernels)
    assert total <= ticks <= total + 3 * min(graph_ticks, 64)
