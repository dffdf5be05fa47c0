"""Ticks run as a loop on the device that ends with the last lane: graphs of any
length give the same bits, and no more ticks run than the longest lane needs,
up to one loop body past it."""

from __future__ import annotations

import numpy as np
import pytest

from xla_cco.box import cubic_box
from xla_cco.energy import make_stealthy_energy
from xla_cco.kvectors import enumerate_kvectors
from xla_cco.minimize import relax_device
from xla_cco.minimize.lbfgs import LBFGSSettings

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("compact", [0, 1])
@pytest.mark.parametrize("graph_ticks", [1, 2, 7, 16, 30])
def test_loop_lengths_give_the_same_bits(monkeypatch, graph_ticks, compact):
    import torch

    box = cubic_box(40, 2)
    en = make_stealthy_energy(box, enumerate_kvectors(box.basis, 0.0, 4.0))
    s0 = torch.from_numpy(np.random.default_rng(3).uniform(size=(9, 40, 2))).cuda()
    cfg = LBFGSSettings(energy_tol=1e-18, max_evals_per_pass=45)
    monkeypatch.setenv("CCO_COMPACT", "0")
    monkeypatch.setenv("CCO_GRAPH_TICKS", "3")
    ref = relax_device(en, s0, cfg)
    monkeypatch.setenv("CCO_COMPACT", str(compact))
    monkeypatch.setenv("CCO_GRAPH_TICKS", str(graph_ticks))
    out = relax_device(en, s0, cfg)
    for k in ("s", "energy", "grad_norm", "n_evals", "n_iters", "status"):
        assert torch.equal(out[k], ref[k]), k
    most = int(out["n_evals"].max())
    assert most <= out["ticks"] < most + 2 + graph_ticks
    assert out["launches"] >= 7 * out["ticks"]
