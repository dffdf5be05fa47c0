"""A captured density call replays after its k-set has left the cache."""

from __future__ import annotations

import gc

import numpy as np
import pytest

from xla_cco import energy

pytestmark = pytest.mark.gpu


def test_captured_density_outlives_the_cache(monkeypatch):
    import torch

    rng = np.random.default_rng(8)
    nv = rng.permutation(np.array([(a, b) for a in range(1, 9) for b in range(-6, 7)], dtype=np.float64))
    s = torch.from_numpy(rng.uniform(size=(90, 2))).cuda()
    energy.collective_density(s, nv)   # the problem is built outside the capture
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        re, im = energy.collective_density(s, nv)
    monkeypatch.setattr(energy, "_DENSITY_SETS", 1)
    for i in range(3):   # push it out, and give its memory to others if it was free
        energy.collective_density(s, nv[: 50 + i])
    gc.collect()
    fresh = torch.from_numpy(rng.uniform(size=(90, 2))).cuda()
    s.copy_(fresh)
    graph.replay()
    torch.cuda.synchronize()
    theta = 2.0 * np.pi * (nv @ fresh.cpu().numpy().T)
    np.testing.assert_allclose(re.cpu().numpy(), np.cos(theta).sum(1), rtol=0, atol=1e-12 * 90)
    np.testing.assert_allclose(im.cpu().numpy(), np.sin(theta).sum(1), rtol=0, atol=1e-12 * 90)
