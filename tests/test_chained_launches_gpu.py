"""Evaluations whose kernels are launched as a chain: they see the positions that
the kernel before them on the stream has just written, and the next writer does
not overtake them - directly, in both forms of the passes, on two streams at
once, and replayed from a captured graph. The same bits as with a synchronisation
around each."""

from __future__ import annotations

import numpy as np
import pytest

from xla_cco.box import cubic_box
from xla_cco.energy import make_stealthy_energy
from xla_cco.kvectors import enumerate_kvectors, k_outer_from_ka, ka_from_chi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,n,b", [(1, 900, 2), (2, 40, 1), (2, 600, 24), (3, 300, 3)])
@pytest.mark.parametrize("form", ["grid", "recurrence"])
def test_chained_evaluations_are_ordered(monkeypatch, d, n, b, form):
    import torch

    if form == "recurrence":
        monkeypatch.setenv("CCO_PASS1_GEMM", "0")
    box = cubic_box(n, d)
    en = make_stealthy_energy(box, enumerate_kvectors(box.basis, 0.0, k_outer_from_ka(ka_from_chi(0.3, 0.05, d), 0.05, d)))
    base = torch.from_numpy(np.random.default_rng(n).uniform(size=(b, n, d))).cuda()
    want = []
    for i in range(8):
        s = base + 0.01 * i
        torch.cuda.synchronize()
        want.append([x.clone() for x in en.evaluate(s)[:2]])
        torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    bufs = [torch.empty_like(base) for _ in streams]
    got = [[], []]
    torch.cuda.synchronize()
    for i in range(8):
        for q, st in enumerate(streams):
            with torch.cuda.stream(st):
                torch.add(base, 0.01 * i, out=bufs[q])      # overwritten again right after the call
                got[q].append(en.evaluate(bufs[q])[:2])
    torch.cuda.synchronize()
    for q in range(2):
        for (e, g), (we, wg) in zip(got[q], want):
            assert torch.equal(e, we) and torch.equal(g, wg)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        torch.add(bufs[0], 0.0, out=bufs[1])
        out = en.evaluate(bufs[1])[:2]
    for i in (3, 6):
        bufs[0].copy_(base + 0.01 * i)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out[0], want[i][0]) and torch.equal(out[1], want[i][1])
