"""The tick schedule of a shape class is chosen from ticks that ran: runs that end
before or inside the trials keep the default schedule and leave none behind, and
the reported ticks are those that ran."""

from __future__ import annotations

import numpy as np
import pytest

from xla_cco import _native
from xla_cco.box import cubic_box
from xla_cco.dynamics import MDSettings, init_state, make_key, make_waves, simulate
from xla_cco.energy import make_stealthy_energy
from xla_cco.kvectors import enumerate_kvectors, k_outer_from_ka, ka_from_chi
from xla_cco.minimize import relax_device
from xla_cco.minimize.descent import DescentSettings

pytestmark = pytest.mark.gpu

DEFAULT = (1, 16)   # branches and ticks of a launch of so small a tick
BODY = 16           # a run ends at most one loop body late


@pytest.fixture(autouse=True)
def _fresh(monkeypatch):
    for name in ("CCO_BRANCHES", "CCO_GRAPH_TICKS", "CCO_OVERLAP", "CCO_AUTOTUNE", "CCO_INFLIGHT"):
        monkeypatch.delenv(name, raising=False)
    _native.load().cco_schedule_reset()
    yield
    _native.load().cco_schedule_reset()


def _system(n, d, chi, b):
    import torch

    box = cubic_box(n, d)
    ks = enumerate_kvectors(box.basis, 0.0, k_outer_from_ka(ka_from_chi(chi, 0.05, d), 0.05, d))
    s0 = torch.from_numpy(np.random.default_rng(n + b).uniform(size=(b, n, d))).cuda()
    return box, make_stealthy_energy(box, ks), s0


@pytest.mark.parametrize("evals", [2, 40, 240, 270, 300, 310])
def test_short_runs_neither_choose_nor_leave_a_schedule(evals):
    """Runs that end at once, inside the first trials of an immediate tuning, and
    shortly before and after the tick from which a table is tuned."""
    _, en, s0 = _system(500, 2, 0.3, 64)
    for _ in range(2):
        out = relax_device(en, s0, DescentSettings(max_evals=evals, step_min=0.0, energy_tol=0.0))
        most = int(out["n_iters"].max()) + 1
        assert most == evals // 2 + 1
        assert out["schedule"] == DEFAULT
        assert most <= out["ticks"] < most + BODY


def test_a_long_run_tunes_its_class_and_counts_its_ticks():
    import torch

    _, en, s0 = _system(500, 2, 0.3, 64)
    st = DescentSettings(max_evals=1600, step_min=0.0, energy_tol=0.0)
    first = relax_device(en, s0, st)
    most = int(first["n_iters"].max()) + 1
    assert first["schedule"] == DEFAULT and most <= first["ticks"] < most + 2 * BODY
    second = relax_device(en, s0, st)   # on the chosen schedule
    branches, ticks = second["schedule"]
    assert branches in (1, 2, 3, 4, 6, 8) and 4 <= ticks <= 32
    assert most <= second["ticks"] < most + 2 * BODY
    for k in ("s", "energy", "n_evals", "n_iters", "status"):
        assert torch.equal(first[k], second[k]), k


def test_md_segments_count_the_ticks_that_ran(monkeypatch):
    """Of no steps (the initial state's) and of 40."""
    n, d, b = 200, 2, 64
    box, en, _ = _system(n, d, 0.3, b)
    seen = []
    lib = _native.load()

    class Recorder:
        def __getattr__(self, name):
            return getattr(lib, name)

        def cco_md_segment(self, *args):
            code = lib.cco_md_segment(*args)
            seen.append(args[-1]._obj.value)
            return code

    rng = np.random.default_rng(4)
    k = k_outer_from_ka(ka_from_chi(0.3, 0.05, d), 0.05, d)
    waves = make_waves(box.basis, k, 1.1 * k)
    keys = np.stack([make_key(i) for i in range(b)])
    st = MDSettings(dt=0.01, chunk_steps=40, drift_tol=np.inf)
    monkeypatch.setattr(_native, "load", lambda: Recorder())
    r0 = rng.uniform(size=(b, n, d)) * box.basis[0, 0]
    state = init_state(en, waves, box.basis, r0, rng.normal(size=(b, n, d)), np.full(b, 0.5), keys, st)
    simulate(en, waves, box.basis, st, state, 40)
    assert seen[0] >= 1 and seen[0] < 1 + BODY
    assert 41 <= seen[1] < 41 + BODY


def test_md_of_many_steps_is_tuned_before_its_first_step(monkeypatch):
    """A segment that lasts as long as the trials counts its own ticks and no others,
    in the call that tunes and in the next."""
    n, d, b = 60, 2, 64
    box, en, _ = _system(n, d, 0.3, b)
    seen = []
    lib = _native.load()

    class Recorder:
        def __getattr__(self, name):
            return getattr(lib, name)

        def cco_md_segment(self, *args):
            code = lib.cco_md_segment(*args)
            seen.append(args[-1]._obj.value)
            return code

    rng = np.random.default_rng(5)
    k = k_outer_from_ka(ka_from_chi(0.3, 0.05, d), 0.05, d)
    waves = make_waves(box.basis, k, 1.1 * k)
    keys = np.stack([make_key(i) for i in range(b)])
    st = MDSettings(dt=0.01, scheme="baoab", gamma=1.0, chunk_steps=400, drift_tol=np.inf)
    r0 = rng.uniform(size=(b, n, d)) * box.basis[0, 0]
    state = init_state(en, waves, box.basis, r0, rng.normal(size=(b, n, d)), np.full(b, 0.5), keys, st)
    monkeypatch.setattr(_native, "load", lambda: Recorder())
    one = simulate(en, waves, box.basis, st, state, 400).state
    two = simulate(en, waves, box.basis, st, state, 400).state
    assert all(401 <= x < 401 + 2 * BODY for x in seen), seen
    assert np.array_equal(one.r, two.r) and np.array_equal(one.v, two.v)
