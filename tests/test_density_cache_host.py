"""Energies kept for density calls (no device): programs that cycle through many
k-sets find them again, what is kept is bounded, and one that a captured stream has
used is never destroyed under the graph."""

from __future__ import annotations

import gc
import weakref

import numpy as np
import pytest

from xla_cco import energy


@pytest.fixture(autouse=True)
def _empty():
    saved = energy._DENSITY_CACHE.copy()
    energy._DENSITY_CACHE.clear()
    yield
    energy._DENSITY_CACHE.clear()
    if isinstance(saved, dict):
        energy._DENSITY_CACHE.update(saved)
    else:
        energy._DENSITY_CACHE.extend(saved)


def _sets(count, rows=7):
    return [np.arange(2 * rows, dtype=np.float64).reshape(rows, 2) + i for i in range(count)]


def test_a_cycle_of_many_sets_finds_every_one_again():
    sets = _sets(300)
    first = [energy._density_energy(nv) for nv in sets]
    assert all(energy._density_energy(nv.copy()) is en for nv, en in zip(sets, first))


def test_sets_that_share_the_sampled_entries_are_told_apart():
    a = np.arange(4000, dtype=np.float64).reshape(2000, 2)
    b = a.copy()
    b[1, 1] = -5.0
    ea, eb = energy._density_energy(a), energy._density_energy(b)
    assert ea is not eb and energy._density_energy(a) is ea and energy._density_energy(b) is eb
    a[3, 0] = 99.0   # the caller's array is its own
    assert energy._density_energy(a) is not ea


def test_what_is_kept_is_bounded(monkeypatch):
    monkeypatch.setattr(energy, "_DENSITY_ROWS", 50, raising=False)
    refs = [weakref.ref(energy._density_energy(nv)) for nv in _sets(400)]
    gc.collect()
    assert sum(r() is not None for r in refs) <= 64
    monkeypatch.setattr(energy, "_DENSITY_SETS", 3, raising=False)
    energy._density_energy(_sets(401)[-1])
    gc.collect()
    assert sum(r() is not None for r in refs) <= 64


def test_a_set_used_under_capture_outlives_its_place_in_the_cache(monkeypatch):
    import torch

    class OnDevice(np.ndarray):   # an input that says it is a CUDA tensor
        is_cuda = True

    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
    monkeypatch.setattr(energy, "require_float64", lambda *a: None)
    seen = []

    def evaluate(self, s, want_grad=True, want_rho=False):
        seen.append(weakref.ref(self))
        return None, None, np.zeros((1, 7)), np.zeros((1, 7))

    monkeypatch.setattr(energy.StealthyEnergy, "evaluate", evaluate)
    nv = _sets(1)[0]
    energy.collective_density(np.zeros((5, 2)).view(OnDevice), nv)
    monkeypatch.setattr(energy, "_DENSITY_SETS", 8, raising=False)
    for other in _sets(200)[1:]:
        energy._density_energy(other)
    gc.collect()
    assert seen[0]() is not None
