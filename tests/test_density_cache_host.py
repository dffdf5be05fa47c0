"""Energies kept for density calls (no device): programs that cycle through many
k-sets find them again, and what is kept is bounded."""

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
