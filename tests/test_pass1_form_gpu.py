"""cco_problem_pass1_form names no form that does not run: a k-set that gives the
bits of the recurrence kernels reports 0, also one dense enough by its rows but too
small for the padded grid."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest

from xla_cco import _native
from xla_cco.box import Box
from xla_cco.energy import make_stealthy_energy
from xla_cco.kvectors import enumerate_kvectors, k_outer_from_ka, ka_from_chi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,chi,aspect,grid", [(1187, 0.02, 6.0, False), (607, 0.05, 6.0, False),
                                               (1000, 0.40, 1.0, True), (400, 0.30, 6.0, True)])  # fmt: skip
def test_the_reported_form_is_the_one_that_runs(monkeypatch, n, chi, aspect, grid):
    basis = np.sqrt(n) * np.diag([1.0 / np.sqrt(aspect), np.sqrt(aspect)])
    ks = enumerate_kvectors(basis, 0.0, k_outer_from_ka(ka_from_chi(chi, 0.05, 2), 0.05, 2))
    s = np.random.default_rng(n).uniform(size=(2, n, 2))
    out, blocks = {}, {}
    for form in ("default", "recurrence"):
        if form == "recurrence":
            monkeypatch.setenv("CCO_PASS1_GEMM", "0")
        en = make_stealthy_energy(Box(basis), ks)
        got = ctypes.c_int(-1)
        _native.check(_native.load().cco_problem_pass1_form(en.problem_handle(0, n), ctypes.byref(got)), "form")
        blocks[form] = got.value
        out[form] = en.evaluate(s)
    same = np.array_equal(out["default"][1], out["recurrence"][1])
    assert same == (not grid)   # what runs
    assert blocks["recurrence"] == 0 and (blocks["default"] > 0) == grid
