"""Mixed lanes whose dimensions run as parallel nodes of the tick graph (1.5 GFLOP
a tick and more) and in order (less) give the bits of lone runs."""

from __future__ import annotations

import numpy as np
import pytest

from xla_cco.box import cubic_box
from xla_cco.energy import make_stealthy_energy
from xla_cco.kvectors import enumerate_kvectors, k_outer_from_ka, ka_from_chi
from xla_cco.minimize import relax, relax_mixed
from xla_cco.minimize.lbfgs import LBFGSSettings

pytestmark = pytest.mark.gpu


def _lane(n, d, chi, seed):
    box = cubic_box(n, d)
    en = make_stealthy_energy(box, enumerate_kvectors(box.basis, 0.0, k_outer_from_ka(ka_from_chi(chi, 0.05, d), 0.05, d)))
    return en, np.random.default_rng(seed).uniform(size=(n, d))


SMALL = [(300, 1, 0.3), (120, 2, 0.4), (90, 3, 0.2), (400, 2, 0.1)]
LARGE = [(4000, 3, 0.4), (5000, 2, 0.45), (4200, 3, 0.45), (3000, 1, 0.4), (60, 2, 0.3)]


@pytest.mark.parametrize("lanes", [SMALL, LARGE], ids=["in_order", "forked"])
def test_mixed_dimensions_equal_lone_runs(lanes):
    inst = [_lane(*x, seed=i) for i, x in enumerate(lanes)]
    st = LBFGSSettings(energy_tol=1e-20, rescales=(1e4,), max_evals_per_pass=7)
    res = relax_mixed([e for e, _ in inst], [s for _, s in inst], st)
    for i, ((en, s0), r) in enumerate(zip(inst, res)):
        alone = relax(en, s0[None], st)
        for f in ("s", "energy", "grad_norm", "n_evals", "n_iters", "status"):
            assert np.array_equal(np.asarray(getattr(r, f)), np.asarray(getattr(alone, f))), (i, f)
