"""cco_energy_grad_noalloc on batches that run in uneven parts.

A k-set of multiples of a few directions takes the line grid in the density
pass and keeps the recurrences in the gradient pass, whose items per lane
depend on how many threads share a particle. The fixed scratch is laid out for
the largest part; a shorter last part must use the same layout.
"""

from __future__ import annotations

import math

import numpy as np
import pytest

from xla_cco import _native
from xla_cco.energy import StealthyEnergy

pytestmark = pytest.mark.gpu

SCRATCH = 16 << 20   # CCO_NOALLOC_SCRATCH_BYTES


def _line_kset(directions: int, multiples: int) -> np.ndarray:
    """The multiples 1..`multiples` of the first primitive (a, b) with a >= 1."""
    v = [(a, b) for a in range(1, 12) for b in range(-3, 12) if math.gcd(a, abs(b)) == 1]
    rows = {(a * i, b * i) for a, b in v[:directions] for i in range(1, multiples + 1)}
    return np.array(sorted(rows), dtype=np.float64)


@pytest.mark.parametrize(
    "batch",
    [
        886,   # two equal parts
        887,   # 444 lanes, one thread a particle, then 443, where alone two threads would share one
        700,   # smaller parts
        600,   # one part
    ],
)
def test_line_grid_batch_in_uneven_parts_has_the_bits_of_the_allocating_call(batch):
    import torch

    n, d = 128, 2
    nv = _line_kset(15, 17)
    m = len(nv)
    assert m == 255
    # what the entry point accepts: rho, w rho and two rows of partials per lane, and some items
    assert 64 * m * batch < SCRATCH * 9 // 10
    rng = np.random.default_rng(batch)
    en = StealthyEnergy(nv, rng.uniform(0.1, 1.0, size=m), np.float64(2.0 * n))
    handle = en.problem_handle(torch.cuda.current_device(), n)
    s = torch.from_numpy(rng.uniform(size=(batch, n, d))).cuda()
    phi = torch.full((batch,), float("nan"), dtype=torch.float64, device="cuda")
    grad = torch.full_like(s, float("nan"))
    stream = torch.cuda.current_stream().cuda_stream
    code = _native.load().cco_energy_grad_noalloc(handle, stream, batch, s.data_ptr(), phi.data_ptr(),
                                                  grad.data_ptr())  # fmt: skip
    assert code == _native.CCO_OK, _native.load().cco_last_error()
    phi_ref, grad_ref, _, _ = en.evaluate(s)
    assert torch.equal(phi, phi_ref) and torch.equal(grad, grad_ref)
