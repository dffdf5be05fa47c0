"""The tensor-core grid form of the FP64 evaluation (cco_grid.cuh) against the
accurate oracle and against the phase-recurrence kernels of the same problem
(built with CCO_PASS1_GEMM=0), at the sizes where its tiling has edges: particle
counts around its tiles, ragged strips, several blocks, 1-D k-sets with holes
and negative rows, annuli, uneven weights. Energies 1e-12 relative, forces
1e-12 of max |F| (the package's own kernel tolerances)."""

from __future__ import annotations

import numpy as np
import pytest

import oracle
from conftest import RTOL_KERNEL_E, RTOL_KERNEL_F
from xla_cco import _native
from xla_cco.box import cubic_box
from xla_cco.energy import StealthyEnergy, make_stealthy_energy
from xla_cco.kvectors import enumerate_kvectors, k_outer_from_ka, ka_from_chi

pytestmark = pytest.mark.gpu


def _kset(kind, d):
    """Integer rows (M, d) of one half space."""
    if kind == "holes":     # 1-D: two runs below and above zero, one row missing in every 97
        n = [x for x in range(-260, -40)] + [x for x in range(300, 900) if x % 97]
        return np.array(n, dtype=np.int64)[:, None]
    r_out, r_in = {"disc": (9.3, 0.0), "wide": (52.6, 0.0), "annulus": (14.2, 7.7), "small": (3.2, 0.0)}[kind]
    r = int(r_out) + 1
    g = np.stack(np.meshgrid(*([np.arange(-r, r + 1)] * d), indexing="ij"), axis=-1).reshape(-1, d)
    first = np.zeros(len(g), dtype=np.int64)
    for a in range(d):
        first = np.where(first == 0, np.sign(g[:, a]), first)
    q = (g * g).sum(1)
    return g[(first > 0) & (q < r_out**2) & (q > r_in**2)]


CASES = [(1, "holes", 257, 2), (1, "wide", 64, 3), (2, "small", 65, 3), (2, "disc", 3, 2),
         (2, "disc", 63, 2), (2, "annulus", 128, 2), (2, "wide", 129, 1), (3, "small", 33, 2),
         (3, "disc", 127, 2), (3, "annulus", 66, 1), (2, "disc", 2049, 1), (3, "small", 8193, 1)]  # fmt: skip


@pytest.mark.parametrize("d,kind,n,b", CASES)
def test_grid_and_recurrence_forms_vs_oracle(monkeypatch, d, kind, n, b):
    nv = _kset(kind, d)
    rng = np.random.default_rng(1000 * d + n)
    w = rng.uniform(0.2, 2.0, size=len(nv))
    w[rng.integers(0, len(nv), size=2)] = 0.0
    s = rng.uniform(size=(b, n, d))
    s[0, 0] = 0.0                                   # a particle at the origin
    vol = 3.0 * n
    out = {}
    for form in ("grid", "recurrence"):
        if form == "recurrence":
            monkeypatch.setenv("CCO_PASS1_GEMM", "0")
        en = StealthyEnergy(nv.astype(np.float64), w, np.float64(vol))   # a fresh problem reads the switch
        out[form] = en.evaluate(s, want_rho=True)
    e_ref, g_ref = oracle.energy_grad_accurate(s, nv, w, vol)
    for form, (phi, g, re, im) in out.items():
        np.testing.assert_allclose(phi, e_ref, rtol=RTOL_KERNEL_E, atol=0, err_msg=form)
        for i in range(b):
            np.testing.assert_allclose(g[i], g_ref[i], rtol=0, atol=RTOL_KERNEL_F * np.abs(g_ref[i]).max(),
                                       err_msg=form)  # fmt: skip
        # rho in the caller's row order: N terms of modulus 1
        theta = 2.0 * np.pi * (nv.astype(np.float64) @ s[0].T % 1.0)
        np.testing.assert_allclose(re[0], np.cos(theta).sum(1), rtol=0, atol=1e-12 * n)
        np.testing.assert_allclose(im[0], np.sin(theta).sum(1), rtol=0, atol=1e-12 * n)


def test_a_lane_alone_and_in_a_batch_has_the_same_bits():
    n, d = 333, 2
    box = cubic_box(n, d)
    ks = enumerate_kvectors(box.basis, 0.0, k_outer_from_ka(ka_from_chi(0.3, 0.05, d), 0.05, d))
    en = make_stealthy_energy(box, ks)
    s = np.random.default_rng(3).uniform(size=(37, n, d))
    phi, g, _, _ = en.evaluate(s)
    for i in (0, 17, 36):
        p1, g1, _, _ = en.evaluate(s[i:i + 1])
        assert p1[0] == phi[i] and np.array_equal(g1[0], g[i])


def test_noalloc_batch_larger_than_the_scratch_in_grid_layout():
    """A batch the fixed scratch admits, whose padded grid layout needs more: it
    runs in parts and gives the bits of the allocating call."""
    import torch

    n, d = 60, 2
    box = cubic_box(n, d)
    ks = enumerate_kvectors(box.basis, 0.0, k_outer_from_ka(ka_from_chi(0.35, 0.05, d), 0.05, d))
    en = make_stealthy_energy(box, ks)
    h = en.problem_handle(torch.cuda.current_device(), n)
    m = ks.n.shape[0]
    b = (16 << 20) * 9 // 10 // (48 * m + 120)
    s = torch.from_numpy(np.random.default_rng(4).uniform(size=(b, n, d))).cuda()
    phi = torch.full((b,), float("nan"), dtype=torch.float64, device="cuda")
    g = torch.full_like(s, float("nan"))
    stream = torch.cuda.current_stream().cuda_stream
    code = _native.load().cco_energy_grad_noalloc(h, stream, b, s.data_ptr(), phi.data_ptr(), g.data_ptr())
    assert code == _native.CCO_OK, _native.load().cco_last_error()
    p_ref, g_ref, _, _ = en.evaluate(s)
    assert torch.equal(phi, p_ref) and torch.equal(g, g_ref)


@pytest.mark.parametrize("d,n,b,dirs,top", [(2, 65, 2, 5.3, 130), (2, 300, 1, 9.1, 700), (3, 129, 2, 3.2, 90),
                                            (2, 1, 1, 5.3, 60)])  # fmt: skip
def test_line_grid_density_vs_direct_sums(monkeypatch, d, n, b, dirs, top):
    """K-sets of multiples of primitive vectors (the structure factor's): rows with
    gaps, lines through both half spaces, uneven weights; density, energy and the
    gradient (whose pass keeps the recurrences) in both forms."""
    r = int(dirs) + 1
    g = np.stack(np.meshgrid(*([np.arange(-r, r + 1)] * d), indexing="ij"), axis=-1).reshape(-1, d)
    g = g[(np.gcd.reduce(np.abs(g), axis=1) == 1) & ((g * g).sum(1) < dirs**2)]
    first = np.array([x[np.flatnonzero(x)[0]] for x in g])
    g = g[first > 0]
    rows = [i * v for v in g for i in range(1, int(top / np.sqrt(v @ v)) + 1) if i % 13 != 5]
    rows += [-3 * v for v in g[::2]]
    nv = np.array(rows, dtype=np.int64)
    rng = np.random.default_rng(n)
    w = rng.uniform(0.1, 1.0, size=len(nv))
    s = rng.uniform(size=(b, n, d))
    out = {}
    for form in ("lines", "recurrence"):
        if form == "recurrence":
            monkeypatch.setenv("CCO_PASS1_GEMM", "0")
        en = StealthyEnergy(nv.astype(np.float64), w, np.float64(2.0 * n))
        out[form] = en.evaluate(s, want_rho=True)
        out[form + " density"] = en.evaluate(s, want_grad=False, want_rho=True)
    e_ref, g_ref = oracle.energy_grad_accurate(s, nv, w, 2.0 * n)
    hi = np.round(s * 2.0**26) / 2.0**26   # n hi exact: its whole part leaves before rounding
    for i in range(b):
        t = nv @ hi[i].T
        theta = 2.0 * np.pi * ((t - np.round(t)) + nv @ (s[i] - hi[i]).T)
        for form, (phi, grad, re, im) in out.items():
            np.testing.assert_allclose(phi[i], e_ref[i], rtol=RTOL_KERNEL_E, atol=0, err_msg=form)
            np.testing.assert_allclose(re[i], np.cos(theta).sum(1), rtol=0, atol=1e-13 * n, err_msg=form)
            np.testing.assert_allclose(im[i], np.sin(theta).sum(1), rtol=0, atol=1e-13 * n, err_msg=form)
            if grad is not None and n > 1:
                np.testing.assert_allclose(grad[i], g_ref[i], rtol=0, atol=RTOL_KERNEL_F * np.abs(g_ref[i]).max())


def test_density_layout_with_zero_rows_inside():
    """Zero (padding) rows anywhere: N and 0 there, every other row in place; the
    same from NumPy and CUDA inputs, and structure-factor sums in the same order."""
    import torch

    from xla_cco.analysis.structure import structure_factor

    nv = np.array([[0, 0], [1, 0], [0, 2], [0, 0], [3, -1], [-2, 5], [0, 0]], dtype=np.float64)
    en = StealthyEnergy(nv, np.where(nv.any(1), 1.0, 0.0), np.float64(5.0))
    s = np.random.default_rng(9).uniform(size=(3, 41, 2))
    _, _, re, im = en.evaluate(s, want_rho=True)
    theta = 2.0 * np.pi * np.einsum("ka,bja->bkj", nv, s)
    np.testing.assert_allclose(re, np.cos(theta).sum(-1), rtol=0, atol=1e-12 * 41)
    np.testing.assert_allclose(im, np.sin(theta).sum(-1), rtol=0, atol=1e-12 * 41)
    assert (re[:, [0, 3, 6]] == 41.0).all() and (im[:, [0, 3, 6]] == 0.0).all()
    _, _, rt, it = en.evaluate(torch.from_numpy(s).cuda(), want_rho=True)
    assert np.array_equal(rt.cpu().numpy(), re) and np.array_equal(it.cpu().numpy(), im)
    sk = structure_factor(s[1], nv)
    np.testing.assert_allclose(sk, (re[1] ** 2 + im[1] ** 2) / 41, rtol=1e-13)
