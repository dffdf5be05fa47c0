"""Performance cases of the collective-coordinate path, through the public API.

``listed()`` names the cases, ``draw(rng)`` gives another one of the same
ranges, ``prepare(case, seed)`` builds what a program holds before the call
(the energy of its system and seeded positions on the GPU), ``run(state)`` is
one call, ``work(case)`` the bytes and operations the call cannot do without,
and ``exact(case, seed)`` the same outputs in plain float64 torch / numpy.

The systems follow the package's own conventions: unit density, packing
fraction 0.05, k-set from chi, uniform random fractional positions. Sizes are
those of the benchmark and its seeded ensembles (``xla_cco.workloads``): N from
100 to 20 000, d = 1..3, chi from 0.05 to 0.49, one lane to 256.
"""

from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

_PKG = str(Path(__file__).resolve().parents[1] / "xla-cco_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from xla_cco import (  # noqa: E402
    DescentSettings,
    LBFGSSettings,
    cubic_box,
    isotropic_structure_factor,
    k_outer_from_ka,
    ka_from_chi,
    pair_distance_histogram,
    relax,
    relax_mixed,
)
from xla_cco.analysis.pairs import nearest_neighbor_distances_batch  # noqa: E402
from xla_cco.dynamics import MDSettings, init_state, make_key, make_waves, simulate  # noqa: E402
from xla_cco.workloads import energy_for  # noqa: E402

PHI_PACK = 0.05
_MAX_PAIRS = 1.4e9   # (k, particle) pairs of the largest listed evaluation


def listed() -> list:
    return [
        # the smallest call: energy, gradient and density of one configuration,
        # as an outer optimiser or a test calls it step by step
        dict(name="value_d2_n100", kind="value", n=100, d=2, chi=0.20),
        # one evaluation of the headline batch (256 lanes, d=2)
        dict(name="evaluate_d2_n1000_b256", kind="evaluate", n=1000, d=2, chi=0.40, batch=256),
        # the large 3-D batch
        dict(name="evaluate_d3_n4000_b64", kind="evaluate", n=4000, d=3, chi=0.45, batch=64),
        # one wide 1-D configuration, N not a multiple of any tile
        dict(name="evaluate_d1_n7777_b1", kind="evaluate", n=7777, d=1, chi=0.48, batch=1),
        # the largest single system of the request stream
        dict(name="evaluate_d2_n20000_b1", kind="evaluate", n=20000, d=2, chi=0.45, batch=1),
        # the headline relaxation, cut to an evaluation budget (a program that
        # checkpoints between budgeted calls): ticks of evaluation and L-BFGS update
        dict(name="relax_lbfgs_d2_n1000_b256", kind="relax", method="lbfgs", n=1000, d=2, chi=0.40,
             batch=256, evals=32),
        # the ground-state driver's small descent, five lanes
        dict(name="relax_descent_d3_n100_b5", kind="relax", method="descent", n=100, d=3, chi=0.05,
             batch=5, evals=400),
        # an ensemble of uneven N, d and chi relaxed together
        dict(name="relax_mixed_48", kind="relax_mixed", count=48, shapes=0, n_lo=200, n_hi=8000,
             evals=20),
        # the Jacobian of an implicit flow step / a vibrational analysis
        dict(name="hessian_d2_n700", kind="hessian", n=700, d=2, chi=0.40, batch=1),
        # a production MD segment: BAOAB, tracked waves, snapshots and trace
        dict(name="md_d2_n1000_l64", kind="md", n=1000, d=2, chi=0.40, batch=64, steps=40),
        # structure factor of relaxed configurations over the driver's k-set
        dict(name="structure_d2_n1000_b16", kind="structure", n=1000, d=2, batch=16, k_max=400.0),
        # g2 and nearest neighbours of the same ensemble
        dict(name="pairs_d2_n1000_b256", kind="pairs", n=1000, d=2, batch=256, bins=200),
    ]


def _log_int(rng, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["value", "evaluate", "evaluate", "evaluate", "relax", "relax", "relax_mixed", "hessian",
                       "md", "structure", "pairs"])  # fmt: skip
    d = rng.choice([1, 2, 2, 3])
    chi = round(rng.uniform(0.05, 0.49), 3)
    if kind == "value":
        return dict(kind=kind, n=_log_int(rng, 50, 2000), d=d, chi=chi)
    if kind == "evaluate":
        n = _log_int(rng, 100, 8000 if d == 1 else 20000)
        most = max(1, min(256, int(_MAX_PAIRS / (n * (chi * d * n + 1)))))
        return dict(kind=kind, n=n, d=d, chi=chi, batch=_log_int(rng, 1, most))
    if kind == "relax":
        if rng.random() < 0.3:
            return dict(kind=kind, method="descent", n=_log_int(rng, 40, 400), d=rng.choice([2, 3]),
                        chi=round(rng.uniform(0.03, 0.10), 3), batch=_log_int(rng, 1, 32),
                        evals=rng.choice([100, 200, 300]))  # fmt: skip
        n = _log_int(rng, 200, 4000)
        most = max(1, min(256, int(2.1e8 / (n * (chi * d * n + 1)))))
        return dict(kind=kind, method="lbfgs", n=n, d=d, chi=chi, batch=_log_int(rng, 1, most),
                    evals=20 if d == 1 else rng.choice([20, 26, 32]))  # fmt: skip
    if kind == "relax_mixed":
        return dict(kind=kind, count=rng.randint(4, 48), shapes=rng.randint(1, 1 << 20), n_lo=200,
                    n_hi=rng.choice([2000, 8000]), evals=rng.choice([12, 16, 20]))  # fmt: skip
    if kind == "hessian":
        return dict(kind=kind, n=_log_int(rng, 60, 900), d=d, chi=chi, batch=rng.choice([1, 1, 1, 3]))
    if kind == "md":
        return dict(kind=kind, n=_log_int(rng, 100, 1500), d=rng.choice([2, 3]), chi=round(rng.uniform(0.1, 0.4), 3),
                    batch=_log_int(rng, 4, 48), steps=rng.choice([20, 30, 40]))  # fmt: skip
    if kind == "structure":
        return dict(kind=kind, n=_log_int(rng, 200, 1500), d=rng.choice([1, 2]), batch=rng.randint(1, 16),
                    k_max=rng.choice([100.0, 200.0, 300.0]))  # fmt: skip
    return dict(kind=kind, n=_log_int(rng, 100, 2000), d=d, batch=_log_int(rng, 1, 100),
                bins=rng.choice([50, 200, 333, 1000]))  # fmt: skip


# ------------------------------------------------------------------ inputs
def _uniform(seed: int, *shape: int) -> torch.Tensor:
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _shapes(case: dict) -> list:
    """(N, d, chi) of an uneven ensemble: log-uniform N, d of 1..3, uniform chi."""
    rng = np.random.default_rng(case["shapes"])
    out = []
    for _ in range(case["count"]):
        n = int(round(float(np.exp(rng.uniform(np.log(case["n_lo"]), np.log(case["n_hi"]))))))
        out.append((n, int(rng.integers(1, 4)), float(rng.uniform(0.05, 0.49))))
    return out


def _settings(case: dict):
    if case.get("method") == "descent":
        return DescentSettings(grow=2.0, max_evals=case["evals"], energy_tol=9.99999968e-21)
    return LBFGSSettings(energy_tol=1e-20, rescales=(1e4,), max_evals_per_pass=case["evals"])


def _edges(case: dict) -> np.ndarray:
    return np.linspace(0.0, 0.2 * case["n"] ** (1.0 / case["d"]), case["bins"] + 1)


def _k_outer(case: dict) -> float:
    d = case["d"]
    return k_outer_from_ka(ka_from_chi(case["chi"], PHI_PACK, d), PHI_PACK, d)


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    st: dict = {"case": case}
    if kind == "relax_mixed":
        shapes = _shapes(case)
        st["energies"] = [energy_for(*s) for s in shapes]
        flat = _uniform(seed, sum(n * d for n, d, _ in shapes))
        at, st["s"] = 0, []
        for n, d, _ in shapes:
            st["s"].append(flat[at:at + n * d].reshape(n, d))
            at += n * d
        st["settings"] = _settings(case)
        return st
    n, d = case["n"], case["d"]
    if kind in ("structure", "pairs"):
        st["box"] = cubic_box(n, d)
        st["s"] = _uniform(seed, case["batch"], n, d)
        if kind == "pairs":
            st["edges"] = _edges(case)
        return st
    st["energy"] = energy_for(n, d, case["chi"])
    if kind == "value":
        st["s"] = _uniform(seed, n, d)
    elif kind == "md":
        b = case["batch"]
        basis = np.asarray(cubic_box(n, d).basis)
        k = _k_outer(case)
        st["waves"] = make_waves(basis, k, 1.5 * k)
        steps = case["steps"]
        st["settings"] = MDSettings(dt=0.02, scheme="baoab", gamma=1.0, chunk_steps=steps, wind_every=10,
                                    record_steps=(steps // 2, steps), record_rho_every=20,
                                    max_rho_records=steps // 20, drift_tol=float("inf"))  # fmt: skip
        u = _uniform(seed, 2, b, n, d)
        r0 = u[0] @ torch.from_numpy(basis).cuda()
        v0 = (u[1] - 0.5) * 0.1
        keys = np.stack([make_key(int(seed) * 1000 + i) for i in range(b)])
        st["basis"] = basis
        st["lanes"] = init_state(st["energy"], st["waves"], basis, r0, v0, np.full(b, 1e-3), keys, st["settings"])
    else:
        st["s"] = _uniform(seed, case["batch"], n, d)
        if kind == "relax":
            st["settings"] = _settings(case)
    return st


# ------------------------------------------------------------------ the calls
def run(st: dict):
    case = st["case"]
    kind = case["kind"]
    if kind == "value":
        return st["energy"].value_grad_density(st["s"])
    if kind == "evaluate":
        phi, grad, _, _ = st["energy"].evaluate(st["s"])
        return phi, grad
    if kind == "relax":
        r = relax(st["energy"], st["s"], st["settings"])
        return r.s, r.energy, r.grad_norm, r.n_evals, r.n_iters, r.status
    if kind == "relax_mixed":
        out = relax_mixed(st["energies"], st["s"], st["settings"])
        cat = lambda key: torch.cat([getattr(r, key).reshape(-1) for r in out])  # noqa: E731
        return tuple(cat(k) for k in ("s", "energy", "grad_norm", "n_evals", "n_iters", "status"))
    if kind == "hessian":
        return st["energy"].hessian(st["s"] if case["batch"] > 1 else st["s"][0])
    if kind == "md":
        end = simulate(st["energy"], st["waves"], st["basis"], st["settings"], st["lanes"], case["steps"]).state
        return (end.r, end.v, end.f, end.phi, end.rho_prev, end.wind_abs, end.wind_net, end.n_valid, end.sum_s,
                end.sum_phi, end.sum_kinetic, end.snap.r, end.snap.rho, end.trace.rho, end.step, end.status)  # fmt: skip
    if kind == "structure":
        return isotropic_structure_factor(st["s"], st["box"], 5.0, case["k_max"])
    counts = pair_distance_histogram(st["s"], st["box"], st["edges"])
    return counts, nearest_neighbor_distances_batch(st["s"], st["box"])


# ------------------------------------------------------------------ work
def _rows(n: int, d: int, chi: float) -> float:
    return chi * d * (n - 1)   # constrained wave vectors, about


def _sk_rows(case: dict) -> float:
    """k-vectors of the isotropic structure factor, about."""
    n, d, k_max = case["n"], case["d"], case["k_max"]
    unit = 2.0 * math.pi / n ** (1.0 / d)
    if d == 1:
        return k_max / unit
    r = 5.0 / unit   # primitive directions of a half disk, each with k_max / |k| multiples
    return (6.0 / math.pi**2) * math.pi * r * (k_max / unit)


def _eval_work(n: int, d: int, m: float, batch: float, grad: bool = True) -> dict:
    # a separable sum: 2 multiply-adds per (k, particle) for the density, 4
    # more for the gradient; positions in, gradient out, the k-set once
    return dict(bytes=batch * (16.0 if grad else 8.0) * n * d + m * (4.0 * d + 8.0),
                flops=batch * (12.0 if grad else 4.0) * n * m)  # fmt: skip


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "relax_mixed":
        total = dict(bytes=0.0, flops=0.0)
        for n, d, chi in _shapes(case):
            w = _eval_work(n, d, _rows(n, d, chi), case["evals"])
            total = dict(bytes=total["bytes"] + 16.0 * n * d, flops=total["flops"] + w["flops"])
        return total
    n, d = case["n"], case["d"]
    if kind == "structure":
        return _eval_work(n, d, _sk_rows(case), case["batch"], grad=False)
    if kind == "pairs":
        # a pair: the difference, its nearest integer, d squares, once for the
        # histogram and once per direction for the nearest neighbours
        pairs = case["batch"] * n * (n - 1) / 2.0
        return dict(bytes=case["batch"] * n * (8.0 * d + 8.0), flops=pairs * 5.0 * d)
    m = _rows(n, d, case["chi"])
    if kind == "value":
        w = _eval_work(n, d, m, 1.0)
        return dict(bytes=w["bytes"] + 16.0 * m, flops=w["flops"])
    if kind == "evaluate":
        return _eval_work(n, d, m, case["batch"])
    if kind == "relax":
        evals = case["evals"] / 2 if case["method"] == "descent" else case["evals"]
        b = case["batch"]
        return dict(bytes=16.0 * b * n * d, flops=evals * _eval_work(n, d, m, b)["flops"])
    if kind == "hessian":
        b = case["batch"]
        # per pair of particles and k: cos of the phase difference from products
        # (2) and d (d + 1) / 2 weighted sums, over half of the symmetric matrix
        return dict(bytes=b * (8.0 * n * d + 8.0 * (n * d) ** 2),
                    flops=b * 0.5 * n * n * m * (4.0 + d * (d + 1)))  # fmt: skip
    b, steps = case["batch"], case["steps"]
    waves = m * 1.5**d
    w = _eval_work(n, d, m, b)
    fresh = (waves - m) * n * b * 4.0 * max(1, steps // 10)
    return dict(bytes=b * (8.0 * 6 * n * d + 8.0 * 8 * waves), flops=steps * w["flops"] + fresh)


# ------------------------------------------------------------------ float64 values
def _phases(nv: torch.Tensor, s: torch.Tensor):
    """cos and sin of 2 pi n . s, (M, N): each product split so that its whole
    part leaves before anything is rounded."""
    hi = torch.round(s * 2.0**26) / 2.0**26   # n hi is exact for |n| < 2^26
    lo = s - hi
    t = torch.zeros(nv.shape[0], s.shape[0], dtype=torch.float64, device=s.device)
    for a in range(s.shape[1]):
        p = nv[:, a:a + 1] * hi[None, :, a]
        t += (p - torch.round(p)) + nv[:, a:a + 1] * lo[None, :, a]
    t -= torch.round(t)
    t *= 2.0 * math.pi
    return torch.cos(t), torch.sin(t)


def _kset(n: int, d: int, k_outer: float) -> np.ndarray:
    """Half of the nonzero integer vectors with |k| < k_outer in the unit-density cube."""
    unit = 2.0 * math.pi / n ** (1.0 / d)
    r = int(k_outer / unit) + 1
    ax = np.arange(-r, r + 1)
    g = np.stack(np.meshgrid(*([ax] * d), indexing="ij"), axis=-1).reshape(-1, d)
    first = np.zeros(len(g), dtype=np.int64)   # sign of the first nonzero component
    for a in range(d):
        first = np.where(first == 0, np.sign(g[:, a]), first)
    return g[(first > 0) & (np.sqrt((g.astype(np.float64) ** 2).sum(1)) * unit < k_outer)].astype(np.float64)


def _exact_eval(case: dict, s: torch.Tensor, energy):
    """(phi, grad, re, im) of s (B, N, d) by direct sums over the energy's rows."""
    nv = torch.from_numpy(np.asarray(energy.n_vectors)).cuda()
    w = torch.from_numpy(np.asarray(energy.weights)).cuda()
    vol = float(energy.volume)
    b, n, d = s.shape
    m = nv.shape[0]
    step = max(1, int(2.5e7) // n)
    phi = torch.zeros(b, dtype=torch.float64, device="cuda")
    grad = torch.zeros_like(s)
    re = torch.zeros(b, m, dtype=torch.float64, device="cuda")
    im = torch.zeros_like(re)
    for i in range(b):
        for lo in range(0, m, step):
            c, sn = _phases(nv[lo:lo + step], s[i])
            wk = w[lo:lo + step]
            r, q = c.sum(1), sn.sum(1)
            re[i, lo:lo + step], im[i, lo:lo + step] = r, q
            phi[i] += (wk * (r * r + q * q)).sum() / vol
            core = (wk * q)[:, None] * c - (wk * r)[:, None] * sn
            grad[i] += (4.0 * math.pi / vol) * (core.T @ nv[lo:lo + step])
    return phi, grad, re, im


def _exact_hessian(s: torch.Tensor, energy):
    nv = torch.from_numpy(np.asarray(energy.n_vectors)).cuda()
    w = torch.from_numpy(np.asarray(energy.weights)).cuda()
    n, d = s.shape
    c, sn = _phases(nv, s)
    re, im = c.sum(1), sn.sum(1)
    h = torch.zeros(n, d, n, d, dtype=torch.float64, device="cuda")
    at = torch.arange(n, device="cuda")
    for a in range(d):
        for e in range(d):
            q = w * nv[:, a] * nv[:, e]
            blk = (c * q[:, None]).T @ c + (sn * q[:, None]).T @ sn
            blk[at, at] -= (q[:, None] * (re[:, None] * c + im[:, None] * sn)).sum(0)
            h[:, a, :, e] = blk
    return (2.0 * (2.0 * math.pi) ** 2 / float(energy.volume)) * h.reshape(n * d, n * d)


def _exact_structure(case: dict, s: torch.Tensor):
    n, d, k_max = case["n"], case["d"], case["k_max"]
    unit = 2.0 * math.pi / n ** (1.0 / d)
    if d == 1:
        dirs = np.ones((1, 1))
    else:
        dirs = _kset(n, d, 5.0)
        dirs = dirs[np.gcd.reduce(np.abs(dirs).astype(np.int64), axis=1) == 1]
    rows = []
    for v in dirs:
        top = int(k_max / (unit * math.sqrt(float(v @ v)))) + 2
        g = np.arange(1, top)[:, None] * v[None, :]
        rows.append(g[((g * unit) ** 2).sum(1) <= k_max * k_max])
    nv = torch.from_numpy(np.concatenate(rows)).cuda()
    tot = torch.zeros(nv.shape[0], dtype=torch.float64, device="cuda")
    tot2 = torch.zeros_like(tot)
    step = max(1, int(2.5e7) // n)
    for x in s:
        for lo in range(0, nv.shape[0], step):
            c, sn = _phases(nv[lo:lo + step], x)
            sk = (c.sum(1) ** 2 + sn.sum(1) ** 2) / n
            tot[lo:lo + step] += sk
            tot2[lo:lo + step] += sk * sk
    b = s.shape[0]
    k = np.sqrt(((nv.cpu().numpy() * unit) ** 2).sum(1))
    idx = np.floor(k / 0.01).astype(np.int64)
    sums = [np.bincount(idx, weights=v) for v in (np.ones(k.size), k, tot.cpu().numpy() / b, tot2.cpu().numpy() / b)]
    cnt, sk1, ss, ss2 = (v[sums[0] > 0] for v in sums)
    mean = ss / cnt
    # the standard error of |k| is rounding alone in a bin of one shell: no exact value
    with np.errstate(invalid="ignore"):
        return sk1 / cnt, mean, None, np.sqrt((ss2 / cnt - mean**2) / (cnt * b))


def _exact_nearest(case: dict, s: torch.Tensor) -> torch.Tensor:
    n, d = case["n"], case["d"]
    side = n ** (1.0 / d)
    out = torch.empty(s.shape[0], n, dtype=torch.float64, device="cuda")
    for i, x in enumerate(s):
        r2 = torch.zeros(n, n, dtype=torch.float64, device="cuda")
        for a in range(d):
            t = x[None, :, a] - x[:, None, a]
            r2 += ((t - torch.round(t)) * side) ** 2
        r2.fill_diagonal_(side * side)   # a particle's own nearest image
        out[i] = r2.min(1).values.sqrt()
    return out


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind in ("relax", "relax_mixed", "md"):   # iterated maps: no closed value
        return None
    st = prepare(case, seed)
    if kind == "value":
        phi, grad, re, im = _exact_eval(case, st["s"][None], st["energy"])
        return phi[0], grad[0], re[0], im[0]
    if kind == "evaluate":
        return _exact_eval(case, st["s"], st["energy"])[:2]
    if kind == "hessian":
        h = [_exact_hessian(x, st["energy"]) for x in st["s"]]
        return torch.stack(h) if case["batch"] > 1 else h[0]
    if kind == "structure":
        return _exact_structure(case, st["s"])
    return None, _exact_nearest(case, st["s"])
