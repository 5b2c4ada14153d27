"""Workloads of the stochastic-KPM transport path, each through an entry point that a program calls.

A case names one operation on one model:

* ``moments``   Jackson-KPM moments of a block of random-phase vectors (``B200Operators.moments``)
* ``series``    one Bessel propagation of the augmented state [psi | phi] (``B200Operators.series``)
* ``stepwise``  a whole stepwise MSD run (``stochastic.stepwise_samples``)
* ``solve``     the metric solve S^-1 B (``B200Metric.solve``)
* ``vac``       the correlation tables of the spectral VAC (``B200Operators.chain_correlate``)
* ``batch``     moments of a ragged batch of disorder realisations (``B200Batch.moments``)

The models are the lattices of this package: the orthogonal square and honeycomb lattices with Anderson disorder, and the
nonorthogonal sp3 diamond with 4x4 atom blocks of H and S, condition number about 50 and block-Jacobi preconditioning.
The uploaded operators belong to the model and are kept, as a program does that runs many vector blocks through them;
the vectors are drawn from the seed.
"""
from __future__ import annotations

import functools
from types import SimpleNamespace

import numpy as np
import scipy.linalg as la
import scipy.sparse as sp
import torch

from kubomsd_b200 import kpm, lattices, stochastic
from kubomsd_b200.batch import B200Batch
from kubomsd_b200.config import RunConfig
from kubomsd_b200.native import B200Metric, B200Operators
from kubomsd_b200.operators import build_operators

WINDOW = {"square": 11.2, "honeycomb": 9.2, "diamond": 40.}  # half-width of the spectral window, eV
BAND = {"square": 11., "honeycomb": 9., "diamond": 35.}


def listed():
    return [
        # the small reference system: 64 x 64 sites, 8 vectors, the default direct FP64 moments
        {"name": "moments_sq64_fp64", "op": "moments", "model": "square", "lx": 64, "ly": 64, "R": 8, "M": 512,
         "precision": "fp64", "doubling": False},
        # the same system's stepwise MSD, moments and propagation alternating (a whole call)
        {"name": "stepwise_sq64_fp64", "op": "stepwise", "model": "square", "lx": 64, "ly": 64, "R": 8, "M": 512,
         "precision": "fp64", "doubling": True, "tmax": 4},
        # a small resident lattice of the serving stream, odd in every size
        {"name": "moments_sq127_mixed", "op": "moments", "model": "square", "lx": 127, "ly": 127, "R": 31, "M": 511,
         "precision": "mixed", "doubling": True},
        # the middle resident lattice of the serving stream (1M sites) with 32 vectors
        {"name": "moments_hc1M_mixed", "op": "moments", "model": "honeycomb", "lx": 1024, "ly": 512, "R": 32, "M": 256,
         "precision": "mixed", "doubling": True},
        # the 4,194,304-site lattice of the precision form with its 64 vectors
        {"name": "moments_hc4M_mixed", "op": "moments", "model": "honeycomb", "lx": 2048, "ly": 1024, "R": 64, "M": 64,
         "precision": "mixed", "doubling": True},
        # the plain FP64 form on a lattice far larger than the caches, direct moments
        {"name": "moments_hc1M_fp64", "op": "moments", "model": "honeycomb", "lx": 1024, "ly": 512, "R": 64, "M": 64,
         "precision": "fp64", "doubling": False},
        # one 1 fs step of the stepwise MSD on the 1M-site lattice
        {"name": "series_hc1M_mixed", "op": "series", "model": "honeycomb", "lx": 1024, "ly": 512, "R": 16, "dt": 1.,
         "precision": "mixed"},
        # a small nonorthogonal cell of the serving stream: a metric solve in every Chebyshev step
        {"name": "moments_sp3_2k", "op": "moments", "model": "diamond", "lx": 4, "ly": 4, "R": 8, "M": 32,
         "precision": "fp64", "doubling": False},
        # the 32,000-orbital nonorthogonal system with its 32 vectors
        {"name": "moments_sp3_32k", "op": "moments", "model": "diamond", "lx": 10, "ly": 10, "R": 32, "M": 8,
         "precision": "fp64", "doubling": False},
        # one metric solve as velocity actions and sampling call it, on an odd number of vectors
        {"name": "solve_sp3_7k", "op": "solve", "model": "diamond", "lx": 6, "ly": 6, "R": 13},
        # the velocity-autocorrelation tables of one segment on a 16k-site lattice
        {"name": "vac_sq128", "op": "vac", "model": "square", "lx": 128, "ly": 128, "R": 8, "M": 256, "K": 40,
         "precision": "fp64"},
        # a ragged batch of disorder realisations, all moments in one call
        {"name": "batch_sq_mixed", "op": "batch", "model": "square", "lx": 24, "ly": 160, "count": 24, "R": 16,
         "M": 256, "precision": "mixed", "doubling": True},
    ]


def _log(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]."""
    return max(lo, min(hi, round(lo * (hi / lo) ** rng.random())))


# vector-block elements times operator applications of one pass, at most (the 4,194,304-site case)
MOST = 4194304 * 64 * 32


def draw(rng):
    op = rng.choice(["moments"] * 6 + ["series"] * 3 + ["sp3"] * 3 + ["solve"] * 2 + ["stepwise", "vac", "batch"])
    precision = rng.choice(["fp64", "mixed"])
    if op in ("moments", "series"):
        if rng.random() < .5:
            size = {"model": "square", "lx": _log(rng, 24, 700), "ly": _log(rng, 24, 700)}
            size["ly"] = size["lx"]
        else:
            size = {"model": "honeycomb", "lx": _log(rng, 24, 1200), "ly": _log(rng, 24, 700)}
        n = _sites(size)
        if op == "moments":
            c = {"op": op, **size, "R": _log(rng, 1, 64), "M": _log(rng, 32, 1024), "precision": precision,
                 "doubling": rng.random() < .5}
            apps = c["M"] // 2 if c["doubling"] else c["M"]
            if n * c["R"] * apps > MOST // 8:
                c["M"] = max(32, int(c["M"] * (MOST // 8) / (n * c["R"] * apps)))
            return c
        r = _log(rng, 1, 32)
        if n * r > 2 ** 24:
            r = max(1, 2 ** 24 // n)
        return {"op": op, **size, "R": r + r % 2 if precision == "mixed" else r, "dt": rng.choice([.25, .5, 1.]),
                "precision": precision}
    if op == "sp3":
        cells = rng.randint(3, 10)
        return {"op": "moments", "model": "diamond", "lx": cells, "ly": cells, "R": _log(rng, 1, 32),
                "M": max(4, min(32, round(32 * (4 / cells) ** 2))) + rng.randint(0, 3), "precision": "fp64",
                "doubling": False}
    if op == "solve":
        cells = rng.randint(3, 12)
        return {"op": op, "model": "diamond", "lx": cells, "ly": cells, "R": _log(rng, 1, 48)}
    if op == "stepwise":
        side = _log(rng, 24, 200)
        return {"op": op, "model": "square", "lx": side, "ly": side, "R": 2 * _log(rng, 1, 16),
                "M": _log(rng, 64, 512), "precision": precision, "doubling": rng.random() < .5,
                "tmax": rng.randint(1, 4)}
    if op == "vac":
        side = _log(rng, 32, 256)
        return {"op": op, "model": "square", "lx": side, "ly": side, "R": 2 * rng.randint(1, 4),
                "M": _log(rng, 64, 512), "K": rng.randint(10, 48), "precision": precision}
    return {"op": op, "model": "square", "lx": rng.randint(20, 40), "ly": _log(rng, 60, 256),
            "count": rng.randint(4, 48), "R": _log(rng, 2, 32), "M": _log(rng, 32, 512), "precision": precision,
            "doubling": rng.random() < .5}


# ------------------------------------------------------------------ models
def _sites(case):
    if case["model"] == "diamond":
        return 32 * case["lx"] ** 3
    return case["lx"] * case["ly"] * (2 if case["model"] == "honeycomb" else 1)


def _sides(case):
    """Lattice sides of the batch's instances, from lx to ly over their logarithm."""
    k = case["count"]
    return [round(case["lx"] * (case["ly"] / case["lx"]) ** (i / max(1, k - 1))) for i in range(k)]


@functools.lru_cache(maxsize=2)
def _model(kind, lx, ly, seed=20261203):
    if kind == "square":
        return lattices.square_lattice(lx, seed=seed)
    if kind == "honeycomb":
        return lattices.honeycomb(lx, ly, seed=seed)
    return lattices.diamond_sp3(cells=lx, scale_hint=.24, seed=seed)


def _config(case):
    w, e = WINDOW[case["model"]], BAND[case["model"]]
    return RunConfig(energy_eV=np.linspace(-e, e, 201), time_fs=np.arange(case.get("tmax", 0) + 1.),
                     spectral_bounds=(-w, w), n_moments=case.get("M", 64), axes=("x",), include_vac=False,
                     stochastic_method="stepwise", precision=case.get("precision", "fp64"),
                     moment_doubling=bool(case.get("doubling", False)))


@functools.lru_cache(maxsize=1)
def _operators(kind, lx, ly, precision, with_velocity):
    """The uploaded operators of a model: an orthogonal lattice, or the sp3 model with its block-Jacobi metric."""
    m = _model(kind, lx, ly)
    cfg = _config({"model": kind, "precision": precision})
    S = sp.csr_matrix(m.S)
    blocks = []
    if kind == "diamond":
        blocks = [(a, b, la.cholesky(S[a:b, a:b].toarray(), lower=True)) for a, b in m.atom_slices]
    metric = B200Metric(S, S.diagonal().real.copy(), blocks, cfg)
    return B200Operators(SimpleNamespace(host_H=m.H, metric=SimpleNamespace(native=metric),
                                         velocity=m.velocity if with_velocity else {}, position={}, composite={}), cfg)


@functools.lru_cache(maxsize=1)
def _bundle(kind, lx, ly, M, tmax, precision, doubling):
    cfg = _config({"model": kind, "M": M, "tmax": tmax, "precision": precision, "doubling": doubling})
    return build_operators(_model(kind, lx, ly), cfg), cfg


@functools.lru_cache(maxsize=1)
def _batch(sides, precision):
    return B200Batch([lattices.square_lattice(side, seed=100 + i).H for i, side in enumerate(sides)],
                     precision=precision)


# ------------------------------------------------------------------ inputs
def _phases(n, columns, seed):
    """Unit-modulus random phases, (n, columns) complex128."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    u = torch.rand((n, columns), dtype=torch.float64, device="cuda", generator=g)
    return torch.polar(torch.ones_like(u), u.mul_(2 * np.pi))


def _gauss(shape, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(shape, dtype=torch.complex128, device="cuda", generator=g)


def _inputs(case, seed):
    n, r = _sites(case), case["R"]
    if case["op"] == "batch":
        return {"B": _phases(sum(s * s for s in _sides(case)), r, seed)}
    if case["op"] == "series":  # a state under way: psi of unit modulus, phi grown to a few angstrom
        return {"B": torch.cat([_phases(n, r, seed), 3 * _gauss((n, r), seed + 1)], dim=1).contiguous()}
    if case["op"] == "vac":
        return {"B": _phases(n, r, seed), "cov": _gauss((n, case["K"] + 1, r), seed + 1)}
    return {"B": _phases(n, r, seed)}


def _coefficients(case):
    return kpm.bessel_coefficients(case["dt"], _config(case), weighted_tail=True)[0]


def prepare(case, seed):
    s = {"case": case, "half": WINDOW[case["model"]], **_inputs(case, seed)}
    key = case["model"], case["lx"], case["ly"]
    precision = case.get("precision", "fp64")
    if case["op"] == "stepwise":
        s["ops"], s["cfg"] = _bundle(*key, case["M"], case["tmax"], precision, bool(case["doubling"]))
    elif case["op"] == "batch":
        s["batch"] = _batch(tuple(_sides(case)), precision)
    else:
        s["ops"] = _operators(*key, precision, case["op"] == "series")
        s["cfg"] = _config(case)
    if case["op"] == "series":
        s["coeff"] = _coefficients(case)
    return s


def run(s):
    case, op = s["case"], s["case"]["op"]
    if op == "moments":
        return s["ops"].moments(s["B"], case["M"], 0., s["half"], doubling=bool(case["doubling"]))
    if op == "series":
        return s["ops"].series(s["B"], s["coeff"], 0., s["half"], [[1., 0., 0.]])
    if op == "stepwise":
        dos, numerators, _ = stochastic.stepwise_samples(s["ops"], s["cfg"], s["B"], device=True)
        return [dos, numerators["msd_A2/commutator"]]
    if op == "solve":
        return s["ops"].metric.solve(s["B"], s["cfg"])[0]
    if op == "vac":
        return s["ops"].chain_correlate(s["B"], s["cov"], case["M"] + case["K"], 0., s["half"])
    return s["batch"].moments(s["B"], case["M"], 0., s["half"], doubling=bool(case["doubling"]))


# ------------------------------------------------------------------ work
def work(case):
    """Inputs read once and outputs written once; the operations of the recurrences (a complex multiply by a real
    matrix entry is 4) and, where S is not the identity, of about 80 CG iterations for each application."""
    n, r, op = _sites(case), case["R"], case["op"]
    row = {"square": 5, "honeycomb": 4, "diamond": 65}[case["model"]]
    m = case.get("M", 0)
    if op == "batch":
        n = sum(s * s for s in _sides(case))
    apps = (m + 1) // 2 if case.get("doubling") else m - 1
    matrix, step = 12. * row * n, (4. * row + 14.) * n * r
    cg = (4. * row + 4 * 4. + 30.) * n * r * 80
    if op == "moments":
        if case["model"] == "diamond":
            return {"bytes": 2 * matrix + 16. * n * r + 8. * m * r, "flops": apps * (step + cg)}
        return {"bytes": matrix + 16. * n * r + 8. * m * r, "flops": apps * step}
    if op == "batch":
        return {"bytes": matrix + 16. * n * r + 8. * m * r * case["count"], "flops": apps * step}
    if op == "solve":
        return {"bytes": matrix + 32. * n * r, "flops": cg}
    if op == "series":
        k = len(_coefficients(case)) - 1
        return {"bytes": 2 * matrix + 64. * n * r, "flops": k * (2 * step + 8. * row * n * r)}
    if op == "stepwise":
        k = len(kpm.bessel_coefficients(1., _config(case), weighted_tail=True)[0]) - 1
        t = case["tmax"]
        return {"bytes": 2 * matrix + 16. * n * r + 8. * (t + 2) * r * 201,
                "flops": (t + 2) * (apps * step + 2. * m * r * 201) + t * k * (2 * step + 8. * row * n * r)}
    length, k1 = m + case["K"], case["K"] + 1
    return {"bytes": matrix + 16. * n * r * (1 + k1) + 16. * r * length * k1,
            "flops": length * step + 8. * n * r * length * k1}


# ------------------------------------------------------------------ values in 64 bits
def _dense_apply(A):
    """x -> A x for a host CSR matrix, in complex128 on the GPU."""
    A = sp.csr_matrix(A).astype(np.complex128)
    a = torch.sparse_csr_tensor(torch.from_numpy(A.indptr.astype(np.int64)), torch.from_numpy(A.indices.astype(np.int64)),
                                torch.from_numpy(A.data), size=A.shape).cuda()
    return lambda x: a @ x


def _columns(x, y):
    return (x.conj() * y).sum(0).real


def _solver(S, slices):
    """x -> S^-1 x by block-preconditioned CG to rounding."""
    apply = _dense_apply(S)
    width = slices[0][1] - slices[0][0]
    inverse = torch.from_numpy(np.stack([np.linalg.inv(S[a:b, a:b].toarray()) for a, b in slices])).cuda().to(torch.complex128)

    def precondition(r):
        return torch.bmm(inverse, r.reshape(len(slices), width, -1)).reshape(r.shape)

    def solve(b):
        x, r = torch.zeros_like(b), b.clone()
        z = precondition(r)
        p, rz = z.clone(), _columns(r, z)
        goal = 1e-28 * _columns(b, b)
        for k in range(400):
            if k % 20 == 0 and bool((_columns(r, r) <= goal).all()):
                break
            q = apply(p)
            alpha = rz / _columns(p, q).clamp_min(1e-300)
            x += alpha * p
            r -= alpha * q
            z = precondition(r)
            new = _columns(r, z)
            p = z + (new / rz.clamp_min(1e-300)) * p
            rz = new
        return x

    return solve


def _moments(act, bra, B, count, half, doubling):
    mu = torch.empty((count, B.shape[1]), dtype=torch.float64, device=B.device)
    mu[0] = _columns(bra, B)
    prev, cur = B, act(B) / half
    if count > 1:
        mu[1] = _columns(bra, cur)
    k = 1
    while (2 * k if doubling else k + 1) < count:  # prev = T_{k-1}, cur = T_k
        if doubling:
            mu[2 * k] = 2 * _columns(cur, cur) - mu[0]
        nxt = act(cur).mul_(2 / half).sub_(prev)
        if not doubling:
            mu[k + 1] = _columns(bra, nxt)
        elif 2 * k + 1 < count:
            mu[2 * k + 1] = 2 * _columns(nxt, cur) - mu[1]
        prev, cur, k = cur, nxt, k + 1
    return mu


def _series(h, v, x, coeff, half):
    r = x.shape[1] // 2

    def act(y):
        out = h(y) / half
        out[:, r:] += (-1j * kpm.HBAR_EV_FS / half) * v(y[:, :r].contiguous())
        return out

    prev, cur = x, act(x)
    out = complex(coeff[0]) * prev + complex(coeff[1]) * cur
    for c in coeff[2:]:
        prev, cur = cur, 2 * act(cur) - prev
        out += complex(c) * cur
    return out


def _jackson(energy, half, count):
    """(G mu): the Jackson-damped reconstruction at the energies, (energies, moments)."""
    m = np.arange(count)
    t = np.pi / (count + 1)
    g = ((count + 1 - m) * np.cos(m * t) + np.sin(m * t) / np.tan(t)) / (count + 1)
    g[1:] *= 2
    x = np.asarray(energy) / half
    return torch.from_numpy(np.cos(np.arccos(x)[:, None] * m) * g / (np.pi * half * np.sqrt(1 - x * x))[:, None]).cuda()


def exact(case, seed):
    op, half = case["op"], WINDOW[case["model"]]
    i = _inputs(case, seed)
    B = i["B"]
    if op == "batch":
        at, out = 0, []
        for k, side in enumerate(_sides(case)):
            b = B[at:at + side * side]
            out.append(_moments(_dense_apply(lattices.square_lattice(side, seed=100 + k).H), b, b, case["M"], half, True))
            at += side * side
        return torch.stack(out)
    m = _model(case["model"], case["lx"], case["ly"])
    if op == "solve":
        return _solver(m.S.tocsr(), m.atom_slices)(B)
    h = _dense_apply(m.H)
    if op == "moments":
        if case["model"] == "diamond":
            solve = _solver(m.S.tocsr(), m.atom_slices)
            return _moments(lambda x: solve(h(x)), _dense_apply(m.S)(B), B, case["M"], half, False)
        return _moments(h, B, B, case["M"], half, True)
    if op == "series":
        return _series(h, _dense_apply(m.velocity["x"]), B, _coefficients(case), half)
    if op == "stepwise":
        v, count, cfg = _dense_apply(m.velocity["x"]), case["M"], _config(case)
        coeff = kpm.bessel_coefficients(1., cfg, weighted_tail=True)[0]
        G = _jackson(cfg.energy_eV, half, count)
        r = case["R"]
        x = torch.cat([B, torch.zeros_like(B)], dim=1)
        msd = torch.zeros((r, 1, case["tmax"] + 1, len(cfg.energy_eV)), dtype=torch.float64, device="cuda")
        for j in range(1, case["tmax"] + 1):
            x = _series(h, v, x, coeff, half)
            phi = x[:, r:].contiguous()
            msd[:, 0, j] = (G @ _moments(h, phi, phi, count, half, True)).T
        return [(G @ _moments(h, B, B, count, half, True)).T.contiguous(), msd]
    out = torch.empty((case["R"], case["M"] + case["K"], case["K"] + 1), dtype=torch.complex128, device="cuda")
    cov = i["cov"].permute(2, 0, 1).contiguous()  # (column, site, k)
    prev, cur = None, B
    for j in range(out.shape[1]):
        out[:, j] = torch.bmm(cur.T.conj().unsqueeze(1), cov)[:, 0]
        prev, cur = cur, h(cur) / half if prev is None else 2 * h(cur) / half - prev
    return out
