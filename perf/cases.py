"""What a user of this library has it do, as measurable cases.

A case names a kind of system (the seeded generators of
libecp_gb300.workloads), its sizes and the entry point that computes it:

* ``dropin``    getIntegrals as a linked host program calls it (plain FP64
                kernels), host arrays in, AO matrix out;
* ``batched``   ecpgb_getIntegrals with the batched FP64 engine, the same;
* ``mixed``     the same with the mixed-precision engine;
* ``resident``  a device-resident job: inputs copied once (an SCF or scan code
                keeps the job), then a run and its AO matrix;
* ``blocks``    every block and unit status of the batched engine (the
                derivative order is the case's: 0, 1 or 2);
* ``gradient``  energy and nuclear gradient of a density matrix, contracted on
                the GPU;
* ``serve``     a burst of requests through the request server.

The systems: ``one_centre`` (the reference's example: one heavy atom, four
light ones, s p d shells), ``cluster`` (ECP atoms in a box, s..f shells of 1 to
8 primitives), ``g_batch`` (s..g shells of up to 10 primitives, exponents 0.02
to 200), ``sweep`` (s..g shells, exponents 0.015 to 500, ECP channels to L = 5),
``molecules`` (requests of 5 to 40 atoms).
"""
from __future__ import annotations

import math

import numpy as np
import torch

import libecp_gb300 as eg
from libecp_gb300 import workloads as W

# Sizes: centres (ECP atoms), atoms (with basis, three shells each) or shells.
_LISTED = [
    # the smallest call: the reference's own example through its own interface
    dict(name="one_centre_dropin", path="dropin", system="one_centre"),
    # the same call of a program that switched to the batched engine
    dict(name="one_centre_batched", path="batched", system="one_centre"),
    # an unchanged program with a mid-size cluster
    dict(name="cluster6_dropin", path="dropin", system="cluster", centres=6, atoms=21),
    # a small molecule with three heavy atoms, one call per geometry
    dict(name="cluster3_batched", path="batched", system="cluster", centres=3, atoms=11),
    # the 50-centre cluster of the benchmark, kept on the device
    dict(name="cluster50_resident", path="resident", system="cluster", centres=50, atoms=21),
    # mixed precision on a part of it
    dict(name="cluster16_mixed", path="mixed", system="cluster", centres=16, atoms=21),
    # high angular momentum and long contractions, all blocks read back
    dict(name="g_batch_blocks", path="blocks", system="g_batch", centres=5, shells=83, deriv=0),
    # diffuse to very compact primitives, L = 5 channels
    dict(name="sweep_batched", path="batched", system="sweep", centres=4, shells=150),
    # a geometry step: energy and forces of a density
    dict(name="cluster5_gradient", path="gradient", system="cluster", centres=5, atoms=13),
    # second-derivative blocks (s..d shells, shifted up to g)
    dict(name="hessian_blocks", path="blocks", system="spd", centres=3, atoms=7, deriv=2),
    # a burst of requests of different sizes
    dict(name="serve_burst", path="serve", system="molecules", requests=12, max_atoms=40),
]


def listed():
    return [dict(c) for c in _LISTED]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["dropin", "batched", "batched", "resident", "mixed", "blocks", "gradient", "serve"])
    if path == "serve":
        return dict(path=path, system="molecules", requests=rng.randint(3, 14), max_atoms=_log_int(rng, 8, 40))
    if path == "gradient":
        return dict(path=path, system="cluster", centres=rng.randint(1, 6), atoms=_log_int(rng, 3, 13))
    system = rng.choice(["cluster", "cluster", "g_batch", "sweep"])
    if path == "blocks":
        deriv = rng.randint(0, 2)
        if deriv:  # shifted shells stay within g
            return dict(path=path, system="spd" if deriv == 2 else "cluster", centres=rng.randint(1, 4),
                        atoms=_log_int(rng, 2, 8), deriv=deriv)
        if system == "cluster":
            return dict(path=path, system=system, centres=_log_int(rng, 1, 30), atoms=_log_int(rng, 3, 21), deriv=0)
        return dict(path=path, system=system, centres=rng.randint(1, 5), shells=_log_int(rng, 9, 90), deriv=0)
    if system == "cluster":
        return dict(path=path, system=system, centres=_log_int(rng, 1, 8 if path == "dropin" else 40),
                    atoms=_log_int(rng, 3, 21))
    return dict(path=path, system=system, centres=rng.randint(1, 4),
                shells=_log_int(rng, 9, 45 if path == "dropin" else 120))


def _system(case, seed):
    """A system of the case's kind: its shells and channels (l, contraction)
    are the case's, so every seed has the same shapes; positions, exponents
    and coefficients come from the seed, in the generator's distributions."""
    kind = case["system"]
    box, elo, ehi = {"one_centre": (4.0, 0.05, 50.0), "cluster": (12.0, 0.05, 50.0), "spd": (8.0, 0.05, 50.0),
                     "g_batch": (14.0, 0.02, 200.0), "sweep": (16.0, 0.015, 500.0)}[kind]
    if kind == "one_centre":
        s = W.example_like(0)
    elif kind == "cluster":
        s = W.batched_cluster(0, n_centres=case["centres"], n_basis_atoms=case["atoms"])
    elif kind == "spd":
        s = W.batched_cluster(0, n_centres=case["centres"], n_basis_atoms=case["atoms"],
                              l_weights=(0.4, 0.35, 0.25), kmax=4)
    elif kind == "g_batch":
        s = W.mixed_batch(0, n_shells=case["shells"], n_centres=case["centres"])
    else:
        s = W.large_sweep(0, n_shells=case["shells"], n_centres=case["centres"])
    return _redraw(s, np.random.default_rng(seed), box, elo, ehi, fixed=1 if kind == "one_centre" else 0)


def _redraw(s, rng, box, elo, ehi, fixed=0):
    s.geometry[3 * fixed:] = rng.uniform(-box / 2, box / 2, s.geometry.size - 3 * fixed)
    s.nECP[:] = rng.integers(0, 3, s.nECP.size)
    s.dECP[:] = rng.uniform(-10.0, 10.0, s.dECP.size)
    s.aECP[:] = np.exp(rng.uniform(np.log(0.1), np.log(20.0), s.aECP.size))
    s.dBS[:] = rng.uniform(0.1, 1.0, s.dBS.size)
    s.aBS[:] = np.exp(rng.uniform(np.log(elo), np.log(ehi), s.aBS.size))
    return s


class _State:
    """The inputs of a pass and the handle a program keeps for it."""

    def __init__(self, path):
        self.path = path
        self.systems, self.density, self.job, self.server = [], None, None, None

    def __del__(self):
        for handle in (self.job, self.server):
            if handle is not None:
                handle.close()


def prepare(case, seed):
    s = _State(case["path"])
    if case["path"] == "serve":
        rng, n, top = np.random.default_rng(seed), case["requests"], case["max_atoms"]
        # 5 atoms up to the largest, log-spaced, small and large ones mixed
        for i in range(n):
            atoms = int(round(5 * (top / 5) ** (((5 * i) % n) / max(1, n - 1))))
            m = W.serving_molecule(np.random.default_rng(i), atoms, 1 + (3 * i) % min(atoms, 8))
            s.systems.append(_redraw(m, rng, 2.5 * atoms ** (1.0 / 3.0) + 2.0, 0.05, 50.0))
        s.server = eg.Server(mode=eg.ECPGB_FAST, budget_bytes=8 << 30, slots=8)
        return s
    system = _system(case, seed)
    system.derivative = case.get("deriv", 0)
    s.systems.append(system)
    if case["path"] == "gradient":
        d = np.random.default_rng(seed + 1).standard_normal((system.dim, system.dim))
        s.density = (d + d.T) / (2 * system.dim)
    if case["path"] == "resident":
        s.job = eg.Job(system, mode=eg.ECPGB_FAST)
    return s


def run(state):
    system = state.systems[0]
    if state.path == "dropin":
        return eg.get_integrals(system)
    if state.path == "batched":
        return eg.get_integrals_info(system, mode=eg.ECPGB_FAST)[1]
    if state.path == "mixed":
        return eg.get_integrals_info(system, mode=eg.ECPGB_MIXED)[1]
    if state.path == "resident":
        state.job.run(1, flush_l2=False)
        return state.job.matrix()
    if state.path == "blocks":
        values, _, status, _ = eg.raw_blocks(system, eg.ECPGB_FAST)
        return {"values": values, "status": status}
    if state.path == "gradient":
        energy, grad = eg.gradient(system, state.density, mode=eg.ECPGB_FAST)
        return {"energy": energy, "gradient": grad}
    ids = [state.server.submit(s) for s in state.systems]
    return [state.server.wait(i)[1] for i in ids]


def work(case):
    """Bytes of the results and inputs, and the floating-point operations of
    a lean evaluation: per (shell pair, centre) unit and primitive pair, both
    radial rules at the level they commonly stop at (95 of 383 and 255 of
    1023 points, a tenth of the latter not negligible), an exponential, five
    multiply-adds per Bessel row and one per quadrature and point."""
    kind = case["system"]
    # mean primitive pairs, Bessel rows and quadratures per unit of the kind
    prims, rows, quads = {"one_centre": (9, 4, 30), "cluster": (20, 4, 40), "spd": (6, 4, 60),
                          "g_batch": (30, 6, 90), "sweep": (12, 6, 120), "molecules": (12, 4, 40)}[kind]
    if kind == "molecules":
        n, top = case["requests"], case["max_atoms"]
        units = values = 0
        for i in range(n):
            atoms = int(round(5 * (top / 5) ** (((5 * i) % n) / max(1, n - 1))))
            units += (2 * atoms) * (2 * atoms + 1) // 2 * (1 + (3 * i) % min(atoms, 8))
            values += (2 * atoms * 5) ** 2
    else:
        shells = 12 if kind == "one_centre" else case["shells"] if "shells" in case else 3 * case["atoms"]
        shifts = (1, 4, 10)[case.get("deriv", 0)]
        if case["path"] == "gradient":
            shifts = 5
        units = shells * (shells + 1) // 2 * case.get("centres", 1) * shifts
        width = {"one_centre": 3.3, "cluster": 4, "spd": 3, "g_batch": 7, "sweep": 7}[kind]
        values = units * 2 * width * width if case["path"] == "blocks" else (shells * width) ** 2
    points = 95 + 25
    flops = units * prims * points * (2 * 5 * rows + 20 + 2 * quads / 4)
    return {"bytes": 8.0 * values + 16.0 * units / 10, "flops": float(flops)}


# ------------------------------------------------------------- 64-bit values

def _real_sph(lmax, x, y, z):
    """Real spherical harmonics of unit vectors, rows l*l + l + m."""
    ct, st = z, torch.sqrt(torch.clamp(1 - z * z, min=0.0))
    phi = torch.atan2(y, x)
    P, out = {}, []
    for m in range(lmax + 1):
        P[m, m] = torch.ones_like(ct) if m == 0 else P[m - 1, m - 1] * (2 * m - 1) * st
        for l in range(m + 1, lmax + 1):
            P[l, m] = ((2 * l - 1) * ct * P[l - 1, m] - (l + m - 1) * P.get((l - 2, m), 0.0)) / (l - m)
    for l in range(lmax + 1):
        for m in range(-l, l + 1):
            a = abs(m)
            n = math.sqrt((2 * l + 1) / (4 * math.pi) * math.factorial(l - a) / math.factorial(l + a))
            f = n * P[l, a]
            out.append(f if m == 0 else f * math.sqrt(2) * (torch.cos(a * phi) if m > 0 else torch.sin(a * phi)))
    return torch.stack(out)


def _shells_at(s, pts):
    """Contracted Cartesian functions (coefficients as given) at points [n, 3]."""
    geom, rows, sh, pr = s.geometry.reshape(-1, 3), [], 0, 0
    for atom in range(s.n_atoms):
        v = pts - torch.tensor(geom[atom], device=pts.device)
        r2 = (v * v).sum(1)
        for _ in range(int(s.shellsBS[atom])):
            l, k = int(s.lBS[sh]), int(s.KBS[sh])
            radial = sum(float(s.dBS[pr + i]) * torch.exp(-float(s.aBS[pr + i]) * r2) for i in range(k))
            for i in range(l + 1):
                for j in range(i + 1):
                    rows.append(v[:, 0] ** (l - i) * v[:, 1] ** (i - j) * v[:, 2] ** j * radial)
            sh, pr = sh + 1, pr + k
    return torch.stack(rows)


def _matrix64(s):
    """Upper triangle of the ECP matrix by a product quadrature around every
    centre: Gauss-Legendre panels in r, Gauss-Legendre in cos(theta),
    equidistant phi (the radial Jacobian is part of the ECP's r^n, as in the
    library's inputs)."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    geom = s.geometry.reshape(-1, 3)
    starts = np.concatenate([[0], np.cumsum(s.KECP)]).astype(int)
    xg, wg = np.polynomial.legendre.leggauss(12)
    edges = np.concatenate([np.linspace(0.0, 6.0, 73), np.linspace(6.0, 24.0, 25)[1:]])
    r = np.concatenate([(a + b) / 2 + (b - a) / 2 * xg for a, b in zip(edges[:-1], edges[1:])])
    wr = np.concatenate([(b - a) / 2 * wg for a, b in zip(edges[:-1], edges[1:])])
    nt, nph = 96, 192
    ct, wt = np.polynomial.legendre.leggauss(nt)
    phi = (np.arange(nph) + 0.5) * 2 * np.pi / nph
    st = np.sqrt(1 - ct * ct)
    unit = torch.tensor(np.stack([np.outer(st, np.cos(phi)), np.outer(st, np.sin(phi)),
                                  np.outer(ct, np.ones(nph))], -1).reshape(-1, 3), device=dev)
    wa = torch.tensor(np.repeat(wt, nph) * 2 * np.pi / nph, device=dev)
    V, e = torch.zeros(s.dim, s.dim, dtype=torch.float64, device=dev), 0
    for atom in range(s.n_atoms):
        n = int(s.shellsECP[atom])
        if n == 0:
            continue
        L = int(max(s.lECP[e:e + n]))
        U = np.zeros((L + 1, len(r)))
        for q in range(e, e + n):
            for t in range(starts[q], starts[q + 1]):
                U[int(s.lECP[q])] += s.dECP[t] * r ** s.nECP[t] * np.exp(-s.aECP[t] * r * r)
        e += n
        Y = _real_sph(max(L - 1, 0), unit[:, 0], unit[:, 1], unit[:, 2]) * wa
        centre = torch.tensor(geom[atom], device=dev)
        for i in range(len(r)):
            if np.abs(U[:, i]).max() < 1e-18:
                continue
            f = _shells_at(s, centre + float(r[i]) * unit)
            V += (wr[i] * U[L, i]) * ((f * wa) @ f.T)
            for l in range(L):
                T = f @ Y[l * l:(l + 1) * (l + 1)].T
                V += (wr[i] * U[l, i]) * (T @ T.T)
    return torch.triu(V).cpu().numpy()


def exact(case, seed):
    """The integrals by plain quadrature where that is quick: the one-centre
    systems.  (The library reproduces the reference's adaptive rules, which
    can stop early on a coarse level, and whose large-grid rule reads values
    of an earlier primitive pair beyond a contracted shell's break point: its
    matrices differ from the integrals by more than rounding.)"""
    if case["system"] != "one_centre":
        return None
    return _matrix64(_system(case, seed))
