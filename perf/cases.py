"""Timed cases of the engine's public entry points (alps_b200).

Each case is one call that an exact-diagonalisation program makes in its inner loop, or one whole solve:

  mult       y = H x in an Sz sector of a spin-1/2 model (Hamiltonian.mult): the matrix product of every
             Krylov method a program builds on the engine
  step       one Lanczos step with its alpha and beta read back (Hamiltonian.lanczos_step): the ietl
             recurrence driven from the caller's loop
  momentum   y = H x in a momentum sector (complex vectors), spin 1/2 or spin S
  spin       y = H x in an Sz sector of a spin-S model
  solve      set_couplings + solve on a kept handle (a scan over couplings); the FP64 solve with its Ritz
             vectors, as a program that measures in the ground state asks for them
  sector     create a momentum sector's handle, solve it, destroy it: one turn of sparsediag's default loop
  batch      submit a set of independent chains to a running Server and run them to completion

Vectors hold normalised Gaussian values, as Lanczos vectors do.  Couplings, vectors and start seeds come from
the case's seed.
"""

from __future__ import annotations

import math
import random

import numpy as np
import torch

import alps_b200 as ed


def listed():
    return [
        # the smallest sector of the test suite's solves: launch latency
        {"name": "mult_chain16_fp64", "kind": "mult", "lattice": "chain", "L": 16, "W": 1, "n_up": 8, "fp": 64},
        # a caller-driven recurrence on a mid-size chain: three kernels and two scalars per call
        {"name": "step_chain20_fp64", "kind": "step", "lattice": "chain", "L": 20, "W": 1, "n_up": 10, "fp": 64},
        # an odd number of sites away from half filling, every bond its own coupling
        {"name": "mult_square5x5_fp64", "kind": "mult", "lattice": "square", "L": 5, "W": 5, "n_up": 11, "fp": 64},
        # the benchmark's sector, full precision
        {"name": "mult_chain28_fp64", "kind": "mult", "lattice": "chain", "L": 28, "W": 1, "n_up": 14, "fp": 64},
        # the largest sector of the benchmark, the product of the mixed-precision path
        {"name": "mult_square6x5_fp32", "kind": "mult", "lattice": "square", "L": 6, "W": 5, "n_up": 15, "fp": 32},
        # the default (translation symmetric) path's product at the benchmark's size
        {"name": "momentum_chain28", "kind": "momentum", "L": 28, "two_s": 1, "sz": 0, "k": 0},
        # spin-1 chain, Sz = 0
        {"name": "spin1_chain18", "kind": "spin", "L": 18, "two_s": 2, "sz": 0, "biquadratic": False},
        # its momentum sectors
        {"name": "spin1_momentum_chain18", "kind": "momentum", "L": 18, "two_s": 2, "sz": 0, "k": 5},
        # a scan's solve in a small sector, with the Ritz vectors
        {"name": "solve_chain16_fp64", "kind": "solve", "lattice": "chain", "L": 16, "W": 1, "n_up": 8, "fp": 64,
         "nev": 4},
        # a served request's single-instance solve in mixed precision
        {"name": "solve_ladder2x12_mixed", "kind": "solve", "lattice": "ladder", "L": 12, "W": 2, "n_up": 12,
         "fp": 32, "nev": 2},
        # one turn of the loop over momenta: tables, solve, release
        {"name": "sector_chain22", "kind": "sector", "L": 22, "two_s": 1, "sz": 0, "k": 11, "nev": 2},
        # independent chains through the batched engine
        {"name": "batch_64_chains_mixed", "kind": "batch", "requests": 64, "largest": 20, "fp": 32, "nev": 1},
    ]


def draw(rng: random.Random):
    kind = rng.choice(["mult", "mult", "mult", "step", "momentum", "spin", "solve", "sector", "batch"])
    if kind in ("mult", "step", "solve"):
        top = 28 if kind == "mult" else 26 if kind == "step" else 22
        lattice = rng.choice(["chain", "ladder", "square"])
        if lattice == "chain":
            length, width = rng.randint(12, top), 1
        elif lattice == "ladder":
            length, width = rng.randint(6, min(13, top // 2)), 2
        else:
            length, width = rng.choice([s for s in ((4, 3), (5, 3), (4, 4), (6, 3), (5, 4), (7, 3), (6, 4), (5, 5),
                                                    (9, 3)) if s[0] * s[1] <= top])
        n = length * width
        c = {"kind": kind, "lattice": lattice, "L": length, "W": width, "n_up": n // 2 - rng.choice([0, 0, 1, 2, 3]),
             "fp": rng.choice([64, 32])}
        if kind == "solve":
            c["nev"] = rng.randint(1, 2)
        return c
    if kind == "batch":
        return {"kind": "batch", "requests": int(round(8 * 8 ** rng.random())), "largest": rng.choice([14, 16, 18, 20]),
                "fp": rng.choice([64, 32]), "nev": 1}
    two_s = rng.choice([1, 1, 2, 3]) if kind == "momentum" else rng.choice([2, 2, 3, 4]) if kind == "spin" else 1
    top = {("momentum", 1): 28, ("momentum", 2): 17, ("momentum", 3): 12, ("spin", 2): 18, ("spin", 3): 13,
           ("spin", 4): 11, ("sector", 1): 22}[kind, two_s]
    n = rng.randint(top // 2, top)
    sz = rng.choice([0, 0, 1, 2]) * 2 + (n * two_s) % 2  # twice Sz_total, the parity of the sector
    c = {"kind": kind, "L": n, "two_s": two_s, "sz": sz}
    if kind == "spin":
        c["biquadratic"] = rng.random() < 0.25
    else:
        c["k"] = rng.randrange(n)
    if kind == "sector":
        c["nev"] = 1
    return c


# ---------------------------------------------------------------- models


def chain_bonds(n, j1, j2):
    """J1-J2 chain, periodic: per site the nearest and the next-nearest bond."""
    out = []
    for i in range(n):
        out.append((i, (i + 1) % n, j1, j1, 0.0))
        out.append((i, (i + 2) % n, j2, j2, 0.0))
    return out


def ladder_bonds(length, jl, jr):
    """Two-leg ladder, periodic legs; site = 2 x + y."""
    out = []
    for x in range(length):
        for y in range(2):
            s = 2 * x + y
            out.append((s, 2 * ((x + 1) % length) + y, jl, jl, 0.0))
            if y == 0:
                out.append((s, s + 1, jr, jr, 0.0))
    return out


def square_bonds(length, width, js):
    """Periodic square lattice, site = x W + y, one coupling per bond."""
    out = []
    for x in range(length):
        for y in range(width):
            s = x * width + y
            for t in (x * width + (y + 1) % width, ((x + 1) % length) * width + y):
                j = float(js[len(out)])
                out.append((s, t, j, j, 0.0))
    return out


def model(case, seed):
    """(sites, digit sum, bonds) of a case; digit sum = Sz_total + N S (the up spins for spin 1/2)."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind in ("momentum", "sector", "spin"):
        n = case["L"]
        digit_sum = (case["sz"] + n * case["two_s"]) // 2
        j1, j2 = 1.0, float(rng.uniform(0.0, 0.45))
        if case["two_s"] == 1:
            return n, digit_sum, chain_bonds(n, j1, j2)
        j, kq = float(rng.uniform(0.8, 1.2)), float(rng.uniform(0.1, 0.4)) if case.get("biquadratic") else 0.0
        return n, digit_sum, [(i, (i + 1) % n, j, j, kq) for i in range(n)]
    n = case["L"] * case["W"]
    if case["lattice"] == "chain":
        bonds = chain_bonds(n, 1.0, float(rng.uniform(0.0, 0.45)))
    elif case["lattice"] == "ladder":
        bonds = ladder_bonds(case["L"], *(float(v) for v in rng.uniform(0.5, 1.5, 2)))
    else:
        bonds = square_bonds(case["L"], case["W"], rng.uniform(0.8, 1.2, 2 * n))
    return n, case["n_up"], bonds


def batch_models(case, seed):
    """[(sites, bonds)] of a batch: J1-J2 chains of even length."""
    rng = np.random.default_rng(seed)
    sizes = rng.choice(np.arange(12, case["largest"] + 1, 2), size=case["requests"])
    return [(int(n), chain_bonds(int(n), 1.0, float(j2))) for n, j2 in zip(sizes, rng.uniform(0.0, 0.45, len(sizes)))]


def dimension(n, digits, digit_sum):
    """States of n sites of `digits` values with that digit sum."""
    row = [1]
    for _ in range(n):
        new = [0] * (len(row) + digits - 1)
        for s, c in enumerate(row):
            for v in range(digits):
                new[s + v] += c
        row = new
    return row[digit_sum] if 0 <= digit_sum < len(row) else 0


# ---------------------------------------------------------------- state and pass


class _Buffer:
    """A device vector of the engine as torch sees it; the tensor made from it keeps it, and so the vector."""

    def __init__(self, vector, n, fp):
        self.vector = vector
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f4" if fp == 32 else "<f8",
                                         "data": (vector.ptr.value, False), "version": 3, "strides": None,
                                         "stream": None}


def _vector(ham, fp):
    v = ham.new_vector()
    return v, torch.as_tensor(_Buffer(v, ham.vlen, fp), device="cuda")


def _values(n, fp, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(n, generator=g, device="cuda", dtype=torch.float32 if fp == 32 else torch.float64)
    return x.div_(torch.linalg.vector_norm(x, dtype=torch.float64).to(x.dtype))


def _translations(case):
    n = case["L"]
    return ed.lattice_translations({"MODEL": "spin", "LATTICE": "chain lattice", "L": n}, (2.0 * math.pi * case["k"] / n,))


def prepare(case, seed):
    kind, fp = case["kind"], case.get("fp", 64)
    precision = ed.FP32 if fp == 32 else ed.FP64
    state = {"case": case, "seed": seed}
    if kind == "batch":
        state["server"] = ed.Server(precision=precision, max_slots=case["requests"], hbm_budget=4 << 30, reserve=-1)
        state["requests"] = batch_models(case, seed)
        return state
    n, digit_sum, bonds = model(case, seed)
    if kind == "sector":
        state.update(n=n, digit_sum=digit_sum, bonds=bonds, translations=_translations(case))
        return state
    ham = ed.Hamiltonian(n, digit_sum, bonds, precision=precision, two_s=case.get("two_s", 1),
                         translations=_translations(case) if kind == "momentum" else None)
    state["ham"] = ham
    if kind == "solve":
        state["bonds"] = bonds
        return state
    state["x"], x = _vector(ham, fp)
    state["y"], state["out"] = _vector(ham, fp)
    x.copy_(_values(ham.vlen, fp, seed))
    if kind == "step":
        state["prev"], prev = _vector(ham, fp)
        prev.copy_(_values(ham.vlen, fp, seed + 1))
        state["beta"] = 0.25 * n
    torch.cuda.synchronize()  # the engine's calls run on the handle's own stream
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("mult", "momentum", "spin"):
        state["ham"].mult(state["x"], state["y"])
        return state["out"]
    if kind == "step":
        alpha, beta = state["ham"].lanczos_step(state["prev"], state["x"], state["y"], state["beta"])
        return {"alpha": alpha, "beta": beta, "next": state["out"]}
    if kind == "solve":
        ham = state["ham"]
        ham.set_couplings(state["bonds"])
        evals = ham.solve(nev=case["nev"], seed=state["seed"])["evals"]
        if case["fp"] == 32:
            return {"evals": evals}
        vectors, _, _ = ham.eigenvectors(1, seed=state["seed"])
        ground = vectors[0].download()
        vectors[0].free()
        return {"evals": evals, "ground": ground}
    if kind == "sector":
        ham = ed.Hamiltonian(state["n"], state["digit_sum"], state["bonds"], two_s=case["two_s"],
                             translations=state["translations"])
        evals = ham.solve(nev=case["nev"], seed=state["seed"])["evals"]
        ham.close()
        return {"evals": evals}
    server = state["server"]
    tickets = [server.submit(n, n // 2, bonds, nev=case["nev"], seed=state["seed"] + i)
               for i, (n, bonds) in enumerate(state["requests"])]
    results = server.run(tickets)
    return [torch.from_numpy(np.concatenate([results[t]["evals"] for t in tickets]))]


# ---------------------------------------------------------------- work

_STEPS = 60  # products of a typical solve


def work(case):
    """Every vector of the call read or written once (x and y of a product; x, v_prev and y of a step), and a
    multiply-add per matrix element.  A solve: its products, at a typical number of them."""
    kind, size = case["kind"], case.get("fp", 64) // 8
    if kind == "batch":
        b = f = 0
        sizes = range(12, case["largest"] + 1, 2)
        for n in sizes:
            d = dimension(n, 2, n // 2)
            b += 2 * size * d * _STEPS * case["requests"] / len(sizes)
            f += 2 * (n + 1) * d * _STEPS * case["requests"] / len(sizes)
        return {"bytes": b, "flops": f}
    n, digit_sum, bonds = model(case, 0)
    d = dimension(n, case.get("two_s", 1) + 1, digit_sum)
    terms = 1 + len(bonds) / 2 * (1 if case.get("two_s", 1) == 1 else 1.4)
    vectors = 3 if kind == "step" else 2
    if kind in ("momentum", "sector"):
        d /= n  # representatives
        size, terms = 16, 4 * terms
    repeat = _STEPS if kind in ("solve", "sector") else 1
    return {"bytes": vectors * size * d * repeat, "flops": 2 * terms * d * repeat}


# ---------------------------------------------------------------- the same in plain torch, 64 bits


def _bits(two_s):
    return max(1, math.ceil(math.log2(two_s + 1)))


class _Sector:
    """States (packed digits, site 0 most significant, ascending) and ranks of one digit sum."""

    def __init__(self, n, two_s, digit_sum):
        self.n, self.d, self.bits = n, two_s + 1, _bits(two_s)
        self.nlo = n // 2
        lo_sum, hi_sum = self._sums(self.nlo), self._sums(n - self.nlo)
        top = two_s * self.nlo
        members = [np.nonzero(lo_sum == s)[0] for s in range(top + 1)]
        count = np.array([len(m) for m in members], np.int64)
        tlo = np.zeros(len(lo_sum), np.int64)
        for m in members:
            tlo[m] = np.arange(len(m))
        rest = np.where(hi_sum >= 0, digit_sum - hi_sum, -1)
        rows = np.where((rest >= 0) & (rest <= top), count[np.clip(rest, 0, top)], 0)
        thi = np.cumsum(rows) - rows
        self.dim = int(rows.sum())
        dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
        self.tlo, self.thi = dev(tlo), dev(thi)
        self.lolist, self.looff = dev(np.concatenate(members)), dev(np.cumsum(count) - count)
        self.rest, self.hi_codes, self.hi_start = dev(rest), dev(np.nonzero(rows)[0]), dev(thi[rows > 0])

    def _sums(self, n):
        codes = np.arange(1 << (self.bits * n))
        s, ok = np.zeros(len(codes), np.int64), np.ones(len(codes), bool)
        for i in range(n):
            v = (codes >> (self.bits * i)) & ((1 << self.bits) - 1)
            s += v
            ok &= v < self.d
        return np.where(ok, s, -1)

    def states(self, first, last):
        rows = torch.arange(first, last, device="cuda")
        b = torch.searchsorted(self.hi_start, rows, right=True) - 1
        hi = self.hi_codes[b]
        return (hi << (self.bits * self.nlo)) | self.lolist[self.looff[self.rest[hi]] + rows - self.hi_start[b]]

    def rank(self, s):
        sh = self.bits * self.nlo
        return self.thi[s >> sh] + self.tlo[s & ((1 << sh) - 1)]


def _bond_elements(two_s, jz, jxy, kq):
    """{k: element of (a, c) -> (a + k, c - k) for every digit pair} of one bond."""
    d, spin = two_s + 1, two_s / 2
    m = np.arange(d) - spin
    sz, sp = np.diag(m), np.zeros((d, d))
    for v in range(d - 1):
        sp[v + 1, v] = math.sqrt(spin * (spin + 1) - m[v] * (m[v] + 1))
    zz, xy = np.kron(sz, sz), 0.5 * (np.kron(sp, sp.T) + np.kron(sp.T, sp))
    h = jz * zz + jxy * xy + kq * (zz + xy) @ (zz + xy)
    out = {}
    for k in range(-two_s, two_s + 1):
        e = np.zeros(d * d)
        for a in range(d):
            for c in range(d):
                if 0 <= a + k < d and 0 <= c - k < d:
                    e[a * d + c] = h[(a + k) * d + c - k, a * d + c]
        if np.any(e != 0.0) or k == 0:
            out[k] = torch.from_numpy(e).cuda()
    return out


def _terms(sector, bonds, s):
    """Diagonal of the states s, and (element, target state) of every off-diagonal term in turn."""
    n, bits, d = sector.n, sector.bits, sector.d
    known = {}
    diag = torch.zeros(len(s), dtype=torch.float64, device="cuda")
    offs = []
    for i, j, jz, jxy, kq in bonds:
        wi, wj = bits * (n - 1 - i), bits * (n - 1 - j)
        if (jz, jxy, kq) not in known:
            known[jz, jxy, kq] = _bond_elements(d - 1, jz, jxy, kq)
        el = known[jz, jxy, kq]
        pair = ((s >> wi) & ((1 << bits) - 1)) * d + ((s >> wj) & ((1 << bits) - 1))
        diag += el[0][pair]
        offs += [(el[k], pair, k * ((1 << wi) - (1 << wj))) for k in el if k]

    def off():
        for e, pair, change in offs:
            v = e[pair]
            yield v, torch.where(v != 0.0, s + change, s)

    return diag, off


def _product(sector, bonds, x):
    """H x, rows in pieces."""
    y = torch.empty(sector.dim, dtype=torch.float64, device="cuda")
    piece = 1 << 22
    for first in range(0, sector.dim, piece):
        last = min(sector.dim, first + piece)
        diag, off = _terms(sector, bonds, sector.states(first, last))
        acc = diag * x[first:last].double()
        for v, target in off():
            acc += v * x[sector.rank(target)].double()
        y[first:last] = acc
    return y


class _Momentum:
    """The representatives of a chain's momentum sector and the way of any state to its representative."""

    def __init__(self, sector, k):
        self.sector, n = sector, sector.n
        self.phase = torch.exp(1j * (2.0 * math.pi * k / n) * torch.arange(n, device="cuda", dtype=torch.float64))
        reps, norms = [], []
        piece = 1 << 22
        for first in range(0, sector.dim, piece):
            s = sector.states(first, min(sector.dim, first + piece))
            low, _, weight = self._orbit(s)
            w = weight.abs().sqrt()
            keep = (low == s) & (w >= 0.01)
            reps.append(s[keep])
            norms.append(w[keep] / math.sqrt(n))
        self.reps, self.norms = torch.cat(reps), torch.cat(norms)
        self.dim = len(self.reps)

    def _orbit(self, s):
        n, bits = self.sector.n, self.sector.bits
        low, which = s.clone(), torch.zeros_like(s)
        weight = torch.ones(len(s), dtype=torch.complex128, device="cuda")
        for t in range(1, n):
            ts = (s >> (bits * t)) | ((s & ((1 << (bits * t)) - 1)) << (bits * (n - t)))
            weight += torch.where(ts == s, self.phase[t], torch.zeros_like(weight))
            which = torch.where(ts < low, t, which)
            low = torch.minimum(low, ts)
        return low, which, weight

    def terms(self, bonds, first, last):
        """As _terms for the representatives [first, last): (element, representative) of every term."""
        diag, off = _terms(self.sector, bonds, self.reps[first:last])

        def mapped():
            for v, target in off():
                low, which, _ = self._orbit(target)
                j = torch.searchsorted(self.reps, low).clamp_(max=self.dim - 1)
                v = torch.where(self.reps[j] == low, v, torch.zeros_like(v))
                yield v * self.norms[j] / self.norms[first:last] * self.phase[which], j

        return diag, mapped

    def product(self, bonds, x):
        y = torch.empty(self.dim, dtype=torch.complex128, device="cuda")
        piece = 1 << 20
        for first in range(0, self.dim, piece):
            last = min(self.dim, first + piece)
            diag, off = self.terms(bonds, first, last)
            acc = diag * x[first:last]
            for v, j in off():
                acc += v * x[j]
            y[first:last] = acc
        return y


def _lowest(sector, bonds, nev, basis=None):
    """The nev lowest distinct eigenvalues: Lanczos with full reorthogonalisation in 64 bits.  With `basis` (a
    _Momentum) in that sector."""
    if basis is None:
        dim = sector.dim
        diag, off = _terms(sector, bonds, sector.states(0, dim))
        pairs = [(v, sector.rank(target).to(torch.int32)) for v, target in off()]
    else:
        dim = basis.dim
        diag, off = basis.terms(bonds, 0, dim)
        pairs = [(v, j.to(torch.int32)) for v, j in off()]
    el, at = torch.stack([p[0] for p in pairs]), torch.stack([p[1] for p in pairs])

    def product(x):
        return diag * x + (el * x[at]).sum(0)

    g = torch.Generator(device="cuda").manual_seed(7)
    kind = torch.float64 if basis is None else torch.complex128
    v = torch.randn(dim, generator=g, device="cuda", dtype=kind)
    most = min(dim, 400)
    room = torch.empty((most, dim), dtype=kind, device="cuda")
    room[0] = v / torch.linalg.vector_norm(v)
    alpha, beta, got = [], [], None
    for j in range(most):
        w = product(room[j])
        alpha.append(float(torch.vdot(room[j], w).real))
        for _ in range(2):
            w = w - room[: j + 1].T @ (room[: j + 1].conj() @ w)
        b = float(torch.linalg.vector_norm(w))
        if j % 5 == 4 or j == most - 1 or b < 1e-10:
            vals, vecs = np.linalg.eigh(np.diag(alpha) + np.diag(beta, 1) + np.diag(beta, -1))
            got = vals[:nev]
            if b < 1e-10 or (len(vals) > nev and np.all(b * np.abs(vecs[-1, :nev]) < 1e-10)):
                return got
        if j + 1 < most:
            beta.append(b)
            room[j + 1] = w / b
    return got


def exact(case, seed):
    kind, fp = case["kind"], case.get("fp", 64)
    if kind == "batch":
        sectors, out = {}, []
        for n, bonds in batch_models(case, seed):
            if n not in sectors:
                sectors[n] = _Sector(n, 1, n // 2)
            out.append(_lowest(sectors[n], bonds, case["nev"]))
        return [torch.from_numpy(np.concatenate(out))]
    n, digit_sum, bonds = model(case, seed)
    sector = _Sector(n, case.get("two_s", 1), digit_sum)
    if kind == "sector":
        return {"evals": _lowest(sector, bonds, case["nev"], _Momentum(sector, case["k"]))}
    if kind == "momentum":
        basis = _Momentum(sector, case["k"])
        x = torch.view_as_complex(_values(2 * basis.dim, 64, seed).view(-1, 2))
        return torch.view_as_real(basis.product(bonds, x)).reshape(-1)
    if kind == "solve":
        evals = _lowest(sector, bonds, case["nev"])
        return {"evals": evals} if fp == 32 else {"evals": evals, "ground": None}
    x = _values(sector.dim, fp, seed).double()
    y = _product(sector, bonds, x)
    if kind != "step":
        return y
    alpha = torch.dot(x, y)
    y = y - alpha * x - 0.25 * n * _values(sector.dim, fp, seed + 1).double()
    beta = torch.linalg.vector_norm(y)
    return {"alpha": float(alpha), "beta": float(beta), "next": y / beta}
