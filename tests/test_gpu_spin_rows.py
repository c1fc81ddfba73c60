"""The spin-S rows apply against the tile apply it replaces (needs a B200)."""

import numpy as np
import pytest

import alps_b200 as ed

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def _chain(n):
    return [(i, (i + 1) % n) for i in range(n)]


def _square(length, width):
    out = []
    for x in range(length):
        for y in range(width):
            s = x * width + y
            out += [(s, x * width + (y + 1) % width), (s, (x + 1) % length * width + y)]
    return out


def _couple(pairs, classes, biquadratic, rng):
    js = rng.uniform(-1.5, 1.5, (classes, 3))
    return [(i, j, *js[q % classes][:2], js[q % classes][2] if biquadratic else 0.0) for q, (i, j) in enumerate(pairs)]


def _row_bound(bonds, site_h, site_d, two_s):
    """A bound of sum_j |H_ij|: |Sz Sz| and the exchange at most S^2 and S (S + 1), the biquadratic their sum squared."""
    s = two_s / 2
    b = sum(abs(jz) * s * s + abs(jxy) * s * (s + 1) + abs(k) * (s * s + s * (s + 1)) ** 2 for _, _, jz, jxy, k in bonds)
    return b + sum(abs(h) * s for h in site_h) + sum(abs(d) * s * s for d in site_d)


# odd and even splits, one-row blocks (nearly polarised), blocks of several 1024-row tiles, crossing digits with and
# without keys (the square lattices have many), one to eight coupling classes, every number of off-diagonal slots
@pytest.mark.parametrize("two_s,pairs,n,total,classes,biq", [
    (2, _chain(4), 4, 4, 1, False), (2, _chain(9), 9, 2, 2, True), (2, _chain(15), 15, 15, 1, False),
    (2, _chain(16), 16, 14, 2, False), (2, _square(3, 3), 9, 9, 8, True), (2, _square(4, 3), 12, 11, 3, False),
    (1, _square(4, 4), 16, 8, 3, False), (3, _chain(9), 9, 13, 2, True), (3, _square(3, 3), 9, 14, 1, False),
    (4, _chain(8), 8, 16, 2, True), (4, _chain(9), 9, 17, 1, False), (4, _chain(5), 5, 1, 1, True),
])
def test_spin_rows_match_the_tile_apply(two_s, pairs, n, total, classes, biq, monkeypatch):
    rng = np.random.default_rng(n * two_s + total)
    bonds = _couple(pairs, classes, biq, rng)
    site_h, site_d = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)

    def pair(b, h, d):
        made = []
        for rows in ("1", "0"):
            monkeypatch.setenv("AED_SPIN_ROWS", rows)
            made.append(ed.Hamiltonian(n, total, b, two_s=two_s, generic=True, site_h=h, site_d=d))
        return made

    rows, tile = pair(bonds, site_h, site_d)
    for step in range(3):  # other couplings on the same handles: a pure Ising model, then more transitions
        x, v = rng.normal(size=rows.dim), rng.normal(size=rows.dim)
        tol = 8 * (len(bonds) + n) * EPS * _row_bound(bonds, site_h, site_d, two_s) * np.max(np.abs(x))
        y0, y1 = tile.apply(x), rows.apply(x)
        assert np.max(np.abs(y1 - y0)) <= tol
        got = []
        for h in (rows, tile):
            a, b, c = h.new_vector().upload(v), h.new_vector().upload(x), h.new_vector()
            got.append(h.lanczos_step(a, b, c, 0.3)[0])
        assert abs(got[0] - got[1]) <= tol * np.sum(np.abs(x)) + EPS * rows.dim * abs(got[1])
        bonds = [(i, j, 0.8, 0.0, 0.0) for i, j in pairs] if step == 0 else _couple(pairs, 2, two_s > 1, rng)
        site_h = site_d = np.zeros(n)
        for h, on in ((rows, "1"), (tile, "0")):
            monkeypatch.setenv("AED_SPIN_ROWS", on)
            h.set_couplings(bonds)


def test_spin_rows_keep_infinities_to_their_rows(monkeypatch):
    n, two_s = 10, 2
    bonds = [(i, j, 1.0, 1.0, 0.0) for i, j in _chain(n)]
    made = []
    for rows in ("1", "0"):
        monkeypatch.setenv("AED_SPIN_ROWS", rows)
        made.append(ed.Hamiltonian(n, n, bonds, two_s=two_s))
    x = np.random.default_rng(1).normal(size=made[0].dim)
    x[[3, 500, made[0].dim - 1]] = np.inf
    x[77] = np.nan
    a, b = (h.apply(x) for h in made)
    assert np.array_equal(np.isfinite(a), np.isfinite(b)) and np.isfinite(a).sum() > made[0].dim // 2
