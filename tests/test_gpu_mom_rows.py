"""The momentum apply from stored rows against the walking apply it replaces, bit for bit (needs a B200)."""

import numpy as np
import pytest

import alps_b200 as ed
from oracle import lattice

pytestmark = pytest.mark.gpu


def _pair(monkeypatch, *a, **kw):
    rows = ed.Hamiltonian(*a, **kw)
    monkeypatch.setenv("AED_MOM_WALK", "1")
    walk = ed.Hamiltonian(*a, **kw)
    monkeypatch.delenv("AED_MOM_WALK")
    return rows, walk


def _same(rows, walk, seed):
    assert rows.dim == walk.dim
    rng = np.random.default_rng(seed)
    x, v = (rng.normal(size=rows.dim) + 1j * rng.normal(size=rows.dim) for _ in range(2))
    assert np.array_equal(rows.apply(x), walk.apply(x))
    out = []
    for h in (rows, walk):
        a, b, c = h.new_vector().upload(v), h.new_vector().upload(x), h.new_vector()
        out.append((*h.lanczos_step(a, b, c, 0.3), c.download()))
    assert out[0][:2] == out[1][:2] and np.array_equal(out[0][2], out[1][2])


# sectors of a few rows (one slice), of a last slice that is not full, of several tiles, and several couplings per row
@pytest.mark.parametrize("lat,geo,two_s,total", [
    ("chain lattice", {"L": 4}, 1, 2), ("chain lattice", {"L": 9}, 1, 4), ("nnn chain lattice", {"L": 16}, 1, 8),
    ("nnn chain lattice", {"L": 20}, 1, 9), ("square lattice", {"L": 4, "W": 4}, 1, 8),
    ("chain lattice", {"L": 6}, 2, 6), ("nnn chain lattice", {"L": 9}, 2, 8), ("chain lattice", {"L": 6}, 3, 9),
    ("square lattice", {"L": 2, "W": 3}, 4, 12),
])
def test_stored_rows_equal_the_walk(lat, geo, two_s, total, monkeypatch):
    params = {"MODEL": "spin", "LATTICE": lat, **geo}
    n, _, graph = lattice.lattice_graph(lat, geo)
    bonds = [(s, t, 1.0 + 0.3 * ty, 0.7 - 0.2 * ty, 0.1 if two_s > 1 else 0.0) for s, t, ty in graph]
    momenta = ed.lattice_momenta(params)
    for k in (momenta[0], momenta[1], momenta[len(momenta) // 2], momenta[-1]):
        rows, walk = _pair(monkeypatch, n, total, bonds, translations=ed.lattice_translations(params, k), two_s=two_s)
        if rows.dim == 0:
            continue
        _same(rows, walk, 3)
        # other couplings on the same handles: fewer terms per row, then more
        few = [(s, t, 0.4, 0.0 if ty else 1.1, 0.0) for s, t, ty in graph]
        many = [(s, t, 1.0, 0.9, 0.25) for s, t, _ in graph]
        for b in (few, many):
            rows.set_couplings(b)
            monkeypatch.setenv("AED_MOM_WALK", "1")
            walk.set_couplings(b)
            monkeypatch.delenv("AED_MOM_WALK")
            _same(rows, walk, 4)
        rows.close()
        walk.close()
