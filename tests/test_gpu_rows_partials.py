"""The <x, y> partials of the rows apply where a block has several 2048-row tiles: alpha, beta and the next vector of a
Lanczos step equal the tile apply's, bit for bit (needs a B200)."""

import numpy as np
import pytest

import alps_b200 as ed

pytestmark = pytest.mark.gpu


def _step(monkeypatch, variant, n, n_up, bonds, precision, vecs):
    monkeypatch.setenv("AED_HV_VARIANT", str(variant))
    ham = ed.Hamiltonian(n, n_up, bonds, precision=precision)
    a, b, c = ham.new_vector().upload(vecs[0]), ham.new_vector().upload(vecs[1]), ham.new_vector()
    try:
        ham.time_apply(b, c, 1, variant, True)
    except ed.AEDError as e:
        assert "does not fit this sector" in str(e)
        return None
    out = (*ham.lanczos_step(a, b, c, 0.3), c.download())
    ham.close()
    return out


# largest blocks of 1716 rows (one tile), 3432 (two; also an odd number of sites), 12870 (seven, the most)
@pytest.mark.parametrize("n,n_up", [(26, 8), (27, 8), (28, 9), (32, 8)])
@pytest.mark.parametrize("precision", [ed.FP64, ed.FP32])
def test_steps_of_the_rows_applies_equal_the_tile_applys(n, n_up, precision, monkeypatch):
    rng = np.random.default_rng(n)
    bonds = [(i, (i + d) % n, *rng.uniform(-1, 1, 2)) for i in range(n) for d in (1, 5)]
    names = ed.apply_variants()
    dim = ed.Hamiltonian(n, n_up, bonds, precision=precision).dim
    vecs = rng.normal(size=(2, dim)) / np.sqrt(dim)
    want = _step(monkeypatch, 0, n, n_up, bonds, precision, vecs)
    ran = []
    for v, name in enumerate(names):
        got = _step(monkeypatch, v, n, n_up, bonds, precision, vecs) if name.startswith("row") else None
        if got is not None:
            ran.append(name)
            assert got[:2] == want[:2] and np.array_equal(got[2], want[2]), name
    assert any(r.startswith("row16") for r in ran) and any(r.startswith("row8") for r in ran), ran
