"""The rows apply where its bundles, slices and lists can go wrong, against the tile apply, bit for bit (needs a B200)."""

import numpy as np
import pytest

import alps_b200 as ed

pytestmark = pytest.mark.gpu


def _bonds(kind, n, rng):
    if kind == "lo":  # every flip inside the lo part
        return [(n - 1 - i, n - 2 - i, *rng.uniform(0.5, 1.5, 2)) for i in range(5)]
    if kind == "hi":  # every flip inside the hi part
        return [(0, 1, 0.9, 1.1), (1, 2, 0.7, 0.6), (0, 2, 0.3, -0.4)]
    if kind == "cross":  # every flip across the parts
        return [(i, n - 1 - j, *rng.uniform(0.5, 1.5, 2)) for i in range(2) for j in range(3)]
    if kind == "ring":
        return [(i, (i + 1) % n, *rng.uniform(-1.5, 1.5, 2)) for i in range(n)]
    return [(i, j, *rng.uniform(-1.0, 1.0, 2)) for i in range(n) for j in range(i + 1, n) if (i + j) % 2][:128]  # dense


# one hi block and few rows, blocks of 1 row, fewer blocks than a bundle, half filling, a nearly empty sector,
# several 2048-row tiles per block
@pytest.mark.parametrize("n,n_up", [(3, 1), (14, 1), (15, 7), (16, 14), (18, 9), (21, 5), (24, 12), (26, 13)])
@pytest.mark.parametrize("kind", ["lo", "hi", "cross", "ring", "dense"])
def test_rows_apply_equals_the_tile_apply(n, n_up, kind):
    rng = np.random.default_rng(n * 10 + n_up)
    if n < 14 and kind != "ring":
        pytest.skip("the bond lists need 14 sites")
    bonds = _bonds(kind, n, rng)
    names = ed.apply_variants()
    for precision in (ed.FP64, ed.FP32):
        ham = ed.Hamiltonian(n, n_up, bonds, precision=precision)
        x, y = ham.new_vector(), ham.new_vector()
        v = rng.normal(size=ham.dim)
        x.upload(v)
        ham.time_apply(x, y, 1, 0, True)
        want = y.download()
        for i, name in enumerate(names):
            if not name.startswith("row"):
                continue
            y.upload(np.full(ham.dim, 3.0))
            try:
                ham.time_apply(x, y, 1, i, True)
            except ed.AEDError:
                continue  # its shared memory does not fit
            assert np.array_equal(y.download(), want), (name, precision)


def test_rows_apply_keeps_infinities_to_their_rows():
    """A row that does not reach an infinite x_j stays finite, whatever its padding and null terms."""
    n, n_up = 16, 8
    rng = np.random.default_rng(3)
    bonds = _bonds("ring", n, rng)
    names = ed.apply_variants()
    for precision in (ed.FP64, ed.FP32):
        ham = ed.Hamiltonian(n, n_up, bonds, precision=precision)
        x, y = ham.new_vector(), ham.new_vector()
        v = rng.normal(size=ham.dim)
        v[[0, 17, 4000, ham.dim - 1]] = np.inf
        v[9000] = np.nan
        x.upload(v)
        ham.time_apply(x, y, 1, 0, False)
        want = y.download()
        assert np.isfinite(want).sum() > ham.dim // 2
        for i, name in enumerate(names):
            if name.startswith("row"):
                ham.time_apply(x, y, 1, i, False)
                assert np.array_equal(y.download(), want, equal_nan=True), (name, precision)


@pytest.mark.parametrize("n_up", [9, 17])
def test_drawn_bundles_are_each_taken_once_apply_after_apply(n_up):
    """Sectors of many bundles per CTA, where CTAs draw their bundles: several applies in a row, odd ones on new states."""
    n = 26
    rng = np.random.default_rng(n_up)
    bonds = _bonds("ring", n, rng)
    names = ed.apply_variants()
    for precision in (ed.FP64, ed.FP32):
        ham = ed.Hamiltonian(n, n_up, bonds, precision=precision)
        x, y = ham.new_vector(), ham.new_vector()
        for reps in (1, 4):
            x.upload(rng.normal(size=ham.dim))
            ham.time_apply(x, y, 1, 0, True)
            want = y.download()
            for i, name in enumerate(names):
                if not name.startswith("row"):
                    continue
                y.upload(np.full(ham.dim, 3.0))
                try:
                    ham.time_apply(x, y, reps, i, True)
                except ed.AEDError:
                    continue  # its shared memory does not fit
                assert np.array_equal(y.download(), want), (name, precision)
