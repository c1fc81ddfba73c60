"""A spin-S handle made with couplings that are not tabulated (more classes than the tables hold), then given ones that
are, and back: the rows apply on a block list ordered for other bonds (needs a B200)."""

import numpy as np
import pytest

import alps_b200 as ed
from test_gpu_spin_rows import EPS, _chain, _couple, _row_bound, _square

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("two_s,pairs,n,total", [(2, _chain(10), 10, 10), (2, _square(3, 3), 9, 8), (4, _chain(6), 6, 12)])
def test_untabulated_then_tabulated_couplings(two_s, pairs, n, total, monkeypatch):
    rng = np.random.default_rng(n + two_s)
    many = [(i, j, *rng.uniform(0.5, 1.5, 2), 0.0) for i, j in pairs + [(i, (i + 3) % n) for i in range(n)]]
    few = _couple(pairs, 2, two_s > 1, rng)
    made = []
    for on in ("1", "0"):
        monkeypatch.setenv("AED_SPIN_ROWS", on)
        made.append(ed.Hamiltonian(n, total, many, two_s=two_s, generic=True))
    zero = np.zeros(n)
    for bonds in (many, few, many, few):
        for h, on in zip(made, ("1", "0")):
            monkeypatch.setenv("AED_SPIN_ROWS", on)
            h.set_couplings(bonds)
        x = rng.normal(size=made[0].dim)
        tol = 8 * (len(bonds) + n) * EPS * _row_bound(bonds, zero, zero, two_s) * np.max(np.abs(x))
        y1, y0 = (h.apply(x) for h in made)
        assert np.max(np.abs(y1 - y0)) <= tol
