"""The stored momentum rows at the sizes of their scan and at the limit of their elements (needs a B200)."""

import numpy as np
import pytest

import alps_b200 as ed
from test_gpu_mom_rows import _pair, _same

pytestmark = pytest.mark.gpu


# slices of 32 rows: 6501, less than one pass of the scan over their widths (8192), and 12501, two
@pytest.mark.parametrize("n,n_up", [(25, 12), (26, 13)])
def test_rows_of_many_slices_equal_the_walk(n, n_up, monkeypatch):
    params = {"MODEL": "spin", "LATTICE": "chain lattice", "L": n}
    bonds = [(i, (i + d) % n, 1.0 / d, 1.0 / d) for i in range(n) for d in (1, 2)]
    rows, walk = _pair(monkeypatch, n, n_up, bonds,
                       translations=ed.lattice_translations(params, (2.0 * np.pi * 3 / n,)))
    _same(rows, walk, n)


# 64 distinct elements, the most that rows hold, and 68, which the walk takes
@pytest.mark.parametrize("own", [4, 8])
def test_elements_up_to_the_limit_and_beyond(own, monkeypatch):
    n, rng = 18, np.random.default_rng(5)
    shift = lambda i: (i + n // 2) % n
    bonds, seen = [], set()
    for i in range(n):
        for j in range(i + 1, n):
            key = frozenset([frozenset([i, j]), frozenset([shift(i), shift(j)])])
            if len(key) == 2 and key not in seen and len(seen) < 60:
                seen.add(key)
                c = rng.uniform(-1, 1, 2)
                bonds += [(i, j, *c), (shift(i), shift(j), *c)]
    bonds += [(i, shift(i), *rng.uniform(-1, 1, 2)) for i in range(own)]
    assert len(seen) == 60
    for phase in (1.0, -1.0):
        tr = [(1 + 0j, list(range(n))), (phase + 0j, [shift(i) for i in range(n)])]
        rows, walk = _pair(monkeypatch, n, n // 2, bonds, translations=tr)
        _same(rows, walk, own)
