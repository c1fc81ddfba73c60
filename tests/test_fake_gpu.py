"""Host code of the engine that a single GPU cannot show: limits per device, the tuner's choice, admission to the
batch.  On a fake CUDA runtime (fake_gpu.py); no GPU."""

import pytest

import fake_gpu


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    return fake_gpu.link(str(tmp_path_factory.mktemp("fake")))


CHAINS = """
def chain(n):
    return [(i, (i + 1) % n, 1.0, 1.0) for i in range(n)]
def product(ham):
    x, y = ham.new_vector(), ham.new_vector()
    ham.mult(x, y)
    x.free(); y.free()
"""


@pytest.mark.parametrize("make", ["ed.Hamiltonian(28, 14, chain(28), device=dev)",  # 55 KB of x rows
                                  "ed.Hamiltonian(30, 15, chain(30), precision=ed.FP32, device=dev)",
                                  "ed.Hamiltonian(16, 8, chain(16), device=dev)",
                                  "ed.Hamiltonian(18, 18, chain(18), two_s=2, device=dev)"])
def test_products_on_the_second_device_of_a_process(lib, make):
    """A kernel's limit of dynamic shared memory belongs to a device: a handle on another one raises it there too."""
    fake_gpu.run(lib, CHAINS + f"""
fake.fake_set_cost(b"9hv_kernel", 1.0)  # the tuner takes a rows apply
for dev in (0, 1, 0):
    ham = {make}
    product(ham)
    ham.close()
""")


def test_servers_on_two_devices_of_a_process(lib):
    fake_gpu.run(lib, CHAINS + """
servers = [ed.Server(precision=ed.FP64, device=dev, max_slots=2, lane_min_dim=-1) for dev in (0, 1)]
tickets = [s.submit(28, 14, chain(28), nev=1) for s in servers]
for s, t in zip(servers, tickets):
    s.step()
    s.cancel(t)
    s.close()
""")


@pytest.mark.parametrize("tile,rows,want", [(1.0, 1.04, "hvr_kernel"), (1.0, 1.0, "hvr_kernel"),
                                            (1.04, 1.0, "hvr_kernel"), (1.0, 1.1, "hv_kernel"), (0.0, 0.0, "hvr_kernel")])
def test_the_tile_apply_wins_no_near_tie(lib, tile, rows, want):
    """The tuner takes the tile apply only where it is more than 5 % faster than every rows apply."""
    fake_gpu.run(lib, CHAINS + f"""
fake.fake_set_cost(b"9hv_kernel", {tile})
fake.fake_set_cost(b"hvr_kernel", {rows})
for precision in (ed.FP64, ed.FP32):
    ham = ed.Hamiltonian(16, 8, chain(16), precision=precision)
    product(ham)
    before = fake.fake_launches(b"{want}")
    product(ham)
    assert fake.fake_launches(b"{want}") == before + 1
""")


OVERFLOW = """
over = lambda n: chain(n) + [(0, 1, 0.0, 1.5e308)] * 4  # finite couplings whose merged flip is not
fake.fake_set_cost(b"9hv_kernel", 1.0)
def takes(ham, kernel):
    before = fake.fake_launches(kernel)
    product(ham)
    return fake.fake_launches(kernel) > before
"""


@pytest.mark.parametrize("precision", ["ed.FP64", "ed.FP32"])
def test_a_handle_without_programs_takes_the_tile_apply(lib, precision):
    """Couplings that overflow when merged have no rows apply: the sizes that are not timed take the tile apply too,
    and the choice is neither kept for other handles nor for the handle's next couplings."""
    fake_gpu.run(lib, CHAINS + OVERFLOW + f"""
for n in (8, 16):  # not timed; timed
    odd = ed.Hamiltonian(n, n // 2, over(n), precision={precision})
    x, y = odd.new_vector(), odd.new_vector()
    assert odd.time_apply(x, y, 1)[1] == 0
    assert takes(odd, b"9hv_kernel") and not takes(odd, b"hvr_kernel")
    ham = ed.Hamiltonian(n, n // 2, chain(n), precision={precision})
    product(ham)
    assert takes(ham, b"hvr_kernel") and not takes(ham, b"9hv_kernel")
    odd.set_couplings(chain(n))
    product(odd)
    assert takes(odd, b"hvr_kernel") and not takes(odd, b"9hv_kernel")
    odd.set_couplings(over(n))
    assert takes(odd, b"9hv_kernel") and not takes(odd, b"hvr_kernel")
    assert odd.time_apply(x, y, 1)[1] == 0
""")


def test_admission_to_the_batch_does_not_depend_on_what_came_before(lib):
    """The largest blocks (32 sites) beside programs of every size up to 128 bonds, one after the other."""
    fake_gpu.run(lib, CHAINS + """
srv = ed.Server(precision=ed.FP64, max_slots=200, lane_min_dim=-1)
tickets = [srv.submit(32, 8, chain(32), nev=1)]
pairs = [(i, j, 1.0, 1.0) for i in range(16) for j in range(16, 32)]
for n in range(1, 129):
    tickets.append(srv.submit(32, 2, pairs[:n], nev=1))
    srv.step()
assert all(srv.poll(t) is None for t in tickets)  # resident: none was refused
assert srv.stats()["resident"] == 129
""")


@pytest.mark.parametrize("precision", ["ed.FP64", "ed.FP32"])
def test_a_request_is_admitted_by_what_it_allocates(lib, precision):
    """The footprint holds what a resident request takes, and little more: also where few of the hi blocks exist."""
    fake_gpu.run(lib, CHAINS + f"""
pairs = [(i, j, 1.0, 1.0) for i in range(32) for j in range(i + 1, 32)]
for n, n_up, bonds in [(32, 2, chain(32)), (32, 1, pairs[:128]), (24, 12, chain(24)), (16, 8, chain(16)),
                       (12, 1, chain(12)), (4, 2, chain(4)), (30, 3, pairs[:100]), (27, 25, chain(27))]:
    bonds = [b for b in bonds if b[1] < n]
    srv = ed.Server(precision={precision}, max_slots=2, lane_min_dim=-1)
    t = srv.submit(n, n_up, bonds, nev=1, max_iter=40)
    srv.step()
    used, held = srv.stats()["bytes_used"], fake.fake_pool_bytes()
    assert held - (1 << 17) <= used <= 1.15 * held + (1 << 17), (n, n_up, used, held)  # tile lists are estimated
    srv.cancel(t)
    srv.step()
    assert srv.stats()["bytes_used"] == 0
    srv.close()
""")


def test_a_lane_is_counted_with_its_programs(lib):
    """Two requests of one sector as single-instance solves, with few and with many flips outside the lo part; and a
    budget that holds the lane but for its programs."""
    fake_gpu.run(lib, CHAINS + """
pairs = [(i, j, 1.0, 1.0) for i in range(15) for j in range(15, 30)]
def counted(bonds, budget):
    srv = ed.Server(precision=ed.FP64, max_slots=2, max_lanes=1, lane_min_dim=1000, hbm_budget=budget)
    t = srv.submit(30, 5, bonds, nev=1, max_iter=20)
    srv.step()
    assert srv.stats()["queued"] == 0
    used = srv.stats()["bytes_used"]  # 0 where the solve is over already
    srv.close()
    return used
few = max(counted(pairs[:10], 8 << 30) for _ in range(5))
many = max(counted(pairs[:120], 8 << 30) for _ in range(5))
blocks = 4944  # hi parts of 15 sites with at most 5 up spins
assert few == 0 or many == 0 or many - few > 110 * 16 * blocks
counted(pairs[:120], (64 << 20) + 142506 * (60 + 16 * 24))
""")


@pytest.mark.parametrize("precision", ["ed.FP64", "ed.FP32"])
def test_couplings_without_memory_leave_the_handle_its_tables(lib, precision):
    """New couplings whose tables find no memory are refused; the tables that a later product reads stay allocated."""
    fake_gpu.run(lib, CHAINS + f"""
ham = ed.Hamiltonian(16, 8, chain(16), precision={precision})
product(ham)
ed.empty_cache()
before = fake.fake_frees()
fake.fake_no_memory(1)
try:
    ham.set_couplings([(i, j, 1.0, 1.0) for i in range(16) for j in range(i + 1, 16)])
    assert False
except ed.AEDError as e:
    assert e.code == ed.ERR_NOMEM
assert fake.fake_frees() == before
fake.fake_no_memory(0)
ham.set_couplings(chain(16))
product(ham)
""")


@pytest.mark.parametrize("n,total,two_s", [(10, 10, 2), (18, 18, 2), (9, 13, 3), (8, 16, 4), (16, 8, 1)])
def test_spin_s_products_take_the_rows_apply(lib, n, total, two_s):
    """What the comparison with the tile apply on a GPU rests on: these sectors have a plan."""
    fake_gpu.run(lib, CHAINS + f"""
ham = ed.Hamiltonian({n}, {total}, chain({n}), two_s={two_s}, generic=True)
product(ham)
assert fake.fake_launches(b"spin_rows_kernel") == 1 and fake.fake_launches(b"spin_hv_kernel") == 0
""")


def test_twosum_rows_of_couplings_beyond_fp32_take_the_tile_apply(lib):
    """The compensated FP32 sums round the couplings to FP32, where they may overflow."""
    fake_gpu.run(lib, CHAINS + OVERFLOW + """
for n in (8, 16):
    big = chain(n) + [(0, 1, 0.0, 1e39)]
    for precision, rows in ((ed.FP32, False), (ed.FP64, True)):
        ham = ed.Hamiltonian(n, n // 2, big, precision=precision)
        product(ham)
        assert takes(ham, b"hvr_kernel") == rows and takes(ham, b"9hv_kernel") != rows
    ham = ed.Hamiltonian(n, n // 2, chain(n) + [(0, 2, 0.0, 1.0)], precision=ed.FP32)
    product(ham)
    assert takes(ham, b"hvr_kernel")
""", {"AED_FP32_ACCUM": "twosum"})
