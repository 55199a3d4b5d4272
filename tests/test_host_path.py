"""Host path of the library on a CPU (see fake_device.py): workspaces, graph
reuse, planning and memory limits.  Nothing is computed here; what is checked
is which memory a launch is given, and which calls are taken or refused."""
import ctypes as C

import pytest

import fake_device
from morphogen_b200 import _native as N
from morphogen_b200 import gpu_dpf as G
from morphogen_b200.server import PirServer


@pytest.fixture(scope="module")
def fake_path():
    return fake_device.build()


@pytest.fixture
def fake(fake_path):
    with fake_device.fake_library(fake_path) as L:
        L.fake_reset(178 * fake_device.GIB, 0)
        yield L


@pytest.fixture
def fscanner(fake):
    s = G.GpuScanner(0)
    yield s
    s.close()
    s._ctx.close()  # now, with this library: pytest may keep the scanner longer


def key(d, target=0):
    return G.generate_chacha_dpf_keys(G.ChaChaParams(d), target)[0].to_bytes()


def delta_args(L):
    """Job list, entry indices, entry rows and count of the last delta launch."""
    out = (C.c_uint64 * 4)()
    L.fake_last_delta(out)
    return tuple(out)


def test_replayed_graphs_never_read_a_freed_job_list(fake, fscanner):
    # 24 keys size the workspace before the table has a delta buffer; with one,
    # 3 keys are captured, 24 keys need a longer job list, and the 3 keys' next
    # replay must not use the first list.
    t = G.GpuPageMatrix.alloc_empty(fscanner, 70_001, 32)
    keys = [key(17, i) for i in range(24)]
    fscanner.scan_keys(t, keys)
    t.delta_reserve(100)
    for n in (3, 3, 24, 3, 3, 24, 24, 3, 3):
        fscanner.scan_keys(t, keys[:n])
        assert fake.fake_dead_launches() == 0, f"{n} keys"
    ws = fscanner.workspace()
    ws.set_keys([t] * 3, keys[:3])
    ws.launch(graph=True)
    for n in (24, 3):
        ws.set_keys([t] * n, keys[:n])
    ws.launch(graph=True)
    graph = delta_args(fake)
    ws.launch()
    assert graph == delta_args(fake) and fake.fake_dead_launches() == 0
    ws.close()
    t.close()


@pytest.mark.parametrize("fails", [1 << i for i in range(4)] + [2**64 - 1, 2**64 - 2])
def test_a_failed_growth_leaves_nothing_launchable(fake, fscanner, fails):
    t = G.GpuPageMatrix.alloc_empty(fscanner, 5000, 32)
    t.delta_reserve(10)
    keys = [key(13, i) for i in range(40)]
    ws = fscanner.workspace()
    ws.set_keys([t] * 2, keys[:2])
    ws.launch()
    fake.fake_fail(fails)
    try:
        ws.set_keys([t] * 40, keys)
    except N.MgError as e:
        assert e.code == N.MG_ENOMEM
        for call in (ws.launch, lambda: ws.launch(graph=True), ws.plan, ws.read):
            with pytest.raises(N.MgError) as err:
                call()
            assert err.value.code == N.MG_EINVAL
    fake.fake_fail(0)
    ws.set_keys([t] * 40, keys)
    ws.launch()
    ws.launch(graph=True)
    assert len(ws.read()) == 40 and fake.fake_dead_launches() == 0
    ws.close()
    t.close()


@pytest.mark.parametrize("call", ["scan", "workspace"])
def test_graphs_follow_a_delta_buffer_that_keeps_its_index_address(fake, fscanner, call):
    # A buffer of 8, 16, then 8 entries again: the index array gets its first
    # address back, the row array, whose memory a table took meanwhile, does not.
    fake.fake_reset(178 * fake_device.GIB, 1)
    t = G.GpuPageMatrix.alloc_empty(fscanner, 5000, 48)
    ws = fscanner.workspace()
    keys = [key(13, i) for i in range(3)]

    def run():
        if call == "scan":
            for _ in range(3):
                fscanner.scan_keys(t, keys)
        else:
            ws.set_keys([t] * 3, keys)
            ws.launch(graph=True)
        replayed = delta_args(fake)
        ws.set_keys([t] * 3, keys)
        ws.launch()
        return replayed[1:], delta_args(fake)[1:]

    t.delta_reserve(8)
    first, direct = run()
    assert first == direct
    t.delta_reserve(16)
    other = G.GpuPageMatrix.alloc_empty(fscanner, 8, 48)
    t.delta_reserve(8)
    again, direct = run()
    assert direct[0] == first[0] and direct[1] != first[1]
    assert again == direct and fake.fake_dead_launches() == 0
    ws.close()
    other.close()
    t.close()


@pytest.mark.parametrize("rows,row_bytes", [(12_000, 128), (30_000, 32), (30_000, 64), (60_000, 128), (140_000, 128),
                                            (100_003, 48), (20_000, 256)])
def test_narrow_scans_of_two_passes_fit_one_sm(fake, fscanner, rows, row_bytes):
    # CTAs of a few warps take the shared memory they use and no more, so that
    # passes of two workspaces can share the SMs.
    t = G.GpuPageMatrix.alloc_empty(fscanner, rows, row_bytes)
    ws = fscanner.workspace()
    ws.set_keys([t] * 3, [key(18, i) for i in range(3)])
    plan = ws.plan()
    assert plan["kernel"] == N.KERNEL_WARP and plan["grid"] <= 148
    assert 2 * (plan["smem_bytes"] + 1024) <= 228 * 1024
    ws.close()
    t.close()


@pytest.mark.parametrize("row_bytes", [48, 80, 496])
@pytest.mark.parametrize("subtree_bits,keys_per_item", [(1, 1), (5, 3), (16, 1), (16, 0), (20, 1), (0, 8), (9, 8)])
def test_shapes_the_warp_kernel_cannot_take_run_on_the_cta_kernel(fake, fscanner, row_bytes, subtree_bits, keys_per_item):
    # Items of 2^1..2^5 or more than 2^15 rows, or of eight keys, were valid
    # for every row size that is no power of two: as CTA tiles.
    t = G.GpuPageMatrix.alloc_empty(fscanner, 1 << 20, row_bytes)
    ws = fscanner.workspace()
    ws.set_shape(subtree_bits, keys_per_item)
    ws.set_keys([t] * 8, [key(20, i) for i in range(8)])
    plan = ws.plan()
    assert plan["kernel"] == N.KERNEL_CTA
    assert plan["subtree_bits"] == subtree_bits or not subtree_bits
    assert plan["keys_per_cta"] == keys_per_item or not keys_per_item
    ws.launch()
    ws.set_shape(0, 0)
    ws.set_keys([t] * 8, [key(20, i) for i in range(8)])
    assert ws.plan()["kernel"] == N.KERNEL_WARP
    ws.close()
    t.close()


@pytest.mark.parametrize("row_bytes", [48, 80, 496])
@pytest.mark.parametrize("subtree_bits,keys_per_item", [(6, 1), (15, 1), (9, 3), (0, 4)])
def test_shapes_the_warp_kernel_takes_stay_on_it(fake, fscanner, row_bytes, subtree_bits, keys_per_item):
    t = G.GpuPageMatrix.alloc_empty(fscanner, 1 << 20, row_bytes)
    ws = fscanner.workspace()
    ws.set_shape(subtree_bits, keys_per_item)
    ws.set_keys([t] * 4, [key(20, i) for i in range(4)])
    plan = ws.plan()
    assert plan["kernel"] == N.KERNEL_WARP
    assert plan["subtree_bits"] == subtree_bits or not subtree_bits
    assert plan["keys_per_cta"] == keys_per_item
    ws.close()
    t.close()


def scratch(rows, row_bytes, nkeys):
    """Device bytes that nkeys over a table are admitted with: keys, a frontier
    node for 2 rows, or for 256 of tables above 2^24 rows, and partial rows of
    32 warps per SM."""
    frontier = rows // 2 if rows <= 1 << 24 else rows >> 8
    return nkeys * (1264 + 17 * (frontier + 32) + 148 * 32 * row_bytes)


BIG = [(37_000_000, 512, 2), (340_000_000, 512, 1), (340_000_000, 512, 24), (690_000_000, 256, 48), (2_200_000_000, 80, 3),
       (1 << 26, 512, 48), (1 << 28, 128, 1), (1 << 26, 32, 1), (1 << 30, 32, 1), (1 << 31, 32, 48), (1 << 25, 16, 48)]


@pytest.mark.parametrize("rows,row_bytes,nkeys", BIG)
def test_a_pass_fits_the_memory_it_is_admitted_with(fake, fscanner, rows, row_bytes, nkeys):
    d = (rows - 1).bit_length()
    keys = [key(d, i) for i in range(nkeys)]
    room = scratch(rows, row_bytes, nkeys)
    fake.fake_reset(rows * row_bytes + room, 0)
    t = G.GpuPageMatrix.alloc_empty(fscanner, rows, row_bytes)
    ws = fscanner.workspace()
    ws.set_keys([t] * nkeys, keys)
    tight = ws.plan()
    ws.launch()
    ws.launch(graph=True)
    assert fake.fake_dead_launches() == 0
    ws.close()
    # With memory to spare the plan is the planner's own choice.
    fake.fake_reset(rows * row_bytes + (1 << 42), 0)
    ws = fscanner.workspace()
    ws.set_keys([t] * nkeys, keys)
    assert ws.plan()["subtree_bits"] <= tight["subtree_bits"]
    ws.close()
    t.close()


@pytest.mark.parametrize("rows,row_bytes,nkeys", BIG)
@pytest.mark.parametrize("spare", [4, 40])
def test_a_workspace_leaves_most_of_the_free_memory_alone(fake, fscanner, rows, row_bytes, nkeys, spare):
    d = (rows - 1).bit_length()
    free = spare << 30
    fake.fake_reset(rows * row_bytes + free, 0)
    t = G.GpuPageMatrix.alloc_empty(fscanner, rows, row_bytes)
    before = fake.fake_used()
    ws = fscanner.workspace()
    ws.set_keys([t] * nkeys, [key(d, i) for i in range(nkeys)])
    assert fake.fake_used() - before <= max(free // 4, scratch(rows, row_bytes, nkeys))
    ws.close()
    t.close()


@pytest.mark.parametrize("subtree_bits", [1, 3, 8])
def test_pinned_cta_tiles_need_no_frontier_when_it_does_not_fit(fake, fscanner, subtree_bits):
    rows, keys = 1 << 30, [key(30, i) for i in range(2)]
    fake.fake_reset(rows * 64 + (64 << 20), 0)
    t = G.GpuPageMatrix.alloc_empty(fscanner, rows, 64)
    ws = fscanner.workspace()
    ws.set_kernel("cta")
    ws.set_shape(subtree_bits, 1)
    ws.set_keys([t] * 2, keys)
    plan = ws.plan()
    assert plan["subtree_bits"] == subtree_bits and plan["frontier_nodes"] == 0
    ws.launch()
    assert fake.fake_dead_launches() == 0
    ws.close()
    t.close()


@pytest.mark.parametrize("rows,row_bytes,nkeys", BIG)
@pytest.mark.parametrize("slots", [1, 2])
def test_a_server_keeps_its_memory_reserve(fake, fscanner, rows, row_bytes, nkeys, slots):
    # Budget for a third of the requests at once: passes take as many as are
    # admitted, none fails and the reserve is never touched.
    d, lookups = (rows - 1).bit_length(), max(3, nkeys)
    reserve, budget = 1 << 30, slots * (scratch(rows, row_bytes, (lookups + 2) // 3) + (1 << 20))
    fake.fake_reset(rows * row_bytes + budget + reserve, 0)
    t = G.GpuPageMatrix.alloc_empty(fscanner, rows, row_bytes)
    srv = PirServer(fscanner, slots=slots, max_keys_per_pass=lookups, memory_reserve=reserve)
    ids = [srv.submit([(t, key(d, i))]) for i in range(lookups)]
    for i in ids:
        assert len(srv.wait(i, 20_000)[0]) == 1
    stats = srv.stats()
    srv.close()
    assert stats["completed"] == lookups and stats["failed"] == 0
    assert fake.fake_peak() <= rows * row_bytes + budget
    t.close()


@pytest.mark.parametrize("slots", [1, 2])
def test_a_server_splits_a_pass_that_finds_no_memory(fake, fscanner, slots):
    # Device memory that others take between the admission and the pass: all
    # of the pass's tries fail (and, later, those of its half).
    t = G.GpuPageMatrix.alloc_empty(fscanner, 5000, 32)
    srv = PirServer(fscanner, slots=slots, max_keys_per_pass=12)
    srv.pause()
    ids = [srv.submit([(t, key(13, i))]) for i in range(24)]
    fake.fake_fail((1 << 20) - 1)
    srv.resume()
    for i in ids:
        assert len(srv.wait(i, 20_000)[0]) == 1
    stats = srv.stats()
    assert stats["completed"] == 24 and stats["failed"] == 0 and stats["passes"] >= 3
    srv.close()
    # One request alone that finds none is answered with the error.
    srv = PirServer(fscanner, slots=slots)
    fake.fake_reset(fake.fake_used(), 0)
    with pytest.raises(N.MgError) as err:
        srv.wait(srv.submit([(t, key(13, 0))]), 20_000)
    assert err.value.code == N.MG_ENOMEM
    srv.close()
    t.close()


@pytest.mark.parametrize("row_bytes", [48, 496])
@pytest.mark.parametrize("subtree_bits,keys_per_item", [(6, 0), (6, 1), (7, 3), (9, 2)])
def test_pinned_items_without_room_for_their_frontier_run_on_the_cta_kernel(fake, fscanner, row_bytes, subtree_bits, keys_per_item):
    # A pinned depth cannot be walked deeper, but the CTA kernel has the same
    # items and needs no frontier.
    rows, nkeys = 200_000_003, 24
    keys = [key(28, i) for i in range(nkeys)]
    room = 24 * 148 * 32 * row_bytes + (16 << 20)
    fake.fake_reset(rows * row_bytes + room, 0)
    t = G.GpuPageMatrix.alloc_empty(fscanner, rows, row_bytes)
    for spare, kernel in ((0, N.KERNEL_CTA), (1 << 42, N.KERNEL_WARP)):
        fake.fake_reset(rows * row_bytes + room + spare, 0)
        ws = fscanner.workspace()
        ws.set_shape(subtree_bits, keys_per_item)
        ws.set_keys([t] * nkeys, keys)
        plan = ws.plan()
        assert plan["kernel"] == kernel and plan["subtree_bits"] == subtree_bits
        assert plan["keys_per_cta"] == keys_per_item or not keys_per_item
        ws.launch()
        ws.launch(graph=True)
        assert fake.fake_dead_launches() == 0
        ws.close()
    t.close()


@pytest.mark.parametrize("rows,row_bytes", [(3_600_000_003, 48), (500_000_001, 336)])
@pytest.mark.parametrize("shape", [(0, 0), (0, 3)])
def test_rows_that_are_no_power_of_two_need_no_frontier_when_none_fits(fake, fscanner, rows, row_bytes, shape):
    nkeys, d = 48, (rows - 1).bit_length()
    fake.fake_reset(rows * row_bytes + (256 << 20), 0)
    t = G.GpuPageMatrix.alloc_empty(fscanner, rows, row_bytes)
    ws = fscanner.workspace()
    ws.set_shape(*shape)
    ws.set_keys([t] * nkeys, [key(d, i) for i in range(nkeys)])
    plan = ws.plan()
    assert plan["kernel"] == N.KERNEL_CTA and plan["frontier_nodes"] == 0
    ws.launch()
    ws.launch(graph=True)
    assert fake.fake_dead_launches() == 0
    ws.close()
    t.close()
