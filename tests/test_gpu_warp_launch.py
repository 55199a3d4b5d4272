"""GPU parity of the warp kernels at their launch edges: leaf pairs walked two
at a time (one pair only at depth 1), CTAs from one warp to the full width as
the items go from fewer than the SMs to several rounds per warp, and the block
scan over row sizes, depths and key groups.  Shares are
exact: the oracle's bytes."""
import numpy as np
import pytest

from conftest import oracle_keypair

from morphogen_b200 import gpu_dpf as G
from morphogen_b200 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("row_bytes", [16, 32])
@pytest.mark.parametrize("M", [1, 2, 3])
@pytest.mark.parametrize("items", [1, 2, 147, 148, 149, 297, 148 * 20, 148 * 20 + 1])
def test_own_rows_cta_widths(scanner, oracle_mod, row_bytes, M, items):
    nrows = items * (32 << M) - 3  # the last warp tile is ragged
    d = max(M + 1, (nrows - 1).bit_length())
    db = G.GpuPageMatrix.from_seed(scanner, nrows, row_bytes, seed=items)
    host = oracle_mod.fill_splitmix(0, nrows * row_bytes, items).reshape(nrows, row_bytes)
    key = oracle_keypair(oracle_mod, d, nrows - 1, seed=90, i=items)[0]
    ws = scanner.workspace()
    ws.set_kernel("warp")
    ws.set_shape(M + 5, 1)
    ws.set_keys([db], [key])
    ws.launch()
    assert ws.read() == oracle_mod.scan_fused([key], host, row_bytes)
    plan = ws.plan()
    assert plan["kernel"] == N.KERNEL_WARP and plan["items"] == items
    assert plan["grid"] <= scanner.device_info()["sm_count"]
    ws.close()
    db.close()


@pytest.mark.parametrize("row_bytes", [32, 48, 256])
@pytest.mark.parametrize("per_cta,extra", [(2, 1), (5, -1), (6, 0), (12, 5), (80, 0), (80, 1)])
def test_scheduler_queues_cover_every_item(scanner, oracle_mod, row_bytes, per_cta, extra):
    # Items that do not divide into four queues, and both sides of the line
    # (80 per CTA of 20 warps, 64 of 16) where the CTAs go over to one queue.
    G_ = 1 if row_bytes == 32 else 3
    per_cta = 64 if per_cta == 80 and G_ == 3 else per_cta
    sms = scanner.device_info()["sm_count"]
    items = per_cta * sms + extra
    nrows = items * 64 - 5
    d = max(7, (nrows - 1).bit_length())
    db = G.GpuPageMatrix.from_seed(scanner, nrows, row_bytes, seed=items)
    host = oracle_mod.fill_splitmix(0, nrows * row_bytes, items).reshape(nrows, row_bytes)
    keys = [oracle_keypair(oracle_mod, d, (nrows - 1) // (j + 1), seed=97, i=items + j)[0] for j in range(G_)]
    ws = scanner.workspace()
    ws.set_shape(6, G_)
    ws.set_keys([db] * G_, keys)
    plan = ws.plan()
    assert plan["items"] == items and plan["grid"] <= sms
    want = oracle_mod.scan_fused(keys, host, row_bytes)
    for graph in (False, True):
        ws.launch(graph=graph)
        assert ws.read() == want
    ws.close()
    db.close()


@pytest.mark.parametrize("row_bytes", [48, 80, 112, 128, 192, 256, 272, 496, 512])
@pytest.mark.parametrize("M,keys_per_item,nkeys", [(1, 3, 4), (2, 3, 3), (3, 3, 7), (4, 1, 2), (5, 2, 3), (9, 3, 3)])
def test_block_scan_shapes(scanner, oracle_mod, row_bytes, M, keys_per_item, nkeys):
    # Row sizes with every number of rows per warp-wide load from 10 to 1, a
    # key group left over (fewer keys than the kernel's), a row range that
    # starts and ends inside a warp tile.
    d, first, nrows = 18, 12_345, 2 * (32 << M) + 77
    db = G.GpuPageMatrix.from_seed(scanner, nrows, row_bytes, seed=M, first_row=first)
    host = oracle_mod.fill_splitmix(first * row_bytes, nrows * row_bytes, M).reshape(nrows, row_bytes)
    keys = [oracle_keypair(oracle_mod, d, first + (7919 * j) % nrows, seed=91, i=j)[0] for j in range(nkeys)]
    ws = scanner.workspace()
    ws.set_shape(M + 5, keys_per_item)
    ws.set_keys([db] * nkeys, keys)
    assert ws.plan()["kernel"] == N.KERNEL_WARP
    want = oracle_mod.scan_fused(keys, host, row_bytes, row_base=first)
    for graph in (False, True, True):
        ws.launch(graph=graph)
        assert ws.read() == want
    ws.close()
    db.close()


def test_row_sizes_beside_each_other_keep_their_own_keys_per_item(scanner, oracle_mod):
    # One pass over 32-, 48-, 64- and 256-B tables (and 528 B on the CTA kernel).
    tabs, keys, want = [], [], []
    for i, (rb, n) in enumerate([(32, 5000), (48, 3001), (64, 4097), (256, 700), (528, 300)]):
        host = oracle_mod.fill_splitmix(0, n * rb, 30 + i).reshape(n, rb)
        t = G.GpuPageMatrix.from_seed(scanner, n, rb, seed=30 + i)
        for j in range(4):
            k = oracle_keypair(oracle_mod, 13, (j * 911) % n, seed=92, i=4 * i + j)[0]
            tabs.append(t)
            keys.append(k)
            want += oracle_mod.scan_fused([k], host, rb)
    assert scanner.scan_multi(list(zip(tabs, keys))) == want


def test_pinning_the_warp_kernel_still_needs_a_power_of_two_row(scanner):
    db = G.GpuPageMatrix.alloc_empty(scanner, 100, 48)
    key = G.generate_chacha_dpf_keys(G.ChaChaParams(8), 3)[0]
    ws = scanner.workspace()
    ws.set_kernel("warp")
    with pytest.raises(N.MgError):
        ws.set_keys([db], [key])
    ws.close()


@pytest.mark.parametrize("d,M,first,nrows", [
    (23, 1, 5, 4_194_304),          # 11 levels per CTA, the last three depth first
    (20, 3, 0, 1_000_000),          # 10 or 11
    (26, 4, 1 << 25, 300_001),      # walk from the root to a range in the middle
    (9, 1, 0, 512), (9, 8, 0, 512), (9, 9, 0, 512),  # 8, 1 and 0 frontier levels
    (32, 1, (1 << 32) - 3001, 3001),
])
def test_frontier_levels_per_cta(scanner, oracle_mod, d, M, first, nrows):
    # The levels a frontier CTA expands (and so its walk) follow the number of
    # nodes; keys with non-binary t correction bytes take the same path.
    db = G.GpuPageMatrix.from_seed(scanner, nrows, 16, seed=d, first_row=first)
    host = oracle_mod.fill_splitmix(first * 16, nrows * 16, d).reshape(nrows, 16)
    keys = [oracle_keypair(oracle_mod, d, first + (12_347 * j) % nrows, seed=93, i=j)[0] for j in range(2)]
    odd = bytearray(keys[1])
    for lvl in range(0, d, 3):
        odd[19 + 18 * lvl + 16] ^= 2  # left t byte 2 or 3
    keys.append(bytes(odd))
    ws = scanner.workspace()
    ws.set_kernel("warp")
    ws.set_shape(M + 5, 1)
    ws.set_keys([db] * 3, keys)
    ws.launch()
    assert ws.read() == oracle_mod.scan_fused(keys, host, 16, row_base=first)
    ws.close()
    db.close()


@pytest.mark.parametrize("row_bytes,keys_per_cta", [(528, 1), (528, 3), (1024, 2), (2048, 4), (1040, 8)])
def test_cta_kernel_with_several_tiles_per_cta(scanner, oracle_mod, row_bytes, keys_per_cta):
    # More tiles than CTAs: the tiles' roots come from a frontier.
    d, first, nrows, nkeys = 24, 1_000_001, 120_007, 9
    db = G.GpuPageMatrix.from_seed(scanner, nrows, row_bytes, seed=7, first_row=first)
    host = oracle_mod.fill_splitmix(first * row_bytes, nrows * row_bytes, 7).reshape(nrows, row_bytes)
    keys = [oracle_keypair(oracle_mod, d, first + (7919 * j) % nrows, seed=94, i=j)[0] for j in range(nkeys)]
    ws = scanner.workspace()
    ws.set_kernel("cta")
    ws.set_shape(8, keys_per_cta)
    ws.set_keys([db] * nkeys, keys)
    plan = ws.plan()
    assert plan["kernel"] == N.KERNEL_CTA and plan["items"] > plan["grid"] and plan["frontier_nodes"] > 0
    want = oracle_mod.scan_fused(keys, host, row_bytes, row_base=first)
    for graph in (False, True):
        ws.launch(graph=graph)
        assert ws.read() == want
    ws.close()
    db.close()


@pytest.mark.parametrize("row_bytes,nrows,kind", [(32, 70_001, "auto"), (48, 20_011, "auto"), (256, 9_001, "auto"),
                                                  (4096, 300, "auto"), (528, 120_007, "cta"), (64, 33, "auto")])
def test_delta_entries_start_from_the_pass_frontier(scanner, oracle_mod, row_bytes, nrows, kind):
    # Pending entries (first and last row, duplicates) are evaluated from their
    # rows' ancestors in the frontier, or from the root when the pass has none.
    d, first = 23, 4_000_003
    db = G.GpuPageMatrix.from_seed(scanner, nrows, row_bytes, seed=8, first_row=first)
    host = oracle_mod.fill_splitmix(first * row_bytes, nrows * row_bytes, 8).reshape(nrows, row_bytes).copy()
    keys = [oracle_keypair(oracle_mod, d, first + (7919 * j) % nrows, seed=95, i=j)[0] for j in range(4)]
    rng = np.random.default_rng(row_bytes)
    idx = np.concatenate([[0, nrows - 1, nrows // 2, nrows // 2], rng.integers(0, nrows, 700)]).astype(np.uint64)
    diffs = rng.integers(0, 256, idx.size * row_bytes, dtype=np.uint8).reshape(-1, row_bytes)
    np.bitwise_xor.at(host, idx.astype(np.int64), diffs)
    db.delta_reserve(1000)
    db.delta_push(idx, diffs)
    ws = scanner.workspace()
    ws.set_kernel(kind)
    if kind == "cta":
        ws.set_shape(8, 3)
    ws.set_keys([db] * 4, keys)
    want = oracle_mod.scan_fused(keys, host, row_bytes, row_base=first)
    for graph in (False, True):
        ws.launch(graph=graph)
        assert ws.read() == want
    ws.close()
    db.close()


@pytest.mark.parametrize("row_bytes", [48, 496])
@pytest.mark.parametrize("subtree_bits,keys_per_item", [(1, 1), (5, 3), (16, 1), (0, 8), (12, 8)])
def test_cta_shapes_of_rows_that_are_no_power_of_two(scanner, oracle_mod, row_bytes, subtree_bits, keys_per_item):
    d, first, nrows, nkeys = 18, 12_345, 9_001, 9
    db = G.GpuPageMatrix.from_seed(scanner, nrows, row_bytes, seed=6, first_row=first)
    host = oracle_mod.fill_splitmix(first * row_bytes, nrows * row_bytes, 6).reshape(nrows, row_bytes)
    keys = [oracle_keypair(oracle_mod, d, first + (7919 * j) % nrows, seed=98, i=j)[0] for j in range(nkeys)]
    ws = scanner.workspace()
    ws.set_shape(subtree_bits, keys_per_item)
    ws.set_keys([db] * nkeys, keys)
    assert ws.plan()["kernel"] == N.KERNEL_CTA
    want = oracle_mod.scan_fused(keys, host, row_bytes, row_base=first)
    for graph in (False, True):
        ws.launch(graph=graph)
        assert ws.read() == want
    ws.close()
    db.close()
