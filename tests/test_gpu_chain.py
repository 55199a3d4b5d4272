"""GPU parity of passes whose kernels are launched while their predecessors
still run: what one kernel of the chain writes for the next (keys, frontiers,
partial rows shared by two reductions, delta jobs) changes from pass to pass.
Shares are exact: the oracle's bytes."""
import numpy as np
import pytest

from conftest import oracle_keypair

from morphogen_b200 import gpu_dpf as G

pytestmark = pytest.mark.gpu


def make(scanner, oracle_mod, rows, row_bytes, seed):
    host = oracle_mod.fill_splitmix(0, rows * row_bytes, seed).reshape(rows, row_bytes).copy()
    return G.GpuPageMatrix.from_seed(scanner, rows, row_bytes, seed=seed), host


@pytest.mark.parametrize("graph", [False, True])
def test_every_pass_sees_its_own_keys(scanner, oracle_mod, graph):
    # 528 B (CTA kernel) and 32 B both end in a reduction over the same partial
    # rows, 256 B reduces in its scan, and the 32-B table has pending entries.
    d = 15
    tabs = [make(scanner, oracle_mod, n, rb, 40 + i) for i, (rb, n) in enumerate([(528, 20_001), (32, 30_011), (256, 9_000)])]
    rng = np.random.default_rng(5)
    idx = rng.integers(0, 30_011, 600).astype(np.uint64)
    diffs = rng.integers(0, 256, idx.size * 32, dtype=np.uint8).reshape(-1, 32)
    tabs[1][0].delta_reserve(700)
    tabs[1][0].delta_push(idx, diffs)
    np.bitwise_xor.at(tabs[1][1], idx.astype(np.int64), diffs)
    ws = scanner.workspace()
    for i in range(8):
        keys = [[oracle_keypair(oracle_mod, d, int(rng.integers(0, len(h))), seed=100 + i, i=10 * k + j)[0] for j in range(3)]
                for k, (_, h) in enumerate(tabs)]
        ws.set_keys([t for t, _ in tabs for _ in range(3)], [k for ks in keys for k in ks])
        ws.launch(graph=graph)
        want = [s for ks, (_, h) in zip(keys, tabs) for s in oracle_mod.scan_fused(ks, h, h.shape[1])]
        assert ws.read() == want, f"pass {i}"
    ws.close()
    for t, _ in tabs:
        t.close()


@pytest.mark.parametrize("row_bytes,rows", [(32, 3001), (32, 30_000), (128, 12_000), (256, 20_000)])
def test_two_workspaces_with_narrow_passes_in_flight(scanner, oracle_mod, row_bytes, rows):
    d = (rows - 1).bit_length()
    db, host = make(scanner, oracle_mod, rows, row_bytes, 60)
    wss = [scanner.workspace() for _ in range(2)]
    for i in range(4):
        keys = [[oracle_keypair(oracle_mod, d, (rows - 1) // (1 + i + j + 3 * w), seed=61, i=100 * i + 10 * w + j)[0]
                 for j in range(3)] for w in range(2)]
        for ws, ks in zip(wss, keys):
            ws.set_keys([db] * 3, ks)
        for _ in range(3):
            for ws in wss:
                ws.launch(graph=bool(i % 2))
        for ws, ks in zip(wss, keys):
            assert ws.read() == oracle_mod.scan_fused(ks, host, row_bytes)
    for ws in wss:
        ws.close()
    db.close()
