"""Performance cases: what one PIR server has this framework do, through its public entry points.

A server holds resident tables and answers DPF key shares over them.  Every
case is one such answer (or one burst of answers): host keys in, host shares
out, over a table that is already on the device.  The ranges:

* tables of 2^11 to 2^30 rows, of any size and not only powers of two, some of
  them a row range of a larger table (keys deeper than the table);
* rows of 16 B to 4 KB: 32-B storage slots, 64-B accounts, 256-B records, the
  4-KB pages of the reference, and sizes between that are not powers of two;
* one query (3 cuckoo keys) up to batches of 16 queries in a pass, direct or
  replayed from a CUDA graph, one table or several;
* tables with a pending epoch delta; the continuous-batching server; point
  evaluation.

Each state has a scanner, tables and keys of its own, made from the seed.
Shares are bytes and have to be equal, bit for bit.
"""
import numpy as np

from morphogen_b200.gpu_dpf import ChaChaParams, GpuPageMatrix, GpuScanner, generate_chacha_dpf_keys
from morphogen_b200.server import PirServer

# Integer operations of one tree-node expansion: two ChaCha8 blocks of 4
# double rounds, 8 quarter rounds each, 12 operations per quarter round.
OPS_PER_NODE = 2 * 4 * 8 * 12
EXACT_MAX_NODES = 1 << 22  # exact() in numpy stays under about ten seconds


def _case(kind, rows, row_bytes, bits, queries=1, graph=False, first_row=0, delta=0, rows2=0, row_bytes2=0,
          bits2=0, queries2=0, points=0, name=None):
    c = dict(kind=kind, rows=rows, row_bytes=row_bytes, bits=bits, queries=queries, graph=graph,
             first_row=first_row, delta=delta, rows2=rows2, row_bytes2=row_bytes2, bits2=bits2,
             queries2=queries2, points=points)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # The smallest table a server would bother to offload: a call's latency is launches and copies.
        _case("query", 4099, 32, 13, name="query 4099 x 32 B"),
        # The 256-B record configuration: one query over 256 MiB.
        _case("query", 1 << 20, 256, 20, name="query 2^20 x 256 B"),
        # Records that are no power of two, neither in number nor in size.
        _case("query", 1_000_003, 48, 20, name="query 1000003 x 48 B"),
        # One shard of a 2^31-row storage table: 31-bit keys over a range of 2^25 rows.
        _case("query", 1 << 25, 32, 31, first_row=5 << 25, name="shard 2^25 of 2^31 x 32 B"),
        # One query over the storage table at the size of which three still fit the card.
        _case("query", 1 << 30, 32, 30, name="query 2^30 x 32 B"),
        # The reference's page mode through its own entry point: 4-KB pages, 25-bit keys.
        _case("scan", 1_300_021, 4096, 25, name="scan 1300021 x 4 KB pages"),
        # A full batch of 16 queries over accounts, replayed from a graph.
        _case("batch", 3_000_000, 64, 22, queries=16, graph=True, name="batch 16 x 3000000 x 64 B"),
        # The mainnet mix of account and storage lookups, 4 : 3, over two tables in one pass.
        _case("mixed", 1 << 21, 64, 21, queries=4, rows2=1 << 24, row_bytes2=32, bits2=24, queries2=3,
              name="mixed 2^21 x 64 B + 2^24 x 32 B"),
        # A query between two epoch merges: 2^16 updated rows are folded into the answer.
        _case("query", 1 << 22, 32, 22, delta=1 << 16, name="query 2^22 x 32 B, 2^16 delta"),
        # A burst of single lookups at the serving loop, batched by the server.
        _case("serve", 1 << 20, 64, 20, queries=24, name="serve 24 lookups 2^20 x 64 B"),
        # Point evaluation of one key, as a consistency check of a share does.
        _case("points", 0, 16, 31, points=100_003, name="eval 100003 points, 31 bits"),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _bits_for(rows):
    return max(1, (rows - 1).bit_length())


def draw(rng):
    """One more case: sizes log-uniform over each kind's range, odd ones among them."""
    kind = rng.choice(["query", "query", "query", "shard", "scan", "batch", "mixed", "delta", "serve", "points"])
    if kind == "points":
        return _case("points", 0, 16, rng.randint(12, 32), points=_log_uniform(rng, 1000, 400_000))
    rb = rng.choice([16, 32, 32, 48, 64, 64, 96, 128, 256, 256, 512, 1024])
    if kind == "scan":
        rows = _log_uniform(rng, 3000, 1_500_000)
        return _case("scan", rows, 4096, rng.choice([_bits_for(rows), 25]))
    if kind == "shard":
        bits = rng.randint(26, 32)
        rows = _log_uniform(rng, 1 << 16, 1 << 25)
        return _case("query", rows, min(rb, 128), bits, first_row=rng.randrange((1 << bits) - rows))
    if kind == "batch":
        rows = _log_uniform(rng, 1 << 14, 1 << 22)
        return _case("batch", rows, rb, _bits_for(rows), queries=rng.randint(2, 16), graph=rng.random() < 0.5)
    if kind == "mixed":
        rows, rows2 = _log_uniform(rng, 1 << 14, 1 << 22), _log_uniform(rng, 1 << 16, 1 << 24)
        return _case("mixed", rows, 64, _bits_for(rows), queries=rng.randint(1, 5), rows2=rows2, row_bytes2=32,
                     bits2=_bits_for(rows2), queries2=rng.randint(1, 4))
    if kind == "delta":
        rows = _log_uniform(rng, 1 << 14, 1 << 24)
        return _case("query", rows, min(rb, 256), _bits_for(rows), delta=_log_uniform(rng, 256, 1 << 16))
    if kind == "serve":
        rows = _log_uniform(rng, 1 << 14, 1 << 21)
        return _case("serve", rows, min(rb, 256), _bits_for(rows), queries=rng.randint(4, 32))
    rows = _log_uniform(rng, 1 << 11, (1 << 28) if rb <= 32 else (8 << 30) // (2 * rb))
    return _case("query", rows, rb, _bits_for(rows))


def _keys(rng, bits, first_row, rows, n):
    """n keys of one party for uniform targets among the rows held, as bytes off the wire."""
    params = ChaChaParams(bits)
    out = []
    for t in rng.integers(first_row, first_row + rows, n):
        pair = generate_chacha_dpf_keys(params, int(t), rng)
        out.append(pair[int(rng.integers(0, 2))].to_bytes())
    return out


def _delta(rng, case):
    idx = rng.integers(0, case["rows"], case["delta"]).astype(np.uint64)
    diffs = rng.integers(0, 256, case["delta"] * case["row_bytes"], dtype=np.uint8)
    return idx, diffs


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    scanner = GpuScanner(0)
    st = {"case": case, "scanner": scanner}
    if case["kind"] == "points":
        st["key"] = _keys(rng, case["bits"], 0, 1 << case["bits"], 1)[0]
        st["idx"] = rng.integers(0, 1 << case["bits"], case["points"]).astype(np.uint64)
        return st
    st["table"] = table = GpuPageMatrix.from_seed(scanner, case["rows"], case["row_bytes"], seed,
                                                  first_row=case["first_row"])
    per_query = 1 if case["kind"] == "serve" else 3  # the server takes single lookups here
    st["keys"] = _keys(rng, case["bits"], case["first_row"], case["rows"], per_query * case["queries"])
    if case["kind"] == "mixed":
        table2 = GpuPageMatrix.from_seed(scanner, case["rows2"], case["row_bytes2"], seed + 1)
        keys2 = _keys(rng, case["bits2"], 0, case["rows2"], 3 * case["queries2"])
        st["items"] = [(table, k) for k in st["keys"]] + [(table2, k) for k in keys2]
    if case["kind"] in ("scan", "batch"):
        k = st["keys"]
        st["queries"] = [k[i:i + 3] for i in range(0, len(k), 3)]
    if case["delta"]:
        table.delta_reserve(case["delta"])
        table.delta_push(*_delta(rng, case))
    if case["kind"] == "serve":
        st["server"] = PirServer(scanner)
    return st


def _bytes(shares):
    return np.frombuffer(b"".join(shares), np.uint8)


def run(st):
    case = st["case"]
    kind, scanner = case["kind"], st["scanner"]
    if kind == "query":
        return _bytes(scanner.scan_keys(st["table"], st["keys"])[0])
    if kind == "scan":
        return _bytes(scanner.scan(st["table"], st["queries"][0]).pages)
    if kind == "batch":
        res = scanner.scan_batch(st["table"], st["queries"], use_cuda_graph=case["graph"])
        return _bytes([page for r in res for page in r.pages])
    if kind == "mixed":
        return _bytes(scanner.scan_multi(st["items"], use_cuda_graph=case["graph"]))
    if kind == "serve":
        srv, table = st["server"], st["table"]
        rids = [srv.submit([(table, k)]) for k in st["keys"]]
        return _bytes([srv.wait(r)[0][0] for r in rids])
    return scanner.eval_points(st["key"], st["idx"])


def _nodes(rows, bits, first_row=0):
    """Tree nodes whose leaves meet rows [first_row, first_row + rows)."""
    last = first_row + rows - 1
    return sum((last >> s) - (first_row >> s) + 1 for s in range(1, bits + 1))


def work(case):
    if case["kind"] == "points":
        return {"bytes": case["points"] * 24, "flops": case["points"] * case["bits"] * OPS_PER_NODE}
    nk = (1 if case["kind"] == "serve" else 3) * case["queries"]
    nbytes = case["rows"] * case["row_bytes"] + nk * (case["row_bytes"] + 35 + 18 * case["bits"])
    nodes = nk * (_nodes(case["rows"], case["bits"], case["first_row"]) + case["delta"] * case["bits"])
    nbytes += case["delta"] * (case["row_bytes"] + 8)
    if case["rows2"]:
        nk2 = 3 * case["queries2"]
        nbytes += case["rows2"] * case["row_bytes2"] + nk2 * (case["row_bytes2"] + 35 + 18 * case["bits2"])
        nodes += nk2 * _nodes(case["rows2"], case["bits2"])
    return {"bytes": nbytes, "flops": nodes * OPS_PER_NODE}


# ---- the same answers in plain numpy ------------------------------------------

def _rotl(x, n):
    return (x << np.uint32(n)) | (x >> np.uint32(32 - n))


def _block(seeds, counter):
    """ChaCha8 blocks of (n, 4) seeds: key = seed || seed, nonce 0."""
    sigma = (0x61707865, 0x3320646E, 0x79622D32, 0x6B206574)
    zero = np.zeros(len(seeds), np.uint32)
    s = [zero + np.uint32(v) for v in sigma] + [seeds[:, i % 4] for i in range(8)]
    s += [zero + np.uint32(counter), zero, zero, zero]
    x = list(s)
    for _ in range(4):
        for a, b, c, d in ((0, 4, 8, 12), (1, 5, 9, 13), (2, 6, 10, 14), (3, 7, 11, 15),
                           (0, 5, 10, 15), (1, 6, 11, 12), (2, 7, 8, 13), (3, 4, 9, 14)):
            for r, q in ((16, 12), (8, 7)):
                x[a] = x[a] + x[b]
                x[d] = _rotl(x[d] ^ x[a], r)
                x[c] = x[c] + x[d]
                x[b] = _rotl(x[b] ^ x[c], q)
    return [u + v for u, v in zip(x, s)]


def _eval(key, index):
    """DPF outputs (n, 16) of one key at sorted distinct indices, level by level."""
    d = key[18]
    seeds = np.frombuffer(key, np.uint32, 4).copy()[None]
    t = np.array([key[16]], np.uint8)
    nodes = np.zeros(1, np.uint64)
    for level in range(d):
        cw = np.frombuffer(key, np.uint32, 4, 19 + 18 * level)
        b0, b1 = _block(seeds, 0), _block(seeds, 1)
        on = t == 1
        child = []
        for side in (0, 1):
            s = np.stack(b0[4 * side:4 * side + 4], axis=1) ^ np.where(on[:, None], cw, 0).astype(np.uint32)
            bit = (b1[side] & 1).astype(np.uint8) ^ np.where(on, key[19 + 18 * level + 16 + side], 0).astype(np.uint8)
            child.append((s, bit))
        want = np.unique(index >> np.uint64(d - 1 - level))
        at = np.searchsorted(nodes, want >> np.uint64(1))
        right = (want & np.uint64(1)).astype(bool)
        seeds = np.where(right[:, None], child[1][0][at], child[0][0][at])
        t = np.where(right, child[1][1][at], child[0][1][at])
        nodes = want
    final = np.frombuffer(key[-16:], np.uint32)
    return (seeds ^ np.where((t == 1)[:, None], final, 0).astype(np.uint32)).view(np.uint8)


def _table(case, seed):
    """Rows of the synthetic table: SplitMix64 outputs of the logical table's words."""
    per = case["row_bytes"] // 8
    w = np.arange(case["first_row"] * per, (case["first_row"] + case["rows"]) * per, dtype=np.uint64)
    z = np.uint64(seed) + (w + np.uint64(1)) * np.uint64(0x9E3779B97F4A7C15)
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return (z ^ (z >> np.uint64(31))).view(np.uint8).reshape(case["rows"], case["row_bytes"])


def exact(case, seed):
    """The shares of the smaller cases in plain numpy; None for the others."""
    if work(case)["flops"] > EXACT_MAX_NODES * OPS_PER_NODE or case["rows2"]:
        return None
    rng = np.random.default_rng(seed)
    if case["kind"] == "points":
        key = _keys(rng, case["bits"], 0, 1 << case["bits"], 1)[0]
        index, back = np.unique(rng.integers(0, 1 << case["bits"], case["points"]).astype(np.uint64),
                                return_inverse=True)
        return _eval(key, index)[back]
    nk = (1 if case["kind"] == "serve" else 3) * case["queries"]
    keys = _keys(rng, case["bits"], case["first_row"], case["rows"], nk)
    table = _table(case, seed)
    if case["delta"]:
        idx, diffs = _delta(rng, case)
        np.bitwise_xor.at(table, idx.astype(np.int64), diffs.reshape(-1, case["row_bytes"]))
    index = np.arange(case["first_row"], case["first_row"] + case["rows"], dtype=np.uint64)
    out = []
    for k in keys:
        mask = np.tile(_eval(k, index), case["row_bytes"] // 16)
        out.append(np.bitwise_xor.reduce(table & mask, axis=0))
    return np.concatenate(out)
