"""Which loads of the pass's kernels may take the read-only path: a kernel that
is launched while its predecessors run must read what they write with plain
loads, so only the table's rows go through __ldg, and no such kernel has
__restrict__ parameters."""
import re

import pytest

from morphogen_b200 import build as B

SOURCES = [p for p in (*B.SOURCES, *B.HEADERS) if p.suffix in (".cu", ".cuh")]


def code(path):
    return re.sub(r"//[^\n]*", "", path.read_text())


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_read_only_loads_are_table_rows(path):
    args = re.findall(r"__ldg\(\s*([A-Za-z_&][\w>\-]*)", code(path))
    assert set(args) <= {"tbl", "bp", "lp"}


@pytest.mark.parametrize("path", SOURCES, ids=lambda p: p.name)
def test_chained_kernels_promise_nothing_about_their_arguments(path):
    bodies = re.split(r"__global__", code(path))[1:]
    chained = [b for b in bodies if re.search(r"chain_(begin|wait)\(\);", b)]
    assert bool(chained) == (path.name == "mg_kernels.cu")
    for b in chained:
        assert "__restrict__" not in b[:b.index("{")]
        # Inside, only pointers to the table's rows.
        names = re.findall(r"__restrict__\s+(\w+)", b[b.index("{"):b.index("\n}\n")])
        assert set(names) <= {"tbl", "bp"}


def test_a_scan_is_not_launched_beside_its_frontier():
    # Its idle CTAs would keep other passes off the SMs.
    bodies = re.split(r"__global__", code(B.CSRC / "mg_kernels.cu"))[1:]
    (frontier,) = [b for b in bodies if re.match(r"[^{]*\bfrontier_kernel\(", b)]
    frontier = frontier[:frontier.index("\n}\n")]
    assert "chain_wait();" in frontier
    assert "chain_begin" not in frontier and "TriggerProgrammatic" not in frontier
