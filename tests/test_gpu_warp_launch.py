"""GPU parity of the own-rows scan at its launch edges: leaf pairs walked two
at a time (one pair only at depth 1), CTAs from one warp to the full width as
the items go from fewer than the SMs to several rounds per warp.  Shares are
exact: the oracle's bytes."""
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
