"""Tiles of the operator where small blocks share an SM: the reported blocks per SM fit its shared memory (228 KB, 1 KB of
it per block beside the block's own 24 values of exchange per thread of the largest block and 1 KB of reduction), and the
operator is right at the tiles that follow (tolerance as in test_row_operator.py)."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover - collected on CPU boxes, skipped
    pytest.skip("CUDA device required", allow_module_level=True)

from test_row_operator import test_row_operator as check_operator  # noqa: E402


@pytest.mark.parametrize("loads", [1, 3, 6])
@pytest.mark.parametrize("precision,block", [("fp64", 24 * 256 * 8 + 2048), ("mixed", 24 * 384 * 4 + 2048)])
def test_reported_blocks_fit(pkg, precision, block, loads):
    for n in (4, 8, 16, 24, 30, 32, 36, 48, 54, 64, 96):
        op = pkg.Operator(n, loads, *pkg.PAPER_MEDIUM, precision=precision)
        config = (ctypes.c_int * 9)()
        assert pkg._lib.lib().pgj_tile_config(op._ctx, config) == 0
        assert 1 <= config[3] <= 228 * 1024 // block, (n, config[3])


@pytest.mark.parametrize("n,loads", [(20, 6), (24, 6), (30, 6), (32, 3), (32, 6)])
def test_operator_at_shared_tiles(pkg, oracle, n, loads):
    check_operator(pkg, oracle, n, loads)
