"""Wide aligned tiles where the walk branches: rows and row groups that end
inside, at and after a chunk of 32 entries, long rows of one to many chunks
(the copies run two chunks ahead), more long rows than the first ones dealt to
the blocks, one and several column panels, the last one partly filled, one to
40 tiles along k.  The order of the multiply-adds is the oracle's, so the
comparison is bit for bit."""
import pytest

from test_gpu_spmm import heavy_rows_matrix
from test_gpu_spmm_narrow import check

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.fixture(scope="module")
def matrix():
    return heavy_rows_matrix(n=2048, light=9, heavy=(2000, 545, 544, 513, 512, 511, 129, 128, 97, 96, 95, 65, 64, 63, 33, 32, 31))


@pytest.fixture(scope="module")
def many_long():
    return heavy_rows_matrix(n=1024, light=3, heavy=(70,) * 600)


@pytest.mark.parametrize("dtype,n", [("f32", 68), ("f32", 128), ("f32", 132), ("f32", 260), ("bf16", 136), ("bf16", 256), ("bf16", 264)])
@pytest.mark.parametrize("rows,long_row,tk", [(1, 64, 2048), (2, 64, 700), (4, 96, 300), (4, 512, 64), (1, 0, 52)])
def test_chunk_edges(monkeypatch, matrix, dtype, n, rows, long_row, tk):
    from bcl_b200.containers import context
    monkeypatch.setenv("BCLX_SPMM_LONG_MIN_ROWS", "0")
    with context(0).tuned(spmm_rows=rows, spmm_long_row=long_row):
        check(matrix, n, (700, tk, n), dtype, seed=n + rows)


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("blocks", [1, 148])
def test_more_long_rows_than_dealt(monkeypatch, many_long, dtype, blocks):
    from bcl_b200.containers import context
    monkeypatch.setenv("BCLX_SPMM_LONG_MIN_ROWS", "0")
    with context(0).tuned(spmm_long_row=64, spmm_long_blocks=blocks):
        check(many_long, 264, (500, 300, 264), dtype)
