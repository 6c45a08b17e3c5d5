"""B rows that name a column twice or more: every entry is a product of its
own, in stored order.  Segments of fewer products than a warp has lanes, and
of more, through every form of the product; repeats in some tiles of the grid
only, at the first and last rows of a tile and of a block's 2,048 rows."""
import numpy as np
import pytest

from bcl_b200 import gen
from oracle import oracle as O

from gpu_util import assert_csr_identical

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def matrix(m, n, deg, dtype, seed, repeat_rows=()):
    """`deg` ascending entries a row; in `repeat_rows` every other one repeats the column before."""
    rng = np.random.default_rng(seed)
    cols = np.sort(np.argsort(rng.random((m, n)), axis=1)[:, :deg], axis=1)
    for r in repeat_rows:
        cols[r, 1::2] = cols[r, :deg - deg % 2:2]
    v = rng.uniform(-1, 1, m * deg).astype(np.float32) if dtype == "f32" else rng.integers(-9, 10, m * deg, np.int32)
    return gen.CSR(m, n, (np.arange(m + 1) * deg).astype(np.int32), cols.reshape(-1).astype(np.int32), v)


def tiled(a, tm, tn):
    import torch
    from bcl_b200.containers import SPMatrix, split_tiles
    parts = [torch.from_numpy(x).cuda() for x in split_tiles(a, tm, tn)]
    return SPMatrix(a.m, a.n, tm, tn, a.vals.dtype, 0, *parts)


@pytest.mark.parametrize("dtype", ["f32", "i32"])
@pytest.mark.parametrize("deg", [2, 13, 14, 20, 31, 32, 33, 70])
def test_whole_tile(deg, dtype):
    from bcl_b200.containers import spgemm
    a, b = matrix(96, 300, 24, dtype, 1), matrix(300, 500, deg, dtype, deg, range(300))
    A, B = tiled(a, 96, 300), tiled(b, 300, 500)
    want = O.gemm_tiled(a, b, 96, 300, 500, mode=dtype)
    assert_csr_identical(spgemm(A, B).get(), *want)


@pytest.mark.parametrize("rows", [(0,), (1023,), (1024,), (2047,), (2048,), (2099,), (50, 51, 1500)])
@pytest.mark.parametrize("tiles", [(96, 2100, 500), (64, 1050, 500), (96, 100, 500)])
def test_a_few_rows_of_a_grid(tiles, rows):
    """1, 2 and 21 tiles along k (the last with a stage map); the repeats in single rows."""
    from bcl_b200.containers import spgemm
    a, b = matrix(96, 2100, 300, "f32", 2), matrix(2100, 500, 22, "f32", 3, rows)
    A, B = tiled(a, *tiles[:2]), tiled(b, *tiles[1:])
    want = O.gemm_tiled(a, b, *tiles)
    for stages in ("fused", "per_stage", "batched_graph"):
        assert_csr_identical(spgemm(A, B, stages).get(), *want)


@pytest.mark.parametrize("predictor", ["default", None])
def test_learned(predictor):
    from bcl_b200.containers import spgemm_learned
    a, b = matrix(200, 700, 60, "f32", 4), matrix(700, 900, 25, "f32", 5, range(0, 700, 3))
    want = O.gemm_tiled(a, b, 100, 350, 900)
    assert_csr_identical(spgemm_learned(tiled(a, 100, 350), tiled(b, 350, 900), predictor=predictor).get(), *want)


def test_without_allocation():
    from test_zz_no_alloc import noalloc_product
    a, b = matrix(80, 300, 30, "f32", 6), matrix(300, 400, 25, "f32", 7, range(300))
    want = O.spgemm_local(a, b)
    rc, k, rp, ci, v = noalloc_product(a, b, capacity=int(want[0][-1]))
    assert rc == 0
    assert_csr_identical(gen.CSR(80, 400, rp, ci, v), *want)


@pytest.mark.parametrize("nparts", [3, 20])
def test_accumulated_parts(nparts):
    """Whole values, as a part's repeats are added up before the parts are."""
    from bcl_b200.containers import tile_accumulate
    parts = [matrix(120, 300, 24, "i32", 10 + p, range(p, 120, 4)) for p in range(nparts)]
    parts = [gen.CSR(p.m, p.n, p.row_ptr, p.col_ind, p.vals.astype(np.float32)) for p in parts]
    assert_csr_identical(tile_accumulate([tiled(p, 120, 300) for p in parts]).get(), *O.accumulate(parts))


@pytest.mark.parametrize("row", [0, 63, 64, 127, 128, 900, 4999])
def test_one_repeat_among_many_short_blocks(row):
    """The rows are dealt to the blocks 64 and more at a time: one row with repeats, at
    the first and last of such a part, in the last tile along k."""
    from bcl_b200.containers import spgemm
    a, b = matrix(64, 10000, 40, "f32", 8), matrix(10000, 300, 20, "f32", 9, (5000 + row,))
    a.col_ind.reshape(64, 40)[:, -1] = 9999  # (ascending still)
    a.col_ind.reshape(64, 40)[:, -2] = 5000 + row if row < 4999 else 9998
    a.col_ind.reshape(64, 40)[:, :-2] = np.arange(38)
    want = O.gemm_tiled(a, b, 64, 5000, 300)
    assert_csr_identical(spgemm(tiled(a, 64, 5000), tiled(b, 5000, 300)).get(), *want)
