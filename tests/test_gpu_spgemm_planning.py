"""The planning passes where they branch: rows of more entries than a warp's
share of the classification (512, taken by the block; more of them than a
block can put off), more than 32 tile columns, rows past the last tile's edge,
B rows around the table's search bound, heavy rows of one and of many items
cut by the warp, products without heavy rows.  Compared with the oracle bit
for bit, and the product count with the closed form."""
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


def random_csr(lens, n, rng, value_type="f32"):
    rp = np.zeros(len(lens) + 1, np.int64)
    np.cumsum(lens, out=rp[1:])
    ci = np.concatenate([np.sort(rng.choice(n, int(k), replace=False)) for k in lens]).astype(np.int32)
    v = rng.uniform(-1, 1, ci.size).astype(np.float32) if value_type == "f32" else rng.integers(-99, 99, ci.size).astype(np.int32)
    return gen.CSR(len(lens), n, rp.astype(np.int32), ci, v)


CASES = {
    # A row lengths, B row lengths, B columns, tiles (tm, tk, tn)
    "long_rows": ([511, 512, 513, 1200, 0, 3] + [5] * 60, [4] * 1300, 900, (17, 1300, 900)),
    "many_long_rows": ([600] * 700, [2] * 700, 400, (350, 350, 400)),
    "many_tile_columns": ([40, 0, 700, 9] + [12] * 30, [30] * 800, 2000, (10, 200, 45)),
    "ragged_last_rows": ([20] * 33, [15] * 64, 500, (32, 50, 130)),
    "table_search": ([200] * 8, [0, 1, 63, 64, 65, 128, 129, 2000] * 40, 8192, (8, 320, 8192)),
    "widest_table": ([60] * 6, [0, 5, 127, 128, 129, 4000] * 20, 16384, (6, 120, 16384)),
    "one_block_rows": ([30] * 40, [20] * 50, 250, (40, 50, 250)),
    "no_heavy_rows": ([3] * 100, [4] * 100, 300, (30, 30, 100)),
}


@pytest.mark.parametrize("value_type", ["f32", "i32"])
@pytest.mark.parametrize("name", list(CASES))
def test_against_oracle(name, value_type):
    from bcl_b200.containers import BlockCustom, SPMatrix, spgemm
    a_lens, b_lens, n, tiles = CASES[name]
    rng = np.random.default_rng(len(name))
    a, b = random_csr(a_lens, len(b_lens), rng, value_type), random_csr(b_lens, n, rng, value_type)
    A, B = SPMatrix.from_csr(a, BlockCustom(tiles[:2])), SPMatrix.from_csr(b, BlockCustom(tiles[1:]))
    C, plan = spgemm(A, B, keep_plan=True)
    st = plan.stats()
    plan.close()
    assert st["products"] == gen.intermediate_products(a, b)
    if name == "no_heavy_rows":
        assert st["heavy_rows"] == 0
    if name in ("table_search", "widest_table"):
        assert st["heavy_items"] > st["heavy_rows"] > 0
    rp, ci, cv = O.gemm_tiled(a, b, *tiles, mode=value_type)
    assert_csr_identical(C.get(), rp, ci, cv)


def band(n, width):
    rows = [np.arange(max(0, i - width), min(n, i + width + 1)) for i in range(n)]
    return [r.size for r in rows], np.concatenate(rows).astype(np.int32)


@pytest.mark.parametrize("value_type", ["f32", "i32"])
@pytest.mark.parametrize("name", ["band", "band_one_row_tiles", "full_few_rows", "full_many_rows", "few_tiles", "empty"])
def test_fine_grids(name, value_type):
    """Grids of 17 stages and more, which have a stage map: few of the C tiles
    with stages and all of them, with few rows and many, tile heights off 32
    and of 1, A-row segments of 16, 17 and more entries in a tile, fewer C
    tiles than SMs, no stages at all."""
    from bcl_b200.containers import BlockCustom, SPMatrix, spgemm
    rng = np.random.default_rng(len(name))
    if name.startswith("band"):
        n, width, tile = (2000, 12, 33) if name == "band" else (150, 20, 1)
        mats = []
        for _ in range(2):
            lens, ci = band(n, width)
            m = random_csr(lens, n, rng, value_type)
            m.col_ind[:] = ci
            mats.append(m)
        a, b, tiles = mats[0], mats[1], (tile, tile, tile)
    elif name == "full_few_rows":
        a = random_csr([5, 0, 380, 40] * 100, 400, rng, value_type)
        b, tiles = random_csr([30] * 400, 400, rng, value_type), (20, 20, 20)
    elif name == "full_many_rows":
        a = random_csr([8] * 39990, 136, rng, value_type)
        b, tiles = random_csr([6] * 136, 100, rng, value_type), (2353, 8, 10)
    elif name == "few_tiles":
        a = random_csr([100, 900, 3] * 20, 1000, rng, value_type)
        b, tiles = random_csr([20] * 1000, 300, rng, value_type), (60, 25, 300)
    else:
        a = random_csr([0] * 100, 100, rng, value_type)
        b, tiles = random_csr([3] * 100, 100, rng, value_type), (5, 5, 5)
    A, B = SPMatrix.from_csr(a, BlockCustom(tiles[:2])), SPMatrix.from_csr(b, BlockCustom(tiles[1:]))
    C, plan = spgemm(A, B, keep_plan=True)
    st = plan.stats()
    plan.close()
    assert st["products"] == gen.intermediate_products(a, b)
    rp, ci, cv = O.gemm_tiled(a, b, *tiles, mode=value_type)
    assert_csr_identical(C.get(), rp, ci, cv)


@pytest.mark.parametrize("n,grid", [(40003, 17), (3000, 20)])
def test_empty_tiles_of_a_without_arrays(n, grid):
    """Grids with a stage map do not read A's tiles that have no entries: their
    descriptors may hold no arrays (rows classified at once, and by tiles)."""
    import torch
    from bcl_b200.containers import BlockCustom, SPMatrix, spgemm
    t = -(-n // grid)
    a = gen.erdos_renyi(n, 12, seed=5)
    rows = np.repeat(np.arange(n), np.diff(a.row_ptr))
    keep = (rows // t * 3 + a.col_ind // t) % 4 != 0  # every fourth tile empty
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows[keep], minlength=n))]).astype(np.int32)
    a = gen.CSR(n, n, rp, a.col_ind[keep], a.vals[keep])
    A, B = SPMatrix.from_csr(a, BlockCustom((t, t))), SPMatrix.from_csr(gen.erdos_renyi(n, 9, seed=6), BlockCustom((t, t)))
    want = spgemm(A, B)
    empty = A.desc[:, 2] == 0
    assert int(empty.sum()) > grid
    A.desc[empty, 3:6] = 0
    got = spgemm(A, B)
    for f in ("tile_row_ptr", "tile_offset", "col_ind", "vals"):
        assert torch.equal(getattr(got, f), getattr(want, f)), f
