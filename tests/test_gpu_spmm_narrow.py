"""Narrow and unaligned dense tiles (k_spmm_narrow, k_spmm_chain): widths around one and two
words per lane and around the bound to the wide kernel, rows on 16, 4 and 2
bytes, tile bases off 16 bytes, one to 40 tiles along k, long rows listed or
not, rows without entries.  The order of the multiply-adds is the oracle's, so
the comparison is bit for bit."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O

from gpu_util import bits
from test_gpu_spmm import heavy_rows_matrix, run

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.fixture(scope="module")
def matrix():
    return heavy_rows_matrix(n=2048, light=5, heavy=(1500, 600, 300, 256, 255, 33, 32, 31))


def check(a, n, tiles, dtype, seed=1):
    rng = np.random.default_rng(seed)
    b = rng.standard_normal((a.n, n)).astype(np.float32)
    c0 = rng.standard_normal((a.m, n)).astype(np.float32)
    empty = np.diff(a.row_ptr) == 0
    assert empty.any()
    if dtype == "f32":
        c0.view(np.uint32)[empty] = np.uint32(0x7FC01234)  # untouched, payload included
        got, want = bits(run(a, b, tiles, c0=c0)), bits(O.spmm_tiled(a, b, c0, *tiles))
        assert np.all(got[empty] == np.uint32(0x7FC01234))
    else:
        b, c0 = O.to_bf16(b), O.to_bf16(c0)
        c0[empty] = np.uint16(0x7FC5)
        got, want = run(a, b, tiles, dtype="bf16", c0=c0), O.spmm_tiled_bf16(a, b, c0, *tiles)
        assert np.all(got[empty] == np.uint16(0x7FC5))
    assert np.array_equal(got[~empty], want[~empty])


@pytest.mark.parametrize("listed", ["0", "65536"])
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 7, 8, 16, 31, 32, 33, 34, 47, 63, 64, 65, 66, 68, 127, 128, 129, 130, 136, 201])
def test_widths(monkeypatch, matrix, n, dtype, listed):
    monkeypatch.setenv("BCLX_SPMM_LONG_MIN_ROWS", listed)
    check(matrix, n, (700, 800, n), dtype, seed=n)


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("n,tiles", [
    (24, (2048, 2048, 24)),   # one stage: 16 rows an item
    (24, (300, 64, 24)),      # 32 stages: one row an item, one lane a stage
    (47, (300, 52, 47)),      # 40 stages: two groups of stages
    (100, (512, 512, 24)),    # several tile columns, a narrower last one
    (300, (512, 700, 260)),   # wide columns, a narrow last one (aligned)
    (301, (512, 700, 260)),   # wide columns for the wide kernel, the last one unaligned
])
def test_grids(monkeypatch, matrix, n, tiles, dtype):
    monkeypatch.setenv("BCLX_SPMM_LONG_MIN_ROWS", "0")
    check(matrix, n, tiles, dtype, seed=n)


@pytest.mark.parametrize("dtype,shift,ld", [("f32", 0, 12), ("f32", 1, 12), ("f32", 3, 13), ("bf16", 0, 16),
                                            ("bf16", 2, 16), ("bf16", 1, 16), ("bf16", 0, 15)])
def test_tile_bases_and_leading_dimensions(matrix, dtype, shift, ld):
    """One tile whose base is `shift` elements past a 256-byte boundary; what
    lies between the rows stays as it was."""
    import torch
    from bcl_b200 import _lib
    from bcl_b200.containers import context
    a, n = matrix, 10
    tdt = torch.float32 if dtype == "f32" else torch.bfloat16
    g = torch.Generator().manual_seed(shift * 100 + ld)
    B = torch.randn(a.n * ld + 8, generator=g).to(tdt).cuda()
    C = torch.randn(a.m * ld + 8, generator=g).to(tdt).cuda()

    def rows(x, m):
        return x[shift:shift + m * ld].view(m, ld)

    b, c0, before = rows(B, a.n)[:, :n].cpu(), rows(C, a.m)[:, :n].cpu(), C.clone()
    rp, ci, v = (torch.from_numpy(x).cuda() for x in (a.row_ptr, a.col_ind, a.vals))
    es = B.element_size()
    _lib.call("bclx_spmm_tile", context().use_current_stream(), a.m, n, a.n, a.nnz,
              ctypes.c_void_p(C.data_ptr() + shift * es), ctypes.c_void_p(B.data_ptr() + shift * es),
              ctypes.c_void_p(v.data_ptr()), ctypes.c_void_p(rp.data_ptr()), ctypes.c_void_p(ci.data_ptr()), ld, ld,
              _lib.F32 if dtype == "f32" else _lib.BF16)
    got = rows(C, a.m)[:, :n].cpu()
    tiles = (a.m, a.n, n)
    if dtype == "f32":
        assert np.array_equal(bits(got.numpy()), bits(O.spmm_tiled(a, b.numpy().copy(), c0.numpy().copy(), *tiles)))
    else:
        as_u16 = lambda t: t.contiguous().view(torch.int16).numpy().view(np.uint16)  # noqa: E731
        assert np.array_equal(as_u16(got), O.spmm_tiled_bf16(a, as_u16(b), as_u16(c0), *tiles))
    rows(C, a.m)[:, :n] = rows(before, a.m)[:, :n]
    assert torch.equal(C, before)


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("n,tiles", [(119, (700, 800, 119)), (13, (2048, 64, 13)), (56, (300, 2048, 56)), (40, (2048, 2048, 16))])
def test_few_rows(matrix, n, tiles, dtype):
    """Few rows, the knob left at its default: rows of 128 entries and of four
    times their tile row's mean go to the chains (and of two and three tile
    columns, the last one narrower)."""
    check(matrix, n, tiles, dtype, seed=n)


@pytest.mark.parametrize("dtype,n", [("f32", 65), ("f32", 119), ("f32", 150), ("f32", 201), ("bf16", 99), ("bf16", 185), ("bf16", 258), ("bf16", 270)])
@pytest.mark.parametrize("tiles", [(700, 800), (2048, 64)])
def test_wide_unaligned_listed(monkeypatch, matrix, dtype, n, tiles):
    """Rows off 16 bytes of more units than a lane group holds, long rows
    listed: the others go to the wide kernel, several to a warp and one."""
    monkeypatch.setenv("BCLX_SPMM_LONG_MIN_ROWS", "0")
    check(matrix, n, (*tiles, n), dtype, seed=n)


def test_scratch_does_not_grow_with_the_tile_columns():
    """Few rows and many narrow tile columns: the long rows are listed once for all of
    them (and run for each)."""
    import torch
    from bcl_b200 import gen
    from bcl_b200.containers import BlockCustom, DMatrix, SPMatrix, context, gemm
    m, k, n = 60000, 600, 512
    rng = np.random.default_rng(0)
    lens = np.where(np.arange(m) % 9000 == 17, 500, 1)
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    ci = np.concatenate([np.sort(rng.choice(k, x, replace=False)) for x in lens]).astype(np.int32)
    a = gen.CSR(m, k, rp, ci, rng.integers(-4, 5, ci.size).astype(np.float32))
    A = SPMatrix.from_csr(a, BlockCustom((m, k)))
    b = torch.from_numpy(rng.integers(-4, 5, (k, n)).astype(np.float32)).cuda()
    B, C = DMatrix.from_array(b, BlockCustom((k, 1))), DMatrix.zeros((m, n), BlockCustom((m, 1)))
    dense = torch.sparse_csr_tensor(*(torch.from_numpy(x).cuda() for x in (a.row_ptr.astype(np.int64), a.col_ind.astype(np.int64), a.vals)), (m, k))
    context().synchronize()
    context().release_cached()
    before = torch.cuda.mem_get_info()[0]
    gemm(A, B, C)
    torch.cuda.synchronize()
    used = before - torch.cuda.mem_get_info()[0]
    assert used <= 64 << 20, used
    assert torch.equal(C.get_matrix(), (dense @ b))  # whole values: exact in any order
