"""The numeric pass's product walk at the lengths where it can go wrong:
B segments around one batch (32 products), chunks on either side of the packed bound,
empty segments between them, columns shared by neighbouring segments, tiles
whose width is no whole number of 256-column blocks, and heavy rows that are
one item (walked by the B rows' own bounds) or several.  Exact arithmetic
order, so the comparison is bit for bit (see test_gpu_spgemm)."""
import numpy as np
import pytest

from bcl_b200 import gen
from oracle import oracle as O

from gpu_util import assert_csr_identical

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 2, 31, 32, 33, 0, 63, 64, 65, 95, 96, 97, 5, 128, 0]


@pytest.fixture(scope="module", autouse=True)
def cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _csr(m, n, rows, vals):
    rp = np.zeros(m + 1, np.int64)
    np.cumsum([len(r) for r in rows], out=rp[1:])
    ci = np.concatenate([np.asarray(r, np.int32) for r in rows]) if rp[-1] else np.zeros(0, np.int32)
    return gen.CSR(m, n, rp.astype(np.int32), ci, vals(int(rp[-1])))


def _operands(n, span, value_type, seed):
    """B: rows of the lengths above, their columns consecutive or spread, all
    within `span` columns; A: rows of 0 to 70 of B's rows."""
    rng = np.random.default_rng(seed)
    k = 96

    def vals(count):
        if value_type == "i32":
            return rng.integers(-2**31, 2**31, count).astype(np.int32)
        v = rng.uniform(-1, 1, count).astype(np.float32)
        v[rng.random(count) < 0.02] = -0.0
        return v

    b_rows = []
    for i in range(k):
        ln = min(LENGTHS[i % len(LENGTHS)], span)
        lo = int(rng.integers(0, n - span + 1)) if span < n else 0
        if i % 2:
            start = lo + int(rng.integers(0, span - ln + 1))
            b_rows.append(np.arange(start, start + ln))
        else:
            b_rows.append(lo + np.sort(rng.choice(span, ln, replace=False)))
    a_rows = [np.sort(rng.choice(k, int(c), replace=False)) for c in rng.integers(0, 71, 64)]
    return _csr(64, k, a_rows, vals), _csr(k, n, b_rows, vals)


@pytest.mark.parametrize("mode", ["fused", "per_stage"])
@pytest.mark.parametrize("value_type", ["f32", "i32"])
@pytest.mark.parametrize("n,span,tiles", [
    (300, 300, (64, 96, 300)),        # dense outputs, one stage, one item a row
    (1000, 1000, (33, 40, 1000)),     # several items a row, three stages, ragged
    (9001, 9001, (64, 48, 9001)),     # tile above 8192 columns: every row heavy, last block of 41 columns
    (16384, 16384, (17, 96, 16384)),  # the widest tile
    (16383, 200, (64, 32, 5000)),     # narrow spans in wide tiles: one-item rows
])
def test_walk_vs_oracle(n, span, tiles, value_type, mode):
    from bcl_b200.containers import BlockCustom, SPMatrix, spgemm
    a, b = _operands(n, span, value_type, n + span)
    A = SPMatrix.from_csr(a, BlockCustom(tiles[:2]))
    B = SPMatrix.from_csr(b, BlockCustom(tiles[1:]))
    rp, ci, cv = O.gemm_tiled(a, b, *tiles, mode=value_type)
    assert_csr_identical(spgemm(A, B, stages=mode).get(), rp, ci, cv)


@pytest.mark.parametrize("long_seg", [1, 8, 14, 33, 1 << 20])
def test_packed_bound_does_not_change_results(long_seg):
    from bcl_b200.containers import BlockCustom, SPMatrix, spgemm
    a, b = _operands(1000, 700, "f32", 5)
    A, B = SPMatrix.from_csr(a, BlockCustom((64, 40))), SPMatrix.from_csr(b, BlockCustom((40, 1000)))
    rp, ci, cv = O.gemm_tiled(a, b, 64, 40, 1000)
    assert_csr_identical(spgemm(A, B, tuning=(1, 4, long_seg)).get(), rp, ci, cv)


@pytest.mark.parametrize("value_type", ["f32", "i32"])
@pytest.mark.parametrize("n,tile", [(3001, 3001), (2900, 700)])
def test_few_very_heavy_rows_cut_finer(n, tile, value_type):
    """Two rows of 32768 products or more (items of half as many outputs), one
    just below, among light ones."""
    from bcl_b200.containers import BlockCustom, SPMatrix, spgemm
    rng = np.random.default_rng(n)
    k, per = 900, 64 * (n // tile + 1)

    def vals(count):
        return (rng.uniform(-1, 1, count).astype(np.float32) if value_type == "f32"
                else rng.integers(-99, 99, count).astype(np.int32))

    b = _csr(k, n, [np.sort(rng.choice(n, per, replace=False)) for _ in range(k)], vals)
    lens = [3] * 20 + [900, 600, 500] + [7] * 20
    a = _csr(len(lens), k, [np.sort(rng.choice(k, c, replace=False)) for c in lens], vals)
    A, B = SPMatrix.from_csr(a, BlockCustom((16, 300))), SPMatrix.from_csr(b, BlockCustom((300, tile)))
    rp, ci, cv = O.gemm_tiled(a, b, 16, 300, tile, mode=value_type)
    assert_csr_identical(spgemm(A, B).get(), rp, ci, cv)


@pytest.mark.parametrize("value_type", ["f32", "i32"])
@pytest.mark.parametrize("n_mid,n_most,grid_k", [(3, 0, 4), (0, 2, 4), (60, 2, 5), (60, 2, 40), (200, 1, 3), (2, 1, 1)])
def test_items_split_by_stage(n_mid, n_most, grid_k, value_type):
    """Rows above 8192 products and above 32768, few or many of each, on one to
    40 tiles along k (with and without a stage map): their items' stages run
    apart and are added in order.  The numeric pass twice on one plan, the
    second time with other values; signed zeros among them."""
    from bcl_b200.containers import BlockCustom, SPMatrix, spgemm_numeric, spgemm_symbolic
    import torch
    rng = np.random.default_rng(n_mid * 10 + grid_k)
    k, n, per = 800, 1500, 60

    def vals(count):
        if value_type == "i32":
            return rng.integers(-2**31, 2**31, count).astype(np.int32)
        v = rng.uniform(-1, 1, count).astype(np.float32)
        v[rng.random(count) < 0.05] = -0.0
        return v

    lens = [2] * 30 + [200] * n_mid + [5] * 10 + [700] * n_most + [40] * 5
    a = _csr(len(lens), k, [np.sort(rng.choice(k, c, replace=False)) for c in lens], vals)
    b = _csr(k, n, [np.sort(rng.choice(n, per, replace=False)) for _ in range(k)], vals)
    tk = -(-k // grid_k)
    A, B = SPMatrix.from_csr(a, BlockCustom((len(lens), tk))), SPMatrix.from_csr(b, BlockCustom((tk, n)))
    plan, out, trp, toff, nnz = spgemm_symbolic(A, B)
    ci = torch.empty(nnz, dtype=torch.int32, device="cuda")
    v = torch.empty(nnz, dtype=A.vals.dtype, device="cuda")
    out.col_ind, out.vals = ci.data_ptr(), v.data_ptr()
    for _ in range(2):
        spgemm_numeric(plan, A, B, out)
        C = SPMatrix(a.m, n, len(lens), n, a.vals.dtype, 0, trp, toff, ci, v)
        rp, cols, cv = O.gemm_tiled(a, b, len(lens), tk, n, mode=value_type)
        assert_csr_identical(C.get_host_gather() if value_type == "i32" else C.get(), rp, cols, cv)
        a.vals[:] = vals(a.nnz)
        A = SPMatrix.from_csr(a, BlockCustom((len(lens), tk)))
    plan.close()
