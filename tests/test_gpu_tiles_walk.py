"""Slicing and gather where their entry chunks (512 entries a warp, 32 at a
time) begin and end: rows of exactly those lengths, runs that cross them, hub
rows over many chunks, empty rows between, one to 100 tile columns; and rows
that must be refused wherever the fault lies."""
import numpy as np
import pytest

from bcl_b200 import gen

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def matrix(lens, n, value_type="f32", seed=0):
    rng = np.random.default_rng(seed)
    rp = np.zeros(len(lens) + 1, np.int64)
    np.cumsum(lens, out=rp[1:])
    cols = [np.sort(rng.choice(n, int(k), replace=False)) for k in lens]
    ci = np.concatenate(cols).astype(np.int32) if rp[-1] else np.zeros(0, np.int32)
    v = rng.uniform(-1, 1, rp[-1]).astype(np.float32) if value_type == "f32" else rng.integers(-9, 9, rp[-1]).astype(np.int32)
    return gen.CSR(len(lens), n, rp.astype(np.int32), ci, v)


LENS = {
    "edges": [31, 1, 32, 0, 448, 512, 511, 1, 0, 0, 513, 33, 480],
    "hub": [0] * 40 + [5, 4000, 7] + [0] * 70 + [1] * 100 + [2500],
    "ones": [1] * 1100,
    "empties": [0] * 600 + [3] + [0] * 600,
}


@pytest.mark.parametrize("value_type", ["f32", "i32"])
@pytest.mark.parametrize("tile", [(1, 4096), (13, 4096), (64, 700), (5, 128), (2000, 41)])
@pytest.mark.parametrize("lens", list(LENS))
def test_round_trip(lens, tile, value_type):
    from bcl_b200.containers import BlockCustom, SPMatrix, split_tiles
    a = matrix(LENS[lens], 4096, value_type, seed=len(lens))
    S = SPMatrix.from_csr(a, BlockCustom(tile))
    trp, toff, ci, v = split_tiles(a, *tile)
    nnz = int(toff[-1])
    assert np.array_equal(S.tile_row_ptr.cpu().numpy(), trp) and np.array_equal(S.tile_offset.cpu().numpy(), toff)
    assert np.array_equal(S.col_ind[:nnz].cpu().numpy(), ci) and np.array_equal(S.vals[:nnz].cpu().numpy(), v)
    back = S.get()
    assert np.array_equal(back.row_ptr, a.row_ptr) and np.array_equal(back.col_ind, a.col_ind)
    assert np.array_equal(back.vals, a.vals)


@pytest.mark.parametrize("at", [0, 30, 31, 32, 511, 512, 513, 4040, 4041])
@pytest.mark.parametrize("fault", ["repeat", "descend", "negative", "beyond"])
def test_refused_wherever_the_fault_lies(at, fault):
    from bcl_b200 import _lib
    from bcl_b200.containers import BlockCustom, SPMatrix
    a = matrix([20, 4000, 30], 6000, seed=3)
    ci = a.col_ind.copy()
    same_row = at not in (0, 20, 4020)
    if fault in ("repeat", "descend"):
        at = at if same_row else at + 1
        ci[at] = ci[at - 1] - (fault == "descend")
    else:
        ci[at] = -1 if fault == "negative" else a.n
    with pytest.raises(_lib.BclxError):
        SPMatrix.from_csr(gen.CSR(a.m, a.n, a.row_ptr, ci, a.vals), BlockCustom((2, 1000)))


def test_descending_row_pointer_refused():
    from bcl_b200 import _lib
    from bcl_b200.containers import BlockCustom, SPMatrix
    a = matrix([20, 40, 30], 600, seed=3)
    rp = a.row_ptr.copy()
    rp[2] = 10
    with pytest.raises(_lib.BclxError):
        SPMatrix.from_csr(gen.CSR(a.m, a.n, rp, a.col_ind, a.vals), BlockCustom((2, 100)))


def test_descriptors_are_the_tiles():
    from bcl_b200.containers import BlockCustom, SPMatrix
    a = matrix(LENS["edges"], 4096)
    S = SPMatrix.from_csr(a, BlockCustom((5, 1500)))
    d, o = S.desc.cpu().numpy(), S.tile_offset.cpu().numpy()
    for t in range(S.gm * S.gn):
        m, n = S.tile_shape((t // S.gn, t % S.gn))
        assert list(d[t]) == [m, n, o[t + 1] - o[t], S.tile_row_ptr.data_ptr() + t * (S.tm + 1) * 4,
                              S.col_ind.data_ptr() + 4 * o[t], S.vals.data_ptr() + 4 * o[t], 0]
