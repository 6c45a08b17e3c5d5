"""Rows that a warp walks alone over a large B, their slices asked for ahead (k_spmm).
Bit for bit the oracle's."""
import numpy as np
import pytest

from bcl_b200 import gen
from oracle import oracle as O

from gpu_util import bits
from test_gpu_spmm import run

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("tile_k", [100000, 3000])
def test_long_rows_alone_with_a_large_b(dtype, tile_k):
    """Rows of 255 to 3,000 entries that warps walk alone over a B of 48 MB and more
    (slices asked for ahead), on one tile along k and on 34."""
    n = 132 if dtype == "f32" else 264
    rng = np.random.default_rng(7)
    lens = np.array([0, 255, 256, 257, 3000, 3, 1000, 288])
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    ci = np.concatenate([np.sort(rng.choice(100000, k, replace=False)) for k in lens]).astype(np.int32)
    a = gen.CSR(len(lens), 100000, rp, ci, rng.uniform(-1, 1, ci.size).astype(np.float32))
    b, c0 = rng.standard_normal((a.n, n)).astype(np.float32), rng.standard_normal((a.m, n)).astype(np.float32)
    tiles = (a.m, tile_k, n)
    if dtype == "f32":
        assert np.array_equal(bits(run(a, b, tiles, c0=c0)), bits(O.spmm_tiled(a, b, c0, *tiles)))
    else:
        b, c0 = O.to_bf16(b), O.to_bf16(c0)
        assert np.array_equal(run(a, b, tiles, dtype="bf16", c0=c0), O.spmm_tiled_bf16(a, b, c0, *tiles))


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("n,tk", [(16, 31), (24, 60), (47, 31), (33, 60), (130, 40), (201, 32)])
def test_chains_over_more_than_32_tiles(monkeypatch, dtype, n, tk):
    """Long rows of narrow and unaligned tiles whose entries lie in two and three
    groups of 32 stages, in the first or the last one alone, and rows without
    entries in the first."""
    monkeypatch.setenv("BCLX_SPMM_LONG_MIN_ROWS", "0")
    rng = np.random.default_rng(n)
    k = 2000
    spans = [(0, k, 1900), (0, k, 1200), (0, 500, 500), (1500, k, 500), (900, 1900, 700), (0, k, 1025), (0, k, 40), (0, 0, 0)] * 6
    rows = [np.sort(lo + rng.choice(hi - lo, c, replace=False)) if c else np.zeros(0, np.int64) for lo, hi, c in spans]
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    ci = np.concatenate(rows).astype(np.int32)
    a = gen.CSR(len(rows), k, rp, ci, rng.uniform(-1, 1, ci.size).astype(np.float32))
    b, c0 = rng.standard_normal((k, n)).astype(np.float32), rng.standard_normal((a.m, n)).astype(np.float32)
    tiles = (20, tk, n)
    if dtype == "f32":
        assert np.array_equal(bits(run(a, b, tiles, c0=c0)), bits(O.spmm_tiled(a, b, c0, *tiles)))
    else:
        b, c0 = O.to_bf16(b), O.to_bf16(c0)
        assert np.array_equal(run(a, b, tiles, dtype="bf16", c0=c0), O.spmm_tiled_bf16(a, b, c0, *tiles))
