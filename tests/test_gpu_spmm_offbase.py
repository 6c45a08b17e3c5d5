"""Dense tiles whose bases lie one element off 16 bytes while their rows are whole
16-byte vectors apart (tiles of a larger array, handed over by address): wide
and narrow ones, a grid where only some tiles do, several rows to a warp and
one, long rows listed or not, a last tile column of another width.  Bit for bit
the oracle's; the elements around the tiles stay as they were."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O

from gpu_util import bits
from test_gpu_spmm import heavy_rows_matrix

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.fixture(scope="module")
def matrix():
    return heavy_rows_matrix(n=1024, light=5, heavy=(900, 600, 300, 129, 128, 127, 33, 32, 31))


def as_u16(t):
    import torch
    return t.contiguous().view(torch.int16).cpu().numpy().view(np.uint16)


@pytest.mark.parametrize("listed", ["0", "65536"])
@pytest.mark.parametrize("which", ["b", "c", "both", "some"])
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("n,tiles", [(264, (300, 400, 264)), (256, (1024, 1024, 256)), (136, (256, 32, 136)),
                                     (300, (512, 350, 200)), (16, (300, 400, 16)), (64, (256, 50, 64)),
                                     (40, (512, 350, 16))])
def test_grid(monkeypatch, matrix, n, tiles, dtype, which, listed):
    import torch
    from bcl_b200 import _lib
    from bcl_b200._lib import DGrid
    from bcl_b200.containers import BlockCustom, DMatrix, SPMatrix, context
    monkeypatch.setenv("BCLX_SPMM_LONG_MIN_ROWS", listed)
    a, tdt, code = matrix, torch.float32 if dtype == "f32" else torch.bfloat16, _lib.F32 if dtype == "f32" else _lib.BF16
    g = torch.Generator().manual_seed(n)
    b, c0 = torch.randn(a.n, n, generator=g).to(tdt), torch.randn(a.m, n, generator=g).to(tdt)
    A = SPMatrix.from_csr(a, BlockCustom(tiles[:2]))
    B, C = DMatrix.from_array(b, BlockCustom(tiles[1:]), dtype=tdt), DMatrix.from_array(c0, BlockCustom((tiles[0], tiles[2])), dtype=tdt)
    keep = []

    def moved(d, off):
        """The tiles in an array of their own, each a whole number of vectors and
        (where `off` says so) one element from its start."""
        pitch = d.tm * d.tn + 16
        store = torch.full((d.gm * d.gn * pitch + 16,), 7.0, dtype=tdt, device="cuda")
        at = torch.arange(d.gm * d.gn, device="cuda") * pitch + torch.as_tensor(off, device="cuda", dtype=torch.int64)
        idx = at[:, None] + torch.arange(d.tm * d.tn, device="cuda")[None]
        store[idx.reshape(-1)] = d.tiles.reshape(-1)
        ptrs = (store.data_ptr() + at * store.element_size()).contiguous()
        keep.append((store, ptrs))
        return DGrid(d.m, d.n, d.tm, d.tn, d.gm, d.gn, ptrs.data_ptr(), code, 0), store, idx

    some = lambda d: [(t % 3 == 1) * 1 for t in range(d.gm * d.gn)]  # noqa: E731
    ones = lambda d: [1] * (d.gm * d.gn)  # noqa: E731
    none = lambda d: [0] * (d.gm * d.gn)  # noqa: E731
    off_b, off_c = {"b": (ones, none), "c": (none, ones), "both": (ones, ones), "some": (some, some)}[which]
    gb, gc = moved(B, off_b(B)), moved(C, off_c(C))
    _lib.call("bclx_spmm_grid", context().use_current_stream(), ctypes.byref(A.spgrid()), ctypes.byref(gb[0]), ctypes.byref(gc[0]))
    C.tiles.copy_(gc[1][gc[2].reshape(-1)].view_as(C.tiles))
    got = C.get_matrix().cpu()
    if dtype == "f32":
        assert np.array_equal(bits(got.numpy()), bits(O.spmm_tiled(a, b.numpy(), c0.numpy(), *tiles)))
    else:
        assert np.array_equal(as_u16(got), O.spmm_tiled_bf16(a, as_u16(b), as_u16(c0), *tiles))
    rest = torch.ones_like(gc[1], dtype=torch.bool)
    rest[gc[2].reshape(-1)] = False
    assert bool((gc[1][rest] == 7).all())
