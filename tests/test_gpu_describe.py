"""Tile descriptors of a packed grid: matrices without rows or columns, and
offsets in every form that the constructor takes."""
import numpy as np
import pytest

from bcl_b200 import gen

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("shape", [(0, 40), (40, 0), (0, 0)])
def test_matrix_without_rows_or_columns(shape):
    from bcl_b200.containers import BlockCustom, SPMatrix
    s = SPMatrix.zeros(shape, BlockCustom((16, 16)))
    assert s.shape() == shape and s.nnz() == 0 and s.desc.shape == (0, 7)


@pytest.mark.parametrize("form", ["int64", "host", "int32", "strided", "host int32"])
def test_offsets_of_any_form(form):
    import torch
    from bcl_b200.containers import SPMatrix, split_tiles
    a = gen.erdos_renyi(300, 4, seed=3)
    rp, off, ci, v = (torch.from_numpy(x).cuda() for x in split_tiles(a, 70, 110))
    given = {"int64": off, "host": off.cpu(), "int32": off.to(torch.int32), "host int32": off.to(torch.int32).cpu(),
             "strided": torch.stack([off, off + 1], 1)[:, 0]}[form]
    s = SPMatrix(a.m, a.n, 70, 110, np.float32, 0, rp, given, ci, v)
    nt = s.gm * s.gn
    ti, tj = np.divmod(np.arange(nt), s.gn)
    o = off.cpu().numpy()
    want = np.stack([np.minimum(70, a.m - 70 * ti), np.minimum(110, a.n - 110 * tj), np.diff(o),
                     rp.data_ptr() + np.arange(nt) * 71 * 4, ci.data_ptr() + 4 * o[:-1], v.data_ptr() + 4 * o[:-1],
                     np.zeros(nt, np.int64)], 1)
    assert np.array_equal(s.desc.cpu().numpy(), want)
    back = s.get()
    assert np.array_equal(back.row_ptr, a.row_ptr) and np.array_equal(back.col_ind, a.col_ind)


@pytest.mark.parametrize("device", [0, None, "cuda:0"])
def test_device_as_the_other_tensors_name_it(device):
    """`device` may be what the caller calls the tensors' device: the tensors decide."""
    import torch
    from bcl_b200.containers import SPMatrix, split_tiles
    a = gen.erdos_renyi(50, 2, seed=4)
    parts = [torch.from_numpy(x).cuda() for x in split_tiles(a, 20, 50)]
    s = SPMatrix(a.m, a.n, 20, 50, np.float32, torch.device(device) if isinstance(device, str) else device, *parts)
    assert s.desc[:, 2].tolist() == np.diff(parts[1].cpu().numpy()).tolist()
