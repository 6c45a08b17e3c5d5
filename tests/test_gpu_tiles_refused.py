"""Calls that the slicing and the gather refuse leave their outputs as they were."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


@pytest.mark.parametrize("rp,ci", [([0, 2, 4, 6], [0, 5, 5, 1, 2, 3]),     # not ascending
                                   ([0, 2, 4, 6], [0, 5, 1, 1, 2, 3]),     # a column twice
                                   ([0, 2, 4, 6], [0, 5, 1, 9, 2, 3]),     # past the last column
                                   ([0, 2, 4, 6], [-1, 5, 1, 2, 2, 3]),    # before the first
                                   ([0, 4, 2, 6], [0, 1, 2, 3, 4, 5])])    # a row pointer that descends
def test_slicing(rp, ci):
    import torch
    from bcl_b200 import _lib
    from bcl_b200._lib import CSRDesc, SpGridOut
    from bcl_b200.containers import context
    m, n, tm, tn = 3, 8, 2, 3
    t = [torch.tensor(x, dtype=torch.int32, device="cuda") for x in (rp, ci, [1] * 6)]
    a = CSRDesc(m, n, 6, t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(), _lib.I32, 0)
    outs = [torch.full((6 * (tm + 1),), -7, dtype=torch.int32, device="cuda"), torch.full((7,), -7, dtype=torch.int64, device="cuda"),
            torch.full((6,), -7, dtype=torch.int32, device="cuda"), torch.full((6,), -7, dtype=torch.int32, device="cuda")]
    out = SpGridOut(m, n, tm, tn, 2, 3, *(o.data_ptr() for o in outs), _lib.I32, 0)
    rc = _lib.load().bclx_csr_to_tiles(context().use_current_stream(), ctypes.byref(a), ctypes.byref(out))
    assert rc == _lib.ERR_INVALID
    for o in outs:
        assert bool((o == -7).all())


def test_gather_without_arrays():
    import torch
    from bcl_b200 import _lib, gen
    from bcl_b200.containers import BlockCustom, SPMatrix, context
    s = SPMatrix.from_csr(gen.erdos_renyi(50, 3, seed=2), BlockCustom((20, 20)))
    rp = torch.full((51,), -7, dtype=torch.int32, device="cuda")
    rc = _lib.load().bclx_tiles_to_csr(context().use_current_stream(), ctypes.byref(s.spgrid()), ctypes.c_void_p(rp.data_ptr()),
                                       None, None)
    assert rc == _lib.ERR_INVALID and bool((rp == -7).all())
    empty = SPMatrix.zeros((50, 50), BlockCustom((20, 20)), dtype=np.float32)
    rc = _lib.load().bclx_tiles_to_csr(context().use_current_stream(), ctypes.byref(empty.spgrid()), ctypes.c_void_p(rp.data_ptr()),
                                       None, None)
    assert rc == _lib.OK and bool((rp == 0).all())
