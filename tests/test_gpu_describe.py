"""Tile descriptors of a packed grid: matrices without rows or columns."""
import pytest

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
