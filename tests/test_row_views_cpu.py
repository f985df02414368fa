"""Rows as the CUDA ops hand them to kernels that read 16-byte pieces."""
import pytest
import torch

from tensorrt_edge_llm_b200.ops.cuda import _aligned, _rows


@pytest.mark.parametrize("rows", [1, 2, 5])
@pytest.mark.parametrize("width,pitch", [(64, 64), (64, 96), (64, 67), (8, 8)])
@pytest.mark.parametrize("offset", [0, 1, 3, 8])
def test_rows_start_on_16_bytes(rows, width, pitch, offset):
    base = torch.arange(rows * pitch + offset + 16, dtype=torch.int16)[offset:]
    t = base[:rows * pitch].view(rows, pitch)[:, :width]
    for view in (t, t.unflatten(1, (2, -1))):
        got, ld = _rows(view)
        assert got.data_ptr() % 16 == 0 and (rows == 1 or ld * got.element_size() % 16 == 0) and ld >= width
        assert torch.equal(got.as_strided((rows, width), (ld, 1)), t)
        if view.data_ptr() % 16 == 0 and pitch % 8 == 0:
            assert got.data_ptr() == view.data_ptr()                     # nothing is copied without need
    packed = _aligned(t)
    assert packed.is_contiguous() and packed.data_ptr() % 16 == 0 and torch.equal(packed, t)


def test_rows_of_an_empty_step():
    t, ld = _rows(torch.empty(0, 64))
    assert t.shape == (0, 64) and ld == 0
