"""The row unpad kernel: odd widths, blocks of rows, alignments."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


# narrow, ordinary and wide rows, row counts around a block's, and tensors that are only 4-byte aligned, which are
# written element by element
@pytest.mark.parametrize("d", [7, 9, 11, 83, 273, 383, 385])
@pytest.mark.parametrize("rows", [1, 31, 33, 1000])
@pytest.mark.parametrize("offset", [0, 2])
def test_unpad_rows(d, rows, offset):
    from flashy_linear_attention_b200 import _lib, ops

    dpad = (d + 7) // 8 * 8
    src = torch.randn(rows, dpad, device=DEV).bfloat16()
    buf = torch.full((offset + rows * d + 16,), 7.0, dtype=torch.bfloat16, device=DEV)
    out = buf[offset:offset + rows * d]
    ops._rows_call("fla_sm100_unpad_rows", src, out, rows, d, dpad)
    assert torch.equal(out.view(rows, d), src[:, :d])
    assert bool((buf[:offset] == 7.0).all()) and bool((buf[offset + rows * d:] == 7.0).all())
