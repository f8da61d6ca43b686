"""Lengths that fp32 attention takes, without a GPU: the call gets as far as the launch (BMB_E_CUDA), it is not refused."""
import pytest

E_CUDA = 2


@pytest.mark.parametrize("T", [64 * 65535, 64 * 65535 + 1, 1 << 23])
def test_no_length_is_refused(bmb, T):
    """Beyond what the split kernels' grids hold, the row-group kernels serve."""
    import torch
    if torch.cuda.is_available():
        pytest.skip("the pointers here are not memory")
    lib, p = bmb.lib(), 4096
    assert lib.bmb_flash_attention_forward_cfg(0, p, p, p, 1, T, 32, 1) == E_CUDA
    assert lib.bmb_flash_attention_backward_cfg(0, p, p, p, p, p, p, 1, T, 32, 1) == E_CUDA
