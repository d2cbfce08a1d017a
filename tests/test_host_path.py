"""The native host path (csrc/host_fast.cpp) against the Python path beside it: which calls it takes, that both give the same,
and that what it does not take raises what the Python path raises."""
import pytest
import torch

from luma_b200 import error as E
from luma_b200 import low

gpu = pytest.mark.gpu


@gpu
def test_sizes_whose_product_does_not_fit_64_bits_are_too_large_for_any_buffer():
    # 2^16 * 2^16 * 2^25 * 2^7 = 2^64, which wraps to 0 elements
    t = torch.zeros(1024, dtype=torch.bfloat16, device="cuda")
    with pytest.raises(E.BufferTooSmall):
        low.flash_attn(t, t, t, t, 1 << 16, 1 << 16, 1 << 16, 1 << 25, 1 << 25, 128, 0, 1.0)
    i = torch.zeros(4, dtype=torch.int32, device="cuda")
    with pytest.raises(E.BufferTooSmall):
        low.kvcache_append(t, t, t, t, i, i, 1 << 16, 1 << 16, 1 << 25, 128, 16, 1)
