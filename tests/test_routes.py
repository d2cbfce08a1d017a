"""Which kernel takes a call that two of them could: the faster one as measured, by a rule on sizes. Results are checked where the
kernels are tested; these are the sides of the line."""
import pytest
import torch

from luma_b200 import ffi, high

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,s,kv,hq,hkv,d,path", [
    # 64 rows per KV head without GQA are four passes over all of K/V here, one there: 1.7 to 2.7 times slower
    (16, 64, 1600, 32, 32, 128, "prefill_tcgen05"), (64, 64, 512, 32, 32, 128, "prefill_tcgen05"), (4, 64, 2048, 32, 32, 64, "prefill_tcgen05"),
    (64, 16, 4096, 32, 8, 128, "prefill_tcgen05"), (64, 64, 64, 32, 32, 128, "prefill_tcgen05"),
    # ... except alone over a long range, which one CTA per tile pair walks by itself
    (1, 64, 8192, 32, 32, 128, "decode_splitk"), (1, 16, 8192, 32, 8, 128, "decode_splitk"), (4, 16, 8192, 32, 8, 128, "decode_splitk"),
    # one or two row blocks: whatever leaves the prefill kernel's CTAs a long walk or several waves
    (16, 4, 8192, 32, 8, 128, "decode_splitk"), (8, 1, 4000, 32, 8, 128, "decode_splitk"), (64, 4, 1600, 64, 8, 128, "decode_splitk"),
    (64, 1, 64, 32, 32, 128, "decode_splitk"), (1, 4, 512, 32, 8, 128, "prefill_tcgen05"), (4, 4, 64, 32, 8, 128, "prefill_tcgen05"),
])
def test_few_rows_go_to_the_faster_kernel(b, s, kv, hq, hkv, d, path):
    q = torch.zeros(b, s, hq, d, dtype=torch.bfloat16, device="cuda")
    k = torch.zeros(b, kv, hkv, d, dtype=torch.bfloat16, device="cuda")
    high.flash_attn_func(q, k, k, start_pos=kv - s)
    torch.cuda.synchronize()
    assert ffi.last_path() == path
