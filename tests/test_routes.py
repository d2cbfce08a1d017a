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
    (64, 1, 64, 32, 32, 128, "decode_splitk"), (16, 4, 64, 32, 8, 128, "decode_splitk"), (4, 16, 1600, 32, 8, 128, "decode_splitk"), (1, 4, 512, 32, 8, 128, "prefill_tcgen05"), (4, 4, 64, 32, 8, 128, "prefill_tcgen05"),
])
def test_few_rows_go_to_the_faster_kernel(b, s, kv, hq, hkv, d, path):
    q = torch.zeros(b, s, hq, d, dtype=torch.bfloat16, device="cuda")
    k = torch.zeros(b, kv, hkv, d, dtype=torch.bfloat16, device="cuda")
    high.flash_attn_func(q, k, k, start_pos=kv - s)
    torch.cuda.synchronize()
    assert ffi.last_path() == path


def _packed(q_lens, k_lens, hq, hkv, d, page=16):
    cu = [torch.tensor([0] + x, dtype=torch.int32).cumsum(0).int().cuda() for x in (q_lens, k_lens)]
    pages = -(-max(k_lens) // page)
    k = torch.zeros(len(k_lens) * pages, page, hkv, d, dtype=torch.bfloat16, device="cuda")
    table = torch.arange(len(k_lens) * pages, dtype=torch.int32, device="cuda").view(len(k_lens), pages)
    q = torch.zeros(sum(q_lens), hq, d, dtype=torch.bfloat16, device="cuda")
    high.flash_attn_varlen_func(q, k, k, *cu, max(q_lens), max(k_lens), block_table=table)
    torch.cuda.synchronize()
    assert ffi.last_path() == "prefill_tcgen05"
    return ffi.last_launches()


@pytest.mark.parametrize("q_lens,keys,hq,hkv,d,launches", [
    ([512] * 4, 8192, 32, 8, 128, 1),                # no room for few rows next to the prompts
    ([512] * 4 + [1], 8192, 32, 8, 128, 1),          # a few that fill up the prefill grid's last wave
    ([64] + [1] * 8, 2048, 32, 8, 128, 1),           # all in one wave
    ([64] * 2 + [1] * 32, 2048, 8, 2, 64, 1),
    ([512] * 4 + [1] * 32, 8192, 32, 8, 128, 2),     # waves of almost empty tiles
    ([64] + [1] * 128, 512, 32, 8, 128, 2),
    ([512] + [1] * 32, 2048, 64, 8, 64, 2),
])
def test_few_rows_of_a_packed_batch_leave_the_prefill_grid_where_they_make_waves(q_lens, keys, hq, hkv, d, launches):
    assert _packed(q_lens, [max(keys, n) for n in q_lens], hq, hkv, d) == launches
