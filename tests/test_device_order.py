"""The order of tile pairs that is found on the device (find_item in csrc/prefill_tcgen05.cu), asked for with option
"prefill_order" = 2 where the launch would not choose it: every row is computed exactly once whatever the lengths are, bit for bit
as in grid order."""
import numpy as np
import pytest
import torch

from luma_b200 import ffi, low
from tests import helpers as H

pytestmark = pytest.mark.gpu


def with_option(name, value, call):
    ffi.lib.flash_attn_set_option(name, value)
    try:
        return call()
    finally:
        ffi.lib.flash_attn_set_option(name, 0)


@pytest.mark.parametrize("sq,hq,hkv,d,page,lens", [
    (128, 8, 2, 128, 16, [1700, 128, 2300, 129, 400]),                      # one row block
    (129, 3, 3, 64, 32, [2200, 129, 0, 1025, 130, 100, 1024]),              # one row more, an empty sequence
    (200, 6, 2, 32, 8, [1281, 200, 640, 1280]),                             # an odd group
    (72, 2, 2, 64, 16, [72 + 37 * (i % 30) for i in range(33)]),            # more sequences than lanes
    (65, 1, 1, 64, 128, [65 + (i * 53) % 200 for i in range(256)]),         # as many as a warp holds
    (65, 1, 1, 64, 128, [65 + (i * 53) % 200 for i in range(257)]),         # one more: grid order
    (512, 32, 8, 128, 16, [8192, 600, 1024, 513]),                          # more than a wave: the launch's own choice
])
def test_chunks_over_pages(sq, hq, hkv, d, page, lens):
    kc, vc, table = H.make_paged_cache(lens, page, hkv, d, seed=sq + d)
    q = H.normal((len(lens), sq, hq, d), 51)
    dev = [H.to_dev(x, "bf16") for x in (q, kc, vc)]
    tab, cl = torch.from_numpy(table).cuda(), torch.tensor(lens, dtype=torch.int32, device="cuda")

    def call():
        o = torch.full_like(dev[0], float("nan"))
        low.flash_attn_with_kvcache(*dev, o, tab, cl, len(lens), sq, hq, hkv, d, page, table.shape[1], 1.0 / np.sqrt(d))
        torch.cuda.synchronize()
        assert ffi.last_path() == "prefill_tcgen05"
        return o
    grid = with_option(b"prefill_band", 1, call)
    assert torch.isfinite(grid).all()
    assert torch.equal(grid, with_option(b"prefill_order", 2, call)) and torch.equal(grid, call())


@pytest.mark.parametrize("total", [True, False])
@pytest.mark.parametrize("q_lens,k_lens,hq,hkv,d", [
    ([256, 1, 130, 1, 3, 200], [2048, 1900, 130, 64, 700, 1500], 8, 2, 128),
    ([100, 0, 128, 7], [2000, 0, 128, 1200], 2, 1, 64),
    ([300] + [1] * 40, [2500] + [1900] * 40, 32, 8, 128),                   # enough of them to go behind
])
def test_packed_chunks_over_pages(q_lens, k_lens, hq, hkv, d, total):
    page = 16
    kc, vc, table = H.make_paged_cache(k_lens, page, hkv, d, seed=9)
    cu_q, cu_k = (torch.from_numpy(np.concatenate([[0], np.cumsum(x)]).astype(np.int32)).cuda() for x in (q_lens, k_lens))
    dev = [H.to_dev(x, "bf16") for x in (H.normal((sum(q_lens), hq, d), 61), kc, vc)]
    tab = torch.from_numpy(table).cuda()

    def call():
        o = torch.full_like(dev[0], float("nan"))
        low.flash_attn_varlen(*dev, o, cu_q, cu_k, len(q_lens), max(q_lens), max(k_lens), hq, hkv, d, 1.0 / np.sqrt(d), tab, page,
                              total_q=sum(q_lens) if total else None)
        torch.cuda.synchronize()
        assert ffi.last_path() == "prefill_tcgen05"
        return o
    grid = with_option(b"prefill_band", 1, call)
    assert torch.isfinite(grid).all()
    assert torch.equal(grid, with_option(b"prefill_order", 2, call)) and torch.equal(grid, call())
