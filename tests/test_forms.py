"""Which form of a kernel ran (flash_attn_last_form), at the sizes of the tests that are there for that form and at more where those leave one out: the f32 kernels with warp-wide products and on
the tensor cores, tile pairs with a CTA and with a cluster, few rows ahead of the prompts of a packed batch and behind them, which kernel takes few rows. Each call is compared with the f64 oracle as well."""
import math

import numpy as np
import pytest
import torch

import tests.test_few_rows_routes as routes
import tests.test_mixed_side_by_side as mixed
import tests.test_shared_keys as shared
import tests.test_tile_f32_tcgen05 as f32
from luma_b200 import ffi, low
from oracle import binding as ob
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,sq,skv,hq,hkv,d,sp,form", [
    (1, 256, 256, 8, 8, 64, 0, "tcgen05 cluster 4"), (2, 257, 257, 4, 4, 32, 0, "mma"), (1, 193, 193, 2, 2, 128, 0, "tcgen05 cluster 4"),
    (1, 1000, 1000, 8, 8, 128, 0, "tcgen05 cluster 2"), (2, 500, 500, 8, 4, 64, 0, "tcgen05 cluster 2"), (2, 400, 400, 9, 9, 32, 0, "tcgen05 cluster 2"),
    (1, 5, 1025, 2, 2, 64, 1020, "tcgen05 cluster 8"), (1, 1, 4000, 4, 1, 128, 3999, "tcgen05 cluster 8"), (1, 3, 449, 1, 1, 32, 446, "tcgen05 cluster 8"),
    (1, 43, 300, 9, 3, 64, 257, "tcgen05 cluster 4"), (1, 64, 257, 4, 2, 64, 193, "tcgen05 cluster 4"), (1, 300, 200, 4, 2, 64, 0, "tcgen05 cluster 4"), (1, 200, 300, 6, 2, 128, 0, "tcgen05 cluster 4"),
    (1, 280, 280, 16, 4, 64, 0, "tcgen05 cluster 2"), (1, 320, 320, 8, 8, 32, 0, "tcgen05 cluster 4"), (1, 256, 256, 8, 2, 32, 0, "mma"), (1, 200, 200, 16, 4, 32, 0, "tcgen05 cluster 4"),
    (4, 64, 64, 16, 4, 64, 0, "mma"), (3, 80, 80, 16, 4, 64, 0, "mma"), (24, 33, 33, 8, 8, 64, 0, "mma"), (5, 80, 80, 16, 4, 64, 0, "tcgen05 cluster 2"), (24, 64, 64, 8, 8, 64, 0, "tcgen05"),
    (3, 160, 160, 8, 8, 32, 0, "mma"), (4, 96, 96, 16, 4, 32, 0, "tcgen05 cluster 2"), (4, 128, 128, 8, 8, 32, 0, "mma"),   # both sides of the line
    (4, 400, 400, 16, 8, 64, 0, "tcgen05"), (2, 513, 513, 24, 24, 32, 0, "tcgen05"), (3, 330, 330, 12, 12, 128, 0, "tcgen05"),
])
def test_f32(b, sq, skv, hq, hkv, d, sp, form):
    f32.test_batched_with_lse(b, sq, skv, hq, hkv, d, sp)
    assert ffi.last_form() == form


@pytest.mark.parametrize("d", [32, 64, 128])
def test_f32_with_a_mask_and_over_pages(d):
    for b, form in ((1, "mma" if d == 32 else "tcgen05 cluster 4"), (2, "tcgen05 cluster 2"), (30, "tcgen05")):
        f32.test_padding_mask(b, d)
        assert ffi.last_form() == form
    for bs in (0, 5, 16):
        for seqs in (1, 12):
            f32.test_packed_and_paged(bs, seqs)
            assert ffi.last_form() == "tcgen05"


@pytest.mark.parametrize("d,dt", [(128, "bf16"), (64, "f16"), (32, "bf16")])
@pytest.mark.parametrize("b,sq,skv,hq,hkv,sp,masked,ctas", [
    (1, 70, 4500, 2, 1, 4430, False, 8), (3, 129, 2100, 4, 4, 1971, False, 4), (1, 1700, 1700, 6, 2, 0, False, 2), (2, 1700, 1700, 6, 2, 0, False, 1), (1, 300, 1800, 3, 3, 0, False, 4),
    (2, 200, 2000, 4, 2, 1800, True, 4), (4, 1, 1100, 8, 2, 1099, True, 4), (3, 4, 1000, 4, 1, 996, True, 4), (3, 400, 1700, 10, 5, 1300, True, 2),
])
def test_shared_keys(b, sq, skv, hq, hkv, sp, masked, ctas, d, dt):
    shared.test_batched(b, sq, skv, hq, hkv, sp, masked, d, dt)
    assert ffi.last_form() in ([f"cluster {ctas}"] if ctas > 1 else ["pairs", "one pair"])


@pytest.mark.parametrize("d", [128, 64])
@pytest.mark.parametrize("sq,hq,hkv,page,lens,ctas", [
    (100, 4, 1, 16, [4200, 100, 130], 8), (130, 3, 1, 32, [1800, 0, 131, 40], 4), (65, 16, 2, 128, [2900, 600], 4), (70, 8, 8, 8, [1700, 70, 1000], 4), (200, 16, 8, 16, [1700, 200, 1000], 2),
])
def test_shared_keys_over_pages(sq, hq, hkv, page, lens, ctas, d):
    shared.test_chunks_over_pages(sq, hq, hkv, page, lens, d)
    assert ffi.last_form() == f"cluster {ctas}"


@pytest.mark.parametrize("paged", [False, True])
@pytest.mark.parametrize("total", [False, True])
def test_shared_keys_of_packed_buffers(paged, total):
    # with four query heads the host has to take sequences of a few rows into account where it does not know the rows; 32 to a KV head are never few
    shared.test_packed(paged, total)
    assert ffi.last_form() == ("cluster 4" if total else "few rows behind")
    dt, d, page, hq, hkv = "f16", 128, 16, 32, 1
    ql, kl = [40, 17, 0, 33, 8], [1900, 17, 0, 2500, 300]
    cu_q, cu_k = (np.concatenate([[0], np.cumsum(x)]).astype(np.int32) for x in (ql, kl))
    q, table = H.round_to(H.normal((sum(ql), hq, d), 5), dt), None
    if paged:
        k, v, table = H.make_paged_cache(kl, page, hkv, d, seed=6)
    else:
        k, v = (H.normal((sum(kl), hkv, d), x) for x in (6, 7))
    k, v = H.round_to(k, dt), H.round_to(v, dt)
    want = ob.attn_f64_varlen(q, k, v, cu_q, cu_k, block_table=table) if paged else ob.attn_f64_varlen(q, k, v, cu_q, cu_k)
    dev = [H.to_dev(x, dt) for x in (q, k, v)]
    o = torch.full_like(dev[0], float("nan"))
    low.flash_attn_varlen(*dev, o, torch.from_numpy(cu_q).cuda(), torch.from_numpy(cu_k).cuda(), len(ql), max(ql), max(kl), hq, hkv, d, 1.0 / math.sqrt(d),
                          torch.from_numpy(table).cuda() if paged else None, page if paged else 1, total_q=sum(ql) if total else None, total_k=sum(kl) if total and not paged else None)
    torch.cuda.synchronize()
    assert (ffi.last_path(), ffi.last_form()) == ("prefill_tcgen05", "cluster 4") and ffi.device_status() == 0
    H.assert_bf16_close(H.to_np(o), want, "packed")


@pytest.mark.parametrize("decoding,prompts,longest,hq,hkv,d,dt,several,form", [
    (200, 1, 1500, 8, 2, 128, "bf16", False, "ahead"), (200, 1, 1500, 8, 2, 128, "f16", True, "ahead"), (80, 2, 1300, 8, 2, 64, "bf16", False, "ahead"), (300, 2, 700, 8, 2, 128, "f16", False, "ahead"),
    (60, 2, 2000, 8, 8, 128, "bf16", True, "ahead"), (120, 3, 1100, 8, 8, 128, "bf16", True, "behind"),
    (16, 1, 260, 32, 8, 64, "bf16", False, "ahead"), (20, 1, 260, 32, 32, 128, "bf16", False, "ahead"), (40, 3, 200, 32, 32, 128, "bf16", False, "behind"),   # the ends of short sequences
])
def test_mixed_batches(decoding, prompts, longest, hq, hkv, d, dt, several, form):
    mixed.test_rows_of_both_kernels(decoding, prompts, longest, hq, hkv, d, dt, several)
    assert ffi.last_form() == f"few rows {form}"


@pytest.mark.parametrize("b,s,kv,hq,hkv,d,path", [
    (9, 16, 1200, 32, 8, 64, "prefill_tcgen05"), (9, 12, 1200, 32, 8, 64, "decode_splitk"), (3, 8, 500, 32, 32, 64, "prefill_tcgen05"), (3, 8, 513, 32, 32, 64, "decode_splitk"),
    (12, 8, 300, 8, 8, 64, "prefill_tcgen05"), (12, 8, 385, 8, 8, 64, "decode_splitk"),
])
def test_few_rows_of_one_wave(b, s, kv, hq, hkv, d, path):
    routes.test_sides_of_the_line(b, s, kv, hq, hkv, d, path)
