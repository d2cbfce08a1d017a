"""What the split-K kernel takes at the edges of its arguments: output alignment, lengths beyond the block table."""
import numpy as np
import pytest
import torch

from luma_b200 import ffi, low
from oracle import binding as ob
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [32, 64, 128])
@pytest.mark.parametrize("entry", ["decode", "noalloc", "allgather"])
def test_output_aligned_to_its_elements_only(entry, d):
    # an output that starts two bytes off a word: a whole sequence (finished by one CTA) and a cut one (merged)
    if entry == "noalloc" and d == 32:
        pytest.skip("the entry point takes head sizes 64 and 128")
    lens, hq, hkv, bs = [5000, 33], 8, 2, 16
    kc, vc, table = H.make_paged_cache(lens, bs, hkv, d, seed=80 + d)
    q = H.normal((2, 1, hq, d), 83)
    dq, dk, dv = (H.to_dev(x, "bf16") for x in (q, kc, vc))
    bt, cl = torch.from_numpy(table).cuda(), torch.tensor(lens, dtype=torch.int32, device="cuda")
    room = torch.zeros(dq.numel() + 2, dtype=torch.bfloat16, device="cuda")
    o = room[1:-1]
    assert o.data_ptr() % 4 == 2
    scale = float(1 / np.sqrt(d))
    if entry == "decode":
        low.flash_attn_with_kvcache(dq, dk, dv, o, bt, cl, 2, 1, hq, hkv, d, bs, bt.shape[1], scale)
    elif entry == "allgather":
        low.flash_attn_with_kvcache_allgather(dq, dk, dv, [o.data_ptr()], hq, 0, bt, cl, 2, hq, hkv, d, bs, bt.shape[1], scale)
    else:
        rc = ffi.lib.flash_attn_decode_bf16_noalloc(dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), o.data_ptr(), bt.data_ptr(), cl.data_ptr(), 2,
                                                    hq, hkv, d, bs, bt.shape[1], scale, torch.cuda.current_stream().cuda_stream)
        assert rc == 0, ffi.last_error()
    torch.cuda.synchronize()
    assert ffi.last_path() in ("decode_splitk", "decode_splitk_static")
    want = ob.attn_f64_kvcache(H.round_to(q, "bf16"), H.round_to(kc, "bf16"), H.round_to(vc, "bf16"), lens, table, scale=scale)
    H.assert_bf16_close(H.to_np(o).reshape(want.shape), want, entry)
    assert room[0] == 0 and room[-1] == 0      # and nothing beside it


@pytest.mark.parametrize("chunk", [0, 64, 1024])
@pytest.mark.parametrize("new", [1, 4])
def test_length_beyond_the_block_table_is_cut_at_its_capacity(chunk, new):
    hq, hkv, d, bs = 8, 2, 128, 16
    table_lens, lens = [2048, 2048, 2048], [2048 + 5000, 700, 2049]
    kc, vc, table = H.make_paged_cache(table_lens, bs, hkv, d, seed=90)
    q = H.normal((3, new, hq, d), 93)
    dq, dk, dv = (H.to_dev(x, "bf16") for x in (q, kc, vc))
    bt = torch.from_numpy(table).cuda()
    scale = float(1 / np.sqrt(d))

    def run(lens):
        o = torch.full_like(dq, float("nan"))
        low.flash_attn_with_kvcache(dq, dk, dv, o, bt, torch.tensor(lens, dtype=torch.int32, device="cuda"), 3, new, hq, hkv, d, bs, bt.shape[1], scale)
        assert ffi.last_path() == "decode_splitk"
        return H.to_np(o)
    rq, rk, rv = (H.round_to(x, "bf16") for x in (q, kc, vc))
    ffi.lib.flash_attn_set_option(b"decode_chunk_tokens", chunk)
    try:
        for _ in range(2):
            got = run(lens)
            for s, n in enumerate(lens):
                # a row at a position past the table sees all that the table holds
                pos = [n - new + t for t in range(new)]
                want = np.concatenate([ob.attn_f64_kvcache(rq[s:s + 1, t:t + 1], rk, rv, [min(2048, p + 1)], table[s:s + 1], scale=scale)
                                       for t, p in enumerate(pos)], axis=1)
                H.assert_bf16_close(got[s:s + 1], want, f"sequence {s} of {n} tokens")
            got = run([2048, 30, 900])        # and the next call finds everything in order
            want = ob.attn_f64_kvcache(rq, rk, rv, [2048, 30, 900], table, scale=scale)
            H.assert_bf16_close(got, want, "after")
    finally:
        ffi.lib.flash_attn_set_option(b"decode_chunk_tokens", 0)


def test_more_kv_heads_than_cta_slots_without_a_cut():
    # 1200 KV heads leave one column: every sequence is finished by one CTA, and the allocation-free entry point needs no partials
    lens, h, d, bs = [300, 65], 1200, 64, 16
    kc, vc, table = H.make_paged_cache(lens, bs, h, d, seed=70)
    q = H.normal((2, 1, h, d), 71)
    dq, dk, dv = (H.to_dev(x, "bf16") for x in (q, kc, vc))
    bt, cl, o = torch.from_numpy(table).cuda(), torch.tensor(lens, dtype=torch.int32, device="cuda"), torch.full_like(dq, float("nan"))
    want = ob.attn_f64_kvcache(H.round_to(q, "bf16"), H.round_to(kc, "bf16"), H.round_to(vc, "bf16"), lens, table, scale=0.125)
    for _ in range(2):
        rc = ffi.lib.flash_attn_decode_bf16_noalloc(dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), o.data_ptr(), bt.data_ptr(), cl.data_ptr(), 2, h, h, d,
                                                    bs, bt.shape[1], 0.125, torch.cuda.current_stream().cuda_stream)
        assert rc == 0, ffi.last_error()
        torch.cuda.synchronize()
        H.assert_bf16_close(H.to_np(o), want, "noalloc")
        o.fill_(float("nan"))
        low.flash_attn_with_kvcache(dq, dk, dv, o, bt, cl, 2, 1, h, h, d, bs, bt.shape[1], 0.125)
        torch.cuda.synchronize()
        H.assert_bf16_close(H.to_np(o), want, "workspace")


@pytest.mark.parametrize("new,hq,hkv,d", [(4, 8, 2, 128), (9, 2, 2, 64), (3, 8, 1, 32)])
def test_several_rows_over_pages_with_nan_in_every_unwritten_slot(new, hq, hkv, d):
    lens, bs = [1701, 65, 2049, 16, new], 16
    kc, vc, table = H.make_paged_cache(lens, bs, hkv, d, seed=60 + d)
    q = H.normal((len(lens), new, hq, d), 61)
    want = ob.attn_f64_kvcache(H.round_to(q, "bf16"), H.round_to(kc, "bf16"), H.round_to(vc, "bf16"), lens, table)
    written = np.zeros(kc.shape[:2], dtype=bool)
    for s, n in enumerate(lens):
        j = np.arange(n)
        written[table[s, j // bs], j % bs] = True
    kc[~written] = np.nan
    vc[~written] = np.nan
    o = torch.empty(len(lens), new, hq, d, device="cuda", dtype=torch.bfloat16)
    low.flash_attn_with_kvcache(H.to_dev(q, "bf16"), H.to_dev(kc, "bf16"), H.to_dev(vc, "bf16"), o, torch.from_numpy(table).cuda(),
                                torch.tensor(lens, dtype=torch.int32, device="cuda"), len(lens), new, hq, hkv, d, bs, table.shape[1], 1.0 / np.sqrt(d))
    torch.cuda.synchronize()
    assert ffi.last_path() == "decode_splitk"
    H.assert_bf16_close(H.to_np(o), want, f"{new} tokens")
