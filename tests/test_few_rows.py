"""A few query rows per sequence over long K/V on the split-K kernel (csrc/decode_splitk.cu) beyond single-token
paged decode: several query tokens over pages, contiguous K/V with start_pos and log-sum-exp, and the decoding
sequences of a packed batch next to prompts. Sizes sit at the edges of its tiles: 1, 15 to 17 and 64 query rows
(16 rows per block, 4 blocks), lengths around the 64-token unit and the 16-token tile, empty sequences, query
tokens that see no key, pages that are no power of two. Tolerances are those of every 16-bit kernel
(max-abs 2e-2, mean-abs 2e-3 against the f64 loop on the rounded inputs; LSE 1e-3)."""
import numpy as np
import pytest
import torch

from luma_b200 import ffi, low
from oracle import binding as ob
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sq,hq,hkv,d,bs,dt", [
    (2, 2, 2, 128, 16, "bf16"),      # 2 rows
    (15, 2, 2, 64, 16, "f16"),       # 15 rows
    (4, 16, 4, 128, 32, "bf16"),     # 16 rows: one full block
    (17, 1, 1, 32, 8, "bf16"),       # 17 rows: a second block of one row
    (8, 16, 2, 128, 16, "f16"),      # 64 rows: four blocks
    (3, 12, 2, 64, 12, "bf16"),      # 18 rows, page of 12 tokens
])
def test_several_tokens_over_pages(sq, hq, hkv, d, bs, dt):
    lens = [1700, sq, sq + 1, 63, 64, 65, 0, 129, 900, max(sq - 1, 0), 16, 1023]
    kc, vc, table = H.make_paged_cache(lens, bs, hkv, d, seed=20 + sq + d)
    kc, vc = H.round_to(kc, dt), H.round_to(vc, dt)
    q = H.round_to(H.normal((len(lens), sq, hq, d), 21), dt)
    want = ob.attn_f64_kvcache(q, kc, vc, lens, table)
    o = torch.full((len(lens), sq, hq, d), float("nan"), device="cuda", dtype=H.TORCH_DT[dt])
    args = (H.to_dev(q, dt), H.to_dev(kc, dt), H.to_dev(vc, dt), o, torch.from_numpy(table).cuda(),
            torch.tensor(lens, dtype=torch.int32, device="cuda"), len(lens), sq, hq, hkv, d, bs, table.shape[1], 1.0 / np.sqrt(d))
    first = None
    for _ in range(2):      # the arrival counts are as the first call found them
        o.fill_(float("nan"))
        low.flash_attn_with_kvcache(*args)
        torch.cuda.synchronize()
        assert ffi.last_path() == "decode_splitk"
        H.assert_bf16_close(H.to_np(o), want, f"{sq} tokens, {hq}/{hkv}, page {bs}")
        assert first is None or torch.equal(first, o)
        first = o.clone()


@pytest.mark.parametrize("b,sq,skv,sp,hq,hkv,d", [(3, 1, 1601, 1600, 8, 2, 128), (2, 4, 2000, 1996, 4, 4, 64),
                                                 (1, 3, 1665, 0, 8, 1, 32), (150, 2, 65, 63, 2, 2, 64)])
def test_contiguous_with_start_pos_and_lse(b, sq, skv, sp, hq, hkv, d):
    dt = "bf16"
    q = H.round_to(H.normal((b, sq, hq, d), 31), dt)
    k, v = H.round_to(H.normal((b, skv, hkv, d), 32), dt), H.round_to(H.normal((b, skv, hkv, d), 33), dt)
    want, lse_want = ob.attn_f64_batch(q, k, v, start_pos=sp, return_lse=True)
    o = torch.full((b, sq, hq, d), float("nan"), device="cuda", dtype=torch.bfloat16)
    lse = torch.full((b, hq, sq), float("nan"), device="cuda", dtype=torch.float32)
    low.flash_attn(H.to_dev(q, dt), H.to_dev(k, dt), H.to_dev(v, dt), o, b, sq, skv, hq, hkv, d, sp, 1.0 / np.sqrt(d), None, None, lse)
    torch.cuda.synchronize()
    assert ffi.last_path() == "decode_splitk"
    H.assert_bf16_close(H.to_np(o), want, "contiguous")
    assert np.abs(lse.cpu().numpy() - lse_want).max() <= 1e-3


@pytest.mark.parametrize("paged", [True, False])
@pytest.mark.parametrize("hq,hkv", [(8, 2), (3, 3)])
def test_decoding_sequences_of_a_packed_batch(paged, hq, hkv):
    dt, d, bs = "bf16", 128, 16
    ql = [1, 200, 1, 4, 1, 5, 16, 17, 130, 1]          # rows of one block and of more, decoded between prompts
    kl = [1650, 300, 1, 64, 777, 5, 400, 900, 130, 65]
    cu_q = np.concatenate([[0], np.cumsum(ql)]).astype(np.int32)
    cu_k = np.concatenate([[0], np.cumsum(kl)]).astype(np.int32)
    q = H.round_to(H.normal((int(cu_q[-1]), hq, d), 41), dt)
    qd = H.to_dev(q, dt)
    o = torch.full_like(qd, float("nan"))
    cq, ck = torch.from_numpy(cu_q).cuda(), torch.from_numpy(cu_k).cuda()
    if paged:
        kc, vc, table = H.make_paged_cache(kl, bs, hkv, d, seed=42)
        kc, vc = H.round_to(kc, dt), H.round_to(vc, dt)
        want = ob.attn_f64_varlen(q, kc, vc, cu_q, cu_k, block_table=table)
        low.flash_attn_varlen(qd, H.to_dev(kc, dt), H.to_dev(vc, dt), o, cq, ck, len(ql), max(ql), max(kl), hq, hkv, d,
                              1.0 / np.sqrt(d), block_tables=torch.from_numpy(table).cuda(), block_size=bs)
    else:
        k, v = H.round_to(H.normal((int(cu_k[-1]), hkv, d), 43), dt), H.round_to(H.normal((int(cu_k[-1]), hkv, d), 44), dt)
        want = ob.attn_f64_varlen(q, k, v, cu_q, cu_k)
        low.flash_attn_varlen(qd, H.to_dev(k, dt), H.to_dev(v, dt), o, cq, ck, len(ql), max(ql), max(kl), hq, hkv, d, 1.0 / np.sqrt(d))
    torch.cuda.synchronize()
    assert ffi.last_path() == "prefill_tcgen05" and ffi.last_launches() == 2 and ffi.device_status() == 0
    H.assert_bf16_close(H.to_np(o), want, "packed batch with decoding sequences")
