"""Chunks of prompts over contexts of different lengths: the tensor-core prefill kernel finds each CTA's tile pair on the
device, heaviest first (find_item in csrc/prefill_tcgen05.cu). Every row has to be computed exactly once whatever the
lengths are: outputs are compared with the f64 loop (16-bit tolerance) and, bit by bit, with the grid-order launch of the
same kernel (option "prefill_band" = 1). Sizes: one row block and one row more, odd group sizes (an unpaired tile), empty
and short sequences, more sequences than lanes (33) and than a warp holds (257: grid order), weights of 1 to 18 tiles (class edges)."""
import numpy as np
import pytest
import torch

from luma_b200 import ffi, high, low
from oracle import binding as ob
from tests import helpers as H

pytestmark = pytest.mark.gpu


def grid_order(call):
    ffi.lib.flash_attn_set_option(b"prefill_band", 1)
    try:
        return call()
    finally:
        ffi.lib.flash_attn_set_option(b"prefill_band", 0)


@pytest.mark.parametrize("sq,hq,hkv,d,page,lens,dt", [
    (128, 8, 2, 128, 16, [1700, 128, 2300, 129, 400], "bf16"),
    (129, 3, 3, 64, 32, [2200, 129, 0, 1025, 130, 100, 1024], "f16"),
    (200, 6, 2, 32, 8, [1281, 200, 640, 1280], "bf16"),
    (72, 2, 2, 64, 16, [72 + 37 * (i % 30) for i in range(33)], "bf16"),
    (65, 1, 1, 64, 128, [65 + (i * 53) % 200 for i in range(257)], "f16"),
])
def test_chunks_over_different_contexts(sq, hq, hkv, d, page, lens, dt):
    kc, vc, table = H.make_paged_cache(lens, page, hkv, d, seed=sq + d)
    kc, vc = H.round_to(kc, dt), H.round_to(vc, dt)
    q = H.round_to(H.normal((len(lens), sq, hq, d), 51), dt)
    want = ob.attn_f64_kvcache(q, kc, vc, lens, table)
    dev = (H.to_dev(q, dt), H.to_dev(kc, dt), H.to_dev(vc, dt))
    tab, cl = torch.from_numpy(table).cuda(), torch.tensor(lens, dtype=torch.int32, device="cuda")

    def call():
        o = torch.full((len(lens), sq, hq, d), float("nan"), device="cuda", dtype=H.TORCH_DT[dt])
        low.flash_attn_with_kvcache(dev[0], dev[1], dev[2], o, tab, cl, len(lens), sq, hq, hkv, d, page, table.shape[1], 1.0 / np.sqrt(d))
        torch.cuda.synchronize()
        assert ffi.last_path() == "prefill_tcgen05"
        return o

    o = call()
    H.assert_bf16_close(H.to_np(o), want, f"{sq} tokens over {lens[:5]}")
    assert torch.equal(o, grid_order(call))


@pytest.mark.parametrize("q_lens,k_lens,hq,hkv,d", [
    ([256, 1, 130, 1, 3, 200], [2048, 1900, 130, 64, 700, 1500], 8, 2, 128),      # chunks next to decoding sequences, which go behind
    ([1, 1, 300], [1300, 17, 300], 4, 4, 64),
    ([100, 0, 128, 7], [2000, 0, 128, 1200], 2, 1, 64),
])
def test_packed_chunks_over_pages(q_lens, k_lens, hq, hkv, d):
    dt, page = "bf16", 16
    kc, vc, table = H.make_paged_cache(k_lens, page, hkv, d, seed=9)
    kc, vc = H.round_to(kc, dt), H.round_to(vc, dt)
    cu_q, cu_k = (np.concatenate([[0], np.cumsum(x)]).astype(np.int32) for x in (q_lens, k_lens))
    q = H.round_to(H.normal((int(cu_q[-1]), hq, d), 61), dt)
    dev = (H.to_dev(q, dt), H.to_dev(kc, dt), H.to_dev(vc, dt))
    cq, ck, tab = (torch.from_numpy(x).cuda() for x in (cu_q, cu_k, table))

    def call():
        o = high.flash_attn_varlen_func(*dev, cq, ck, max(q_lens), max(k_lens), block_table=tab)
        torch.cuda.synchronize()
        return o

    o = call()
    assert torch.equal(o, call()) and torch.equal(o, grid_order(call))
    for s, (a, b) in enumerate(zip(cu_q[:-1], cu_q[1:])):
        if a == b:
            continue
        want = ob.attn_f64_kvcache(q[None, a:b], kc, vc, [k_lens[s]], table[s:s + 1])
        H.assert_bf16_close(H.to_np(o[a:b])[None], want, f"sequence {s}")
