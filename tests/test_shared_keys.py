"""Tile pairs whose keys a cluster of CTAs shares (csrc/prefill_tcgen05.cu): clusters of 2, 4 and 8, sequences shorter than a share next to long ones (CTAs without a tile), tiles without a
partner, rows that end inside a share, query tokens before the first key, padding mask, packed buffers with and without their row counts, pages, scores that are NaN or
infinite, and a wait that runs out in the middle. Against the f64 oracle, and the same bits on repetition and in every launch order."""
import math

import numpy as np
import pytest
import torch

from luma_b200 import error as E
from luma_b200 import ffi, low
from oracle import binding as ob
from tests import helpers as H

pytestmark = pytest.mark.gpu


def _twice(call, want, what):
    first = None
    for _ in range(2):
        o = call()
        torch.cuda.synchronize()
        assert ffi.last_path() == "prefill_tcgen05" and ffi.device_status() == 0
        H.assert_bf16_close(H.to_np(o), want, what)
        assert first is None or torch.equal(first, o)
        first = o
    return first


@pytest.mark.parametrize("d,dt", [(128, "bf16"), (64, "f16"), (32, "bf16")])
@pytest.mark.parametrize("b,sq,skv,hq,hkv,sp,masked", [
    (1, 70, 4500, 2, 1, 4430, False),      # 8 CTAs to a pair
    (3, 129, 2100, 4, 4, 1971, False),     # 4; a pair with one row in its second tile
    (2, 1700, 1700, 6, 2, 0, False),       # 2; early rows see few of the shares
    (1, 300, 1800, 3, 3, 0, False),        # keys that nobody sees
    (2, 200, 2000, 4, 2, 1800, True), (4, 1, 1100, 8, 2, 1099, True), (3, 4, 1000, 4, 1, 996, True),
])
def test_batched(b, sq, skv, hq, hkv, sp, masked, d, dt):
    q, k, v = (H.round_to(H.normal(s, x), dt) for s, x in (((b, sq, hq, d), 1), ((b, skv, hkv, d), 2), ((b, skv, hkv, d), 3)))
    mask = None
    if masked:
        mask = np.ones((b, skv), dtype=np.uint8)
        mask[0, :700] = 0
        mask[-1, skv - 130:] = 0
    want, lse_want = ob.attn_f64_batch(q, k, v, start_pos=sp, mask=mask, return_lse=True)
    dev = [H.to_dev(x, dt) for x in (q, k, v)]
    lse = torch.empty((b, hq, sq), device="cuda")

    def call():
        o = torch.full_like(dev[0], float("nan"))
        lse.fill_(float("nan"))
        low.flash_attn(*dev, o, b, sq, skv, hq, hkv, d, sp, 1.0 / math.sqrt(d), None if mask is None else torch.from_numpy(mask).cuda(), None, lse)
        return o
    _twice(call, want, f"{b} x {sq} over {skv}")
    got, there = lse.cpu().numpy(), np.isfinite(lse_want)
    assert np.array_equal(np.isfinite(got), there) and np.abs(got[there] - lse_want[there]).max() <= 1e-3


@pytest.mark.parametrize("d", [128, 64])
@pytest.mark.parametrize("sq,hq,hkv,page,lens", [
    (100, 4, 1, 16, [4200, 100, 130]), (130, 3, 1, 32, [1800, 0, 131, 40]), (65, 16, 2, 128, [2900, 600]), (70, 8, 8, 8, [1700, 70, 1000]),
])
def test_chunks_over_pages(sq, hq, hkv, page, lens, d):
    dt = "bf16"
    kc, vc, table = H.make_paged_cache(lens, page, hkv, d, seed=sq)
    kc, vc, q = H.round_to(kc, dt), H.round_to(vc, dt), H.round_to(H.normal((len(lens), sq, hq, d), 4), dt)
    want = ob.attn_f64_kvcache(q, kc, vc, lens, table)
    dev = [H.to_dev(x, dt) for x in (q, kc, vc)]
    tab, cl = torch.from_numpy(table).cuda(), torch.tensor(lens, dtype=torch.int32, device="cuda")

    def call():
        o = torch.full_like(dev[0], float("nan"))
        low.flash_attn_with_kvcache(*dev, o, tab, cl, len(lens), sq, hq, hkv, d, page, table.shape[1], 1.0 / math.sqrt(d))
        return o
    o = _twice(call, want, f"{sq} over {lens}")
    for name, value in ((b"prefill_order", 2), (b"prefill_band", 1)):
        ffi.lib.flash_attn_set_option(name, value)
        try:
            assert torch.equal(call(), o)
        finally:
            ffi.lib.flash_attn_set_option(name, 0)


@pytest.mark.parametrize("paged", [False, True])
@pytest.mark.parametrize("total", [False, True])
def test_packed(paged, total):
    dt, d, page, hq, hkv = "f16", 128, 16, 4, 2
    ql, kl = [200, 17, 0, 129, 64], [1900, 17, 0, 2500, 300]
    cu_q, cu_k = (np.concatenate([[0], np.cumsum(x)]).astype(np.int32) for x in (ql, kl))
    q = H.round_to(H.normal((sum(ql), hq, d), 5), dt)
    if paged:
        k, v, table = H.make_paged_cache(kl, page, hkv, d, seed=6)
        k, v = H.round_to(k, dt), H.round_to(v, dt)
        want = ob.attn_f64_varlen(q, k, v, cu_q, cu_k, block_table=table)
    else:
        k, v = (H.round_to(H.normal((sum(kl), hkv, d), x), dt) for x in (6, 7))
        want = ob.attn_f64_varlen(q, k, v, cu_q, cu_k)
    dev, cq, ck = [H.to_dev(x, dt) for x in (q, k, v)], torch.from_numpy(cu_q).cuda(), torch.from_numpy(cu_k).cuda()

    def call():
        o = torch.full_like(dev[0], float("nan"))
        low.flash_attn_varlen(*dev, o, cq, ck, len(ql), max(ql), max(kl), hq, hkv, d, 1.0 / math.sqrt(d), torch.from_numpy(table).cuda() if paged else None, page if paged else 1,
                              total_q=sum(ql) if total else None, total_k=sum(kl) if total and not paged else None)
        return o
    _twice(call, want, "packed")


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_scores_that_are_not_finite(value):
    # a key with such a score makes the rows that see it NaN, whichever share it is in, and leaves the others alone
    b, sq, skv, hq, hkv, d = 1, 260, 2000, 2, 2, 128
    g = torch.Generator(device="cuda").manual_seed(3)
    q, k, v = (torch.randn((b, s, h, d), generator=g, device="cuda").bfloat16() for s, h in ((sq, hq), (skv, hkv), (skv, hkv)))
    q[..., 5] = q[..., 5].abs() + 0.5

    def call():
        o, lse = torch.empty_like(q), torch.empty((b, hq, sq), device="cuda")
        low.flash_attn(q, k, v, o, b, sq, skv, hq, hkv, d, skv - sq, 1.0 / math.sqrt(d), None, None, lse)
        torch.cuda.synchronize()
        assert ffi.last_path() == "prefill_tcgen05" and ffi.device_status() == 0
        return o, lse
    clean, clean_lse = call()
    at = skv - sq + 100
    k[0, at, 1, 5] = value
    o, lse = call()
    hit = torch.zeros((b, sq, hq), dtype=torch.bool, device="cuda")
    hit[0, 100:, 1] = True
    assert torch.isnan(o[hit].float()).all() and torch.equal(o[~hit], clean[~hit])
    assert torch.isneginf(lse.transpose(1, 2)[hit]).all() and torch.equal(lse.transpose(1, 2)[~hit], clean_lse.transpose(1, 2)[~hit])


@pytest.mark.parametrize("d", [128, 64])
@pytest.mark.parametrize("tile", [0, 1, 3])
def test_a_wait_that_runs_out(tile, d):
    # a K tile of every share is never requested: all CTAs of the cluster end, the next call reports it and the one after is right
    b, sq, skv, h = 1, 200, 4500, 1
    g = torch.Generator(device="cuda").manual_seed(d)
    q, k, v = (torch.randn((b, s, h, d), generator=g, device="cuda").bfloat16() for s in (sq, skv, skv))
    o = torch.empty_like(q)
    call = lambda: low.flash_attn(q, k, v, o, b, sq, skv, h, h, d, skv - sq, 1.0 / math.sqrt(d))
    call()
    torch.cuda.synchronize()
    want = o.clone()
    try:
        ffi.set_option("prefill_wait_us", 1000)
        ffi.set_option("prefill_test_skip_k", tile + 1)
        call()
    finally:
        ffi.set_option("prefill_test_skip_k", 0)
        ffi.set_option("prefill_wait_us", 0)
    torch.cuda.synchronize()
    with pytest.raises(E.CudaError, match="bounded wait"):
        call()
    call()
    torch.cuda.synchronize()
    assert ffi.device_status() == 0 and torch.equal(o, want)
