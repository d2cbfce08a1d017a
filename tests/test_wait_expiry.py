"""A bounded wait inside the tensor-core prefill kernel that runs out must be visible through the
ABI. The kernel cannot hang: every wait has a limit, after which the CTA records the wait's code
in a host-mapped status word, drains its copies, frees its tensor memory and returns. The launch
is asynchronous, so the call that made it has already returned OK; the NEXT entry-point call for
that device reports the failure (status 5, a message naming the wait) without launching anything,
and the call after that is clean — the error contract of luma-flash-attn/src/error.rs:38-51
(FlashAttnError::Cuda carrying the library's message).

The expiry is provoked the permitted way: the limit is shortened to about a millisecond and a test
hook makes the K producer leave out one tile, so that the issuer's wait for it runs out and the
kernel returns. Nothing traps, faults or spins without bound."""
import math
import re

import numpy as np
import pytest
import torch

from luma_b200 import error as E
from luma_b200 import ffi, low
from oracle import binding as ob
from tests import helpers as H

pytestmark = pytest.mark.gpu


def test_expired_wait_is_reported_by_the_next_call_and_then_cleared():
    b, s, hq, hkv, d = 1, 512, 4, 2, 128
    q = H.round_to(H.normal((b, s, hq, d), 1), "bf16")
    k = H.round_to(H.normal((b, s, hkv, d), 2), "bf16")
    v = H.round_to(H.normal((b, s, hkv, d), 3), "bf16")
    qd, kd, vd = (H.to_dev(x, "bf16") for x in (q, k, v))
    o = torch.empty_like(qd)
    scale = 1.0 / math.sqrt(d)
    torch.cuda.synchronize()
    assert ffi.device_status() == 0
    try:
        ffi.set_option("prefill_wait_us", 1000)
        ffi.set_option("prefill_test_skip_k", 3)          # K tile 2 is never requested
        low.flash_attn(qd, kd, vd, o, b, s, s, hq, hkv, d, 0, scale)   # returns OK: the launch is asynchronous
        assert ffi.last_path() == "prefill_tcgen05"
    finally:
        ffi.set_option("prefill_test_skip_k", 0)
        ffi.set_option("prefill_wait_us", 0)
    torch.cuda.synchronize()                               # the kernel has given up and returned by now
    with pytest.raises(E.CudaError) as exc:
        low.flash_attn(qd, kd, vd, o, b, s, s, hq, hkv, d, 0, scale)
    assert "bounded wait" in str(exc.value) and "code" in str(exc.value)
    # the word was cleared by that report: the next call runs and is right
    o.fill_(float("nan"))
    low.flash_attn(qd, kd, vd, o, b, s, s, hq, hkv, d, 0, scale)
    torch.cuda.synchronize()
    assert ffi.device_status() == 0
    H.assert_bf16_close(H.to_np(o), ob.attn_f64_batch(q, k, v), "call after the reported expiry")


@pytest.mark.parametrize("d", [128, 64])
@pytest.mark.parametrize("tile", [0, 1, 2, 5])
def test_expiry_at_every_part_of_the_key_loop(tile, d):
    # the first tile, the two that the set-up requests, one behind the rings' first round: the issuer reports nothing as done after its wait has
    # run out, so no producer takes a stage out of turn, and the kernel ends; the call after the report is right
    b, s, hq, hkv = 1, 1024, 2, 1
    q = H.round_to(H.normal((b, s, hq, d), 1), "bf16")
    k = H.round_to(H.normal((b, s, hkv, d), 2), "bf16")
    v = H.round_to(H.normal((b, s, hkv, d), 3), "bf16")
    qd, kd, vd = (H.to_dev(x, "bf16") for x in (q, k, v))
    o = torch.empty_like(qd)
    args = (qd, kd, vd, o, b, s, s, hq, hkv, d, 0, 1.0 / math.sqrt(d))
    assert ffi.device_status() == 0
    try:
        ffi.set_option("prefill_wait_us", 1000)
        ffi.set_option("prefill_test_skip_k", tile + 1)
        low.flash_attn(*args)
    finally:
        ffi.set_option("prefill_test_skip_k", 0)
        ffi.set_option("prefill_wait_us", 0)
    torch.cuda.synchronize()
    with pytest.raises(E.CudaError) as exc:
        low.flash_attn(*args)
    # the issuer's wait for the tile (K tile 0: 11, a step's tiles: 13), or one that waits on what follows from it (the next scores: 20, 21; a
    # free stage: 1, 2); never one that the issuer came to after it had given up (P: 14 to 17)
    assert int(re.search(r"code (-?\d+)", str(exc.value)).group(1)) in ({11, 20, 21, 1, 2} if tile == 0 else {13, 20, 21, 1, 2})
    low.flash_attn(*args)
    torch.cuda.synchronize()
    assert ffi.device_status() == 0
    H.assert_bf16_close(H.to_np(o), ob.attn_f64_batch(q, k, v), "call after the reported expiry")


@pytest.mark.parametrize("d", [128, 64])
@pytest.mark.parametrize("how", ["packed", "packed, rows unknown", "packed over pages", "chunks over pages"])
@pytest.mark.parametrize("tile", [0, 3, 6])
def test_expiry_in_a_tile_pair_that_a_cta_has_taken_over(tile, how, d):
    # pairs of one to three tiles, some twenty for every SM, before a few of eight that alone have tiles 3 and 6. The call ends soon after the limit: what the producers wait for
    # at their end has arrived by then, and their last waits would otherwise run 100 ms
    hq, hkv, page, dt = 16, 8, 16, torch.bfloat16
    rng = np.random.Generator(np.random.Philox(d + tile))
    lens = (128 * rng.integers(1, 4, size=400) - 50 * rng.integers(0, 2, size=400)).tolist() + [1024] * 6
    new = [128 if how == "chunks over pages" else min(x, 128) for x in lens]
    lens = [max(x, n) for x, n in zip(lens, new)]
    g = torch.Generator(device="cuda").manual_seed(tile)
    cu_q, cu_k = (torch.tensor(np.concatenate([[0], np.cumsum(x)]), dtype=torch.int32, device="cuda") for x in (new, lens))
    n, q = len(lens), torch.randn((sum(new), hq, d), generator=g, device="cuda", dtype=dt)
    o, scale = torch.empty_like(q), 1.0 / math.sqrt(d)
    if how.startswith("packed,") or how == "packed":
        k, v = (torch.randn((sum(lens), hkv, d), generator=g, device="cuda", dtype=dt) for _ in range(2))
        totals = dict(total_q=sum(new), total_k=sum(lens)) if how == "packed" else {}
        call = lambda: low.flash_attn_varlen(q, k, v, o, cu_q, cu_k, n, max(new), max(lens), hq, hkv, d, scale, **totals)
    else:
        width = -(-max(lens) // page)
        k, v = (torch.randn((n * width, page, hkv, d), generator=g, device="cuda", dtype=dt) for _ in range(2))
        table = torch.randperm(n * width, generator=g, device="cuda").to(torch.int32).view(n, width)
        if how == "packed over pages":
            call = lambda: low.flash_attn_varlen(q, k, v, o, cu_q, cu_k, n, max(new), max(lens), hq, hkv, d, scale, table, page, total_q=sum(new))
        else:
            ctx = torch.tensor(lens, dtype=torch.int32, device="cuda")
            call = lambda: low.flash_attn_with_kvcache(q, k, v, o, table, ctx, n, 128, hq, hkv, d, page, width, scale)
    call()
    torch.cuda.synchronize()
    assert ffi.last_path() == "prefill_tcgen05" and ffi.device_status() == 0
    want = o.clone()
    begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    try:
        ffi.set_option("prefill_wait_us", 1000)
        ffi.set_option("prefill_test_skip_k", tile + 1)
        begin.record()
        call()
        end.record()
    finally:
        ffi.set_option("prefill_test_skip_k", 0)
        ffi.set_option("prefill_wait_us", 0)
    torch.cuda.synchronize()
    code = ffi.device_status()                       # (read and cleared)
    assert code != 0
    # 1 ms from the tile that does not come, and so for every CTA that starts after one has given up: all pairs have a tile 0, 22 to an SM
    assert begin.elapsed_time(end) < (100 if tile == 0 else 30)
    o.fill_(float("nan"))
    call()
    torch.cuda.synchronize()
    assert ffi.device_status() == 0 and torch.equal(o, want)


def test_a_bound_above_two_seconds_is_kept():
    # the bound is counted in clocks, two to the nanosecond, so that it is no shorter than asked for at any SM clock up to 2 GHz
    b, s, h, d = 1, 256, 1, 128
    q = H.to_dev(H.normal((b, s, h, d), 1), "bf16")
    o = torch.empty_like(q)
    args = (q, q, q, o, b, s, s, h, h, d, 0, 1.0 / math.sqrt(d))
    torch.cuda.synchronize()
    begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    try:
        ffi.set_option("prefill_wait_us", 2300000)
        ffi.set_option("prefill_test_skip_k", 1)
        begin.record()
        low.flash_attn(*args)
        end.record()
    finally:
        ffi.set_option("prefill_test_skip_k", 0)
        ffi.set_option("prefill_wait_us", 0)
    torch.cuda.synchronize()
    assert ffi.device_status() != 0                  # (read and cleared)
    assert begin.elapsed_time(end) >= 2300


def test_workspaces_are_bounded_and_releasable():
    # the decode path keeps one split-K workspace per (device, stream), at most 32, and gives them back on request
    hq, hkv, d, bs = 8, 2, 128, 16
    lens = [300, 40]
    kc, vc, table = H.make_paged_cache(lens, bs, hkv, d, seed=5)
    q = H.round_to(H.normal((2, 1, hq, d), 6), "bf16")
    want = ob.attn_f64_kvcache(q, H.round_to(kc, "bf16"), H.round_to(vc, "bf16"), lens, table)
    qd, kd, vd = H.to_dev(q, "bf16"), H.to_dev(kc, "bf16"), H.to_dev(vc, "bf16")
    td, ld = torch.from_numpy(table).cuda(), torch.tensor(lens, dtype=torch.int32, device="cuda")
    ffi.lib.flash_attn_release_workspaces()
    streams = [torch.cuda.Stream() for _ in range(40)]
    torch.cuda.synchronize()
    outs = []
    for st in streams:
        o = torch.full_like(qd, float("nan"))
        with torch.cuda.stream(st):
            low.flash_attn_with_kvcache(qd, kd, vd, o, td, ld, 2, 1, hq, hkv, d, bs, table.shape[1], 1.0 / math.sqrt(d), st)
        outs.append(o)
    torch.cuda.synchronize()
    for o in outs:
        H.assert_bf16_close(H.to_np(o), want, "decode on one of many streams")
    held = ffi.lib.flash_attn_release_workspaces()
    assert 1 <= held <= 32
    assert ffi.lib.flash_attn_release_workspaces() == 0
