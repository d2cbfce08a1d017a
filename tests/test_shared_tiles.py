"""Query heads of a GQA group that share the tiles of the tensor-core prefill kernel (csrc/prefill_tcgen05.cu): rows of a tile are query token x head. Groups
that are a power of two up to the 32 rows of a warp and beyond, that have a factor of two, and that have none; sequences that end inside a token's last
tile, on its edge and one token past it, whose last warps have no rows; through every entry point, against the f64 oracle with the tolerance of the 16-bit kernels."""
import numpy as np
import pytest
import torch

from luma_b200 import ffi, low
from oracle import binding as ob
from tests import helpers as H

pytestmark = pytest.mark.gpu

GROUPS = [(4, 2), (3, 1), (8, 2), (12, 2), (12, 1), (16, 1), (32, 1), (64, 1)]   # pack 2, 1, 4, 2, 4, 16, 32, 32


def _done(o, want, what):
    torch.cuda.synchronize()
    assert ffi.last_path() == "prefill_tcgen05" and ffi.device_status() == 0
    H.assert_bf16_close(H.to_np(o), want, what)


@pytest.mark.parametrize("hq,hkv", GROUPS)
@pytest.mark.parametrize("s,d,dt", [(65, 128, "bf16"), (129, 64, "f16"), (160, 128, "bf16"), (71, 32, "bf16")])
def test_batched_with_lse_and_mask(hq, hkv, s, d, dt):
    b = 2
    q, k, v = (H.round_to(H.normal((b, s, h, d), 3 + h + s), dt) for h in (hq, hkv, hkv))
    dev = [H.to_dev(x, dt) for x in (q, k, v)]
    mask = np.ones((b, s), dtype=np.uint8)
    mask[0, s - 33:] = 0
    for m in (None, mask):
        want, lse_want = ob.attn_f64_batch(q, k, v, mask=m, return_lse=True)
        o, lse = torch.full_like(dev[0], float("nan")), torch.full((b, hq, s), float("nan"), device="cuda")
        low.flash_attn(*dev, o, b, s, s, hq, hkv, d, 0, 1.0 / np.sqrt(d), None if m is None else torch.from_numpy(m).cuda(), None, lse)
        _done(o, want, f"{hq}/{hkv}")
        got, there = lse.cpu().numpy(), np.isfinite(lse_want)
        assert np.array_equal(np.isfinite(got), there) and np.abs(got[there] - lse_want[there]).max() <= 1e-3


@pytest.mark.parametrize("hq,hkv", GROUPS)
@pytest.mark.parametrize("paged", [False, True])
@pytest.mark.parametrize("total", [True, False])
def test_packed(hq, hkv, paged, total):
    dt, d, page = "bf16", 128, 16
    ql, kl = [33, 64, 0, 65, 127, 32, 5], [33, 190, 0, 300, 127, 32, 129]
    cu_q, cu_k = (np.concatenate([[0], np.cumsum(x)]).astype(np.int32) for x in (ql, kl))
    q = H.round_to(H.normal((sum(ql), hq, d), 7), dt)
    if paged:
        k, v, table = H.make_paged_cache(kl, page, hkv, d, seed=8)
        k, v = H.round_to(k, dt), H.round_to(v, dt)
        want = ob.attn_f64_varlen(q, k, v, cu_q, cu_k, block_table=table)
    else:
        k, v = (H.round_to(H.normal((sum(kl), hkv, d), x), dt) for x in (8, 9))
        want = ob.attn_f64_varlen(q, k, v, cu_q, cu_k)
    qd = H.to_dev(q, dt)
    o = torch.full_like(qd, float("nan"))
    low.flash_attn_varlen(qd, H.to_dev(k, dt), H.to_dev(v, dt), o, torch.from_numpy(cu_q).cuda(), torch.from_numpy(cu_k).cuda(), len(ql), max(ql), max(kl), hq, hkv, d,
                          1.0 / np.sqrt(d), torch.from_numpy(table).cuda() if paged else None, page if paged else 1,
                          total_q=sum(ql) if total else None, total_k=sum(kl) if total and not paged else None)
    _done(o, want, f"{hq}/{hkv}")


@pytest.mark.parametrize("hq,hkv", GROUPS)
@pytest.mark.parametrize("order", [0, 2])
def test_chunks_over_pages(hq, hkv, order):
    dt, d, page, sq, lens = "f16", 64, 16, 66, [66, 700, 67, 0, 40, 1025]
    kc, vc, table = H.make_paged_cache(lens, page, hkv, d, seed=5)
    kc, vc = H.round_to(kc, dt), H.round_to(vc, dt)
    q = H.round_to(H.normal((len(lens), sq, hq, d), 6), dt)
    want = ob.attn_f64_kvcache(q, kc, vc, lens, table)
    o = torch.full((len(lens), sq, hq, d), float("nan"), device="cuda", dtype=H.TORCH_DT[dt])
    ffi.set_option("prefill_order", order)
    try:
        low.flash_attn_with_kvcache(H.to_dev(q, dt), H.to_dev(kc, dt), H.to_dev(vc, dt), o, torch.from_numpy(table).cuda(),
                                    torch.tensor(lens, dtype=torch.int32, device="cuda"), len(lens), sq, hq, hkv, d, page, table.shape[1], 1.0 / np.sqrt(d))
    finally:
        ffi.set_option("prefill_order", 0)
    _done(o, want, f"{hq}/{hkv}")
