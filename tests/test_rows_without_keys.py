"""Query rows that sit before the first key (a sequence with more query tokens than keys, or with no key at all) output exact zeros
(luma-flash-attn/kernels/flash_attn_with_kvcache.cu:185-195,270-275). A 128-row tile of nothing but such rows needs no Q: the tensor-core kernel asks for
none, so that no copy of Q is on its way into the shared memory where the tile's zeros are staged. Many sequences and several runs, Q from
HBM and not from L2 in each; the last sequence's tiles at the end of the packed buffer are those that a warp copies with plain loads."""
import numpy as np
import pytest
import torch

from luma_b200 import ffi, low
from oracle import binding as ob
from tests import helpers as H

pytestmark = pytest.mark.gpu


def _runs(call, o, flush, n=5):
    for _ in range(n):
        o.fill_(float("nan"))
        flush.zero_()   # larger than L2
        call()
        torch.cuda.synchronize()
        assert ffi.last_path() == "prefill_tcgen05" and ffi.device_status() == 0
        yield H.to_np(o)


@pytest.fixture(scope="module")
def flush():
    return torch.empty(192 << 20, dtype=torch.uint8, device="cuda")


@pytest.mark.parametrize("d", [128, 64])
@pytest.mark.parametrize("totals", [False, True])
@pytest.mark.parametrize("hq,hkv", [(8, 2), (4, 4)])
def test_packed(hq, hkv, totals, d, flush):
    ql = [256, 300, 128, 140, 512, 384] * 8 + [300]
    kl = [0, 20, 0, 3, 200, 129] * 8 + [5]
    cu_q, cu_k = (np.concatenate([[0], np.cumsum(x)]).astype(np.int32) for x in (ql, kl))
    q = H.round_to(H.normal((int(cu_q[-1]), hq, d), 1), "bf16")
    k = H.round_to(H.normal((int(cu_k[-1]), hkv, d), 2), "bf16")
    v = H.round_to(H.normal((int(cu_k[-1]), hkv, d), 3), "bf16")
    want = ob.attn_f64_varlen(q, k, v, cu_q, cu_k)
    qd, kd, vd = (H.to_dev(x, "bf16") for x in (q, k, v))
    cq, ck = torch.from_numpy(cu_q).cuda(), torch.from_numpy(cu_k).cuda()
    o = torch.empty_like(qd)
    kw = dict(total_q=int(cu_q[-1]), total_k=int(cu_k[-1])) if totals else {}
    blind = np.concatenate([np.arange(n) < n - m for n, m in zip(ql, kl)])
    for got in _runs(lambda: low.flash_attn_varlen(qd, kd, vd, o, cq, ck, len(ql), max(ql), max(kl), hq, hkv, d, 1.0 / np.sqrt(d), **kw), o, flush):
        assert np.all(got[blind] == 0.0)
        H.assert_bf16_close(got, want, "rows before the first key, packed")


@pytest.mark.parametrize("d", [128, 64])
def test_paged(d, flush):
    hq, hkv, sq, page = 8, 2, 384, 16
    lens = [0, 5, 129, 384, 256, 0, 300, 1000] * 6
    kc, vc, table = H.make_paged_cache(lens, page, hkv, d, seed=7)
    kc, vc = H.round_to(kc, "bf16"), H.round_to(vc, "bf16")
    q = H.round_to(H.normal((len(lens), sq, hq, d), 8), "bf16")
    want = ob.attn_f64_kvcache(q, kc, vc, lens, table)
    qd, kd, vd = (H.to_dev(x, "bf16") for x in (q, kc, vc))
    td, ld = torch.from_numpy(table).cuda(), torch.tensor(lens, dtype=torch.int32, device="cuda")
    o = torch.empty_like(qd)
    blind = np.arange(sq)[None, :] < sq - np.array(lens)[:, None]
    for got in _runs(lambda: low.flash_attn_with_kvcache(qd, kd, vd, o, td, ld, len(lens), sq, hq, hkv, d, page, table.shape[1], 1.0 / np.sqrt(d)), o, flush):
        assert np.all(got[blind] == 0.0)
        H.assert_bf16_close(got, want, "rows before the first key, paged")
