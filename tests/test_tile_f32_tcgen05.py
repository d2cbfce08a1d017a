"""f32 storage on the tcgen05 tensor cores (csrc/tile_f32_tcgen05.cu), against the f64 loop: rows and keys at the edges of its tiles of 128 and 64, one CTA to a
block of rows and clusters of 2, 4 and 8 that share its keys (some without a tile of their own), groups with and without a factor of two, log-sum-exp, padding
mask with NaN in the padded rows of V, packing, pages, values that do not survive the split seen by one CTA of a cluster.

Tolerance: that of test_tile_f32.py (every product to 2^-24, D/16 + 1 accumulations of a score, weights that sum to one). The relative error of a whole
result is bounded by the same terms at their average: a score of N(0,1) is off by some 2^-24 sqrt(D/16), a result by that and a dozen roundings: below 4e-7."""
import numpy as np
import pytest
import torch

from luma_b200 import ffi, low
from oracle import binding as ob
from tests import helpers as H

pytestmark = pytest.mark.gpu
TOL = 5e-5


def _close(o, want, what):
    torch.cuda.synchronize()
    assert ffi.last_path() == "tile_f32" and ffi.device_status() == 0
    got = o.cpu().numpy().astype(np.float64)
    err = np.abs(got - want)
    assert np.isfinite(got).all() and err.max() <= TOL and err.mean() <= TOL / 25, f"{what}: max {err.max()}, mean {err.mean()}"
    if want.size > 1000:
        assert np.linalg.norm(got - want) <= 4e-7 * np.linalg.norm(want), what


@pytest.mark.parametrize("b,sq,skv,hq,hkv,d,sp", [
    (1, 256, 256, 8, 8, 64, 0), (2, 257, 257, 4, 4, 32, 0), (1, 193, 193, 2, 2, 128, 0),      # clusters of 2 to 8
    (1, 5, 1025, 2, 2, 64, 1020), (1, 1, 4000, 4, 1, 128, 3999), (1, 3, 449, 1, 1, 32, 446),  # few rows over many keys
    (1, 43, 300, 9, 3, 64, 257), (1, 64, 257, 4, 2, 64, 193),                                # 129 and 128 rows
    (1, 300, 200, 4, 2, 64, 0), (1, 200, 300, 6, 2, 128, 0),                                  # more tokens than keys, and keys that nobody sees
    (3, 160, 160, 8, 8, 32, 0), (4, 96, 96, 16, 4, 32, 0), (4, 128, 128, 8, 8, 32, 0),          # both sides of the line to the warp-wide products
    (4, 400, 400, 16, 8, 64, 0), (2, 513, 513, 24, 24, 32, 0), (3, 330, 330, 12, 12, 128, 0),  # a CTA to a block
])
def test_batched_with_lse(b, sq, skv, hq, hkv, d, sp):
    q, k, v = H.normal((b, sq, hq, d), 1), H.normal((b, skv, hkv, d), 2), H.normal((b, skv, hkv, d), 3)
    want, lse_want = ob.attn_f64_batch(q, k, v, start_pos=sp, return_lse=True)
    o, lse = torch.full((b, sq, hq, d), float("nan"), device="cuda"), torch.full((b, hq, sq), float("nan"), device="cuda")
    low.flash_attn(H.to_dev(q, "f32"), H.to_dev(k, "f32"), H.to_dev(v, "f32"), o, b, sq, skv, hq, hkv, d, sp, 1.0 / np.sqrt(d), None, None, lse)
    _close(o, want, "batched")
    assert np.abs(lse.cpu().numpy() - lse_want).max() <= TOL


@pytest.mark.parametrize("b", [1, 30])
@pytest.mark.parametrize("d", [32, 64, 128])
def test_padding_mask(b, d):
    s, hq, hkv = 260, 8, 4
    q, k, v = H.normal((b, s, hq, d), 4), H.normal((b, s, hkv, d), 5), H.normal((b, s, hkv, d), 6)
    mask = np.ones((b, s), dtype=np.uint8)
    mask[0, :70] = 0
    mask[0, 130:140] = 0
    mask[b - 1, 201:] = 0
    want, lse_want = ob.attn_f64_batch(q, k, v, mask=mask, return_lse=True)
    v[mask == 0] = np.nan
    o, lse = torch.full((b, s, hq, d), float("nan"), device="cuda"), torch.full((b, hq, s), float("nan"), device="cuda")
    low.flash_attn(H.to_dev(q, "f32"), H.to_dev(k, "f32"), H.to_dev(v, "f32"), o, b, s, s, hq, hkv, d, 0, 1.0 / np.sqrt(d), torch.from_numpy(mask).cuda(), None, lse)
    _close(o, want, "padding mask")
    got, there = lse.cpu().numpy(), np.isfinite(lse_want)
    assert np.array_equal(np.isfinite(got), there) and np.abs(got[there] - lse_want[there]).max() <= TOL


@pytest.mark.parametrize("bs", [0, 5, 16])
@pytest.mark.parametrize("seqs", [1, 12])
def test_packed_and_paged(bs, seqs):
    hq, hkv, d = 12, 4, 64
    ql, kl = [33, 1, 0, 129, 65] * seqs, [200, 650, 0, 129, 3] * seqs      # the last: most of its query tokens before the first key
    cu_q, cu_k = (np.concatenate([[0], np.cumsum(x)]).astype(np.int32) for x in (ql, kl))
    q = H.normal((int(cu_q[-1]), hq, d), 7)
    qd = H.to_dev(q, "f32")
    o = torch.full_like(qd, float("nan"))
    cq, ck = torch.from_numpy(cu_q).cuda(), torch.from_numpy(cu_k).cuda()
    if bs:
        k, v, table = H.make_paged_cache(kl, bs, hkv, d, seed=8)
        want = ob.attn_f64_varlen(q, k, v, cu_q, cu_k, block_table=table)
        paged = dict(block_tables=torch.from_numpy(table).cuda(), block_size=bs)
    else:
        k, v = H.normal((int(cu_k[-1]), hkv, d), 8), H.normal((int(cu_k[-1]), hkv, d), 9)
        want = ob.attn_f64_varlen(q, k, v, cu_q, cu_k)
        paged = {}
    low.flash_attn_varlen(qd, H.to_dev(k, "f32"), H.to_dev(v, "f32"), o, cq, ck, len(ql), max(ql), max(kl), hq, hkv, d, 1.0 / np.sqrt(d), **paged)
    _close(o, want, f"packed, page {bs}")


@pytest.mark.parametrize("b", [1, 40])
@pytest.mark.parametrize("d", [32, 64, 128])
@pytest.mark.parametrize("what", ["k -inf", "k inf", "v inf", "v nan", "q nan", "v large"])
def test_values_that_do_not_split(b, d, what):
    """Infinities, NaN and values that round to a bf16 infinity: what the scalar kernel gives, row by row."""
    sq, hq, hkv, at = 300, 4, 2, 221
    q, k, v = H.normal((b, sq, hq, d), 11), H.normal((b, sq, hkv, d), 12), H.normal((b, sq, hkv, d), 13)
    x = {"q": q, "k": k, "v": v}[what[0]]
    x[0, at, 0, 3] = {"-inf": -np.inf, "inf": np.inf, "nan": np.nan, "large": 3.4e38}[what.split()[1]]
    if what == "k -inf":
        q[0, :, :, 3] = np.abs(q[0, :, :, 3]) + 0.1

    def call():
        o, lse = torch.full((b, sq, hq, d), 7.0, device="cuda"), torch.full((b, hq, sq), 7.0, device="cuda")
        low.flash_attn(H.to_dev(q, "f32"), H.to_dev(k, "f32"), H.to_dev(v, "f32"), o, b, sq, sq, hq, hkv, d, 0, 1.0 / np.sqrt(d), None, None, lse)
        torch.cuda.synchronize()
        return o.cpu().numpy(), lse.cpu().numpy(), ffi.last_path()

    o, lse, path = call()
    ffi.lib.flash_attn_set_option(b"force_generic", 1)
    try:
        want, lse_want, generic = call()
    finally:
        ffi.lib.flash_attn_set_option(b"force_generic", 0)
    assert (path, generic) == ("tile_f32", "tile_simt") and ffi.device_status() == 0
    np.testing.assert_allclose(o, want, rtol=1e-4, atol=TOL)
    np.testing.assert_allclose(lse, lse_want, rtol=1e-4, atol=TOL)
