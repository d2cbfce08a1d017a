"""f32 storage on the tensor cores with split operands (csrc/tile_f32.cu), against the f64 loop, at the edges of its
16/32/64-row tiles and 32/64-key tiles, in the form for small problems (warps share the keys) and for large ones, with
padding mask (NaN in the padded rows of V), log-sum-exp, packing, pages and query tokens that see no key.

Tolerance: every product of two f32 values is formed to 2^-24 or better; a score of at most |s| <= 8 here passes D/16 + 1
accumulations of at most 2^-23 |s| each, D = 128: 9e-6, which is the relative error of its weight; weights sum to
one over values of at most 5, and a dozen tiles add 2^-24 each. 1e-5 * 5 bounds the sum; N(0,1) inputs average far below."""
import numpy as np
import pytest
import torch

from luma_b200 import ffi, low
from oracle import binding as ob
from tests import helpers as H

pytestmark = pytest.mark.gpu
TOL = 5e-5


def _close(got, want, what):
    err = np.abs(np.asarray(got, dtype=np.float64) - want)
    assert np.isfinite(got).all() and err.max() <= TOL and err.mean() <= TOL / 25, f"{what}: max {err.max()}, mean {err.mean()}"


@pytest.mark.parametrize("b,sq,skv,hq,hkv,d,sp", [
    (1, 1, 1, 1, 1, 32, 0), (1, 15, 33, 2, 2, 64, 18), (2, 17, 65, 6, 2, 128, 48), (1, 64, 64, 8, 8, 64, 0),
    (3, 129, 129, 4, 1, 128, 0), (1, 100, 40, 2, 1, 64, 0),                   # later tokens see all of a shorter K/V
    (2, 600, 600, 32, 16, 64, 0), (1, 650, 650, 32, 32, 128, 0), (4, 333, 400, 30, 15, 32, 67),   # a warp per 16 rows
])
def test_batched(b, sq, skv, hq, hkv, d, sp):
    q, k, v = H.normal((b, sq, hq, d), 1), H.normal((b, skv, hkv, d), 2), H.normal((b, skv, hkv, d), 3)
    want, lse_want = ob.attn_f64_batch(q, k, v, start_pos=sp, return_lse=True)
    o = torch.full((b, sq, hq, d), float("nan"), device="cuda")
    lse = torch.full((b, hq, sq), float("nan"), device="cuda")
    low.flash_attn(H.to_dev(q, "f32"), H.to_dev(k, "f32"), H.to_dev(v, "f32"), o, b, sq, skv, hq, hkv, d, sp, 1.0 / np.sqrt(d), None, None, lse)
    torch.cuda.synchronize()
    assert ffi.last_path() == "tile_f32"
    _close(o.cpu().numpy(), want, "batched")
    assert np.abs(lse.cpu().numpy() - lse_want).max() <= TOL


@pytest.mark.parametrize("d", [32, 64, 128])
def test_padding_mask(d):
    b, s, hq, hkv = 3, 150, 4, 2
    q, k, v = H.normal((b, s, hq, d), 4), H.normal((b, s, hkv, d), 5), H.normal((b, s, hkv, d), 6)
    mask = np.ones((b, s), dtype=np.uint8)
    mask[0, 90:] = 0
    mask[1, :40] = 0
    mask[2, 60:70] = 0
    want = ob.attn_f64_batch(q, k, v, mask=mask)
    v[mask == 0] = np.nan
    o = torch.full((b, s, hq, d), float("nan"), device="cuda")
    low.flash_attn(H.to_dev(q, "f32"), H.to_dev(k, "f32"), H.to_dev(v, "f32"), o, b, s, s, hq, hkv, d, 0, 1.0 / np.sqrt(d),
                   torch.from_numpy(mask).cuda())
    torch.cuda.synchronize()
    assert ffi.last_path() == "tile_f32"
    _close(o.cpu().numpy(), want, "padding mask")


@pytest.mark.parametrize("bs", [0, 5, 16])
def test_packed_and_chunked(bs):
    hq, hkv, d = 4, 2, 64
    ql, kl = [33, 1, 70, 5], [33, 65, 200, 3]          # the last: two query tokens before the first key
    cu_q, cu_k = (np.concatenate([[0], np.cumsum(x)]).astype(np.int32) for x in (ql, kl))
    q = H.normal((int(cu_q[-1]), hq, d), 7)
    o = torch.full((int(cu_q[-1]), hq, d), float("nan"), device="cuda")
    cq, ck = torch.from_numpy(cu_q).cuda(), torch.from_numpy(cu_k).cuda()
    if bs:
        kc, vc, table = H.make_paged_cache(kl, bs, hkv, d, seed=8)
        want = ob.attn_f64_varlen(q, kc, vc, cu_q, cu_k, block_table=table)
        low.flash_attn_varlen(H.to_dev(q, "f32"), H.to_dev(kc, "f32"), H.to_dev(vc, "f32"), o, cq, ck, 4, 70, 200, hq, hkv, d,
                              1.0 / np.sqrt(d), block_tables=torch.from_numpy(table).cuda(), block_size=bs)
    else:
        k, v = H.normal((int(cu_k[-1]), hkv, d), 8), H.normal((int(cu_k[-1]), hkv, d), 9)
        want = ob.attn_f64_varlen(q, k, v, cu_q, cu_k)
        low.flash_attn_varlen(H.to_dev(q, "f32"), H.to_dev(k, "f32"), H.to_dev(v, "f32"), o, cq, ck, 4, 70, 200, hq, hkv, d, 1.0 / np.sqrt(d))
    torch.cuda.synchronize()
    assert ffi.last_path() == "tile_f32"
    _close(o.cpu().numpy(), want, f"packed, page {bs}")


@pytest.mark.parametrize("d,sq", [(32, 40), (64, 70), (128, 33)])
@pytest.mark.parametrize("what", ["k -inf", "k inf", "v inf", "v nan", "q nan", "k large", "v large"])
def test_values_that_do_not_split(d, sq, what):
    """Infinities, NaN and values that round to a bf16 infinity: what the scalar kernel gives, row by row (a row that does
    not see the value is not touched by it)."""
    b, hq, hkv, at = 2, 4, 2, 21
    q, k, v = H.normal((b, sq, hq, d), 11), H.normal((b, sq, hkv, d), 12), H.normal((b, sq, hkv, d), 13)
    x = {"q": q, "k": k, "v": v}[what[0]]
    x[1, at, 0, 3] = {"-inf": -np.inf, "inf": np.inf, "nan": np.nan, "large": 3.4e38}[what.split()[1]]
    if what == "k -inf":
        q[1, :, :, 3] = np.abs(q[1, :, :, 3]) + 0.1      # the scores are -inf: the key has no weight

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
    assert (path, generic) == ("tile_f32", "tile_simt")
    np.testing.assert_allclose(o, want, rtol=1e-4, atol=TOL)          # NaN and infinities in the same places
    np.testing.assert_allclose(lse, lse_want, rtol=1e-4, atol=TOL)
    assert np.isfinite(o[1, :at]).all() and np.isfinite(o[0]).all()
