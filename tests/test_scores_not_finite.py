"""Scores that are NaN or infinite, on the tensor-core prefill kernel. The scalar kernel (option "force_generic") says what a row that sees such a key
outputs: NaN for a NaN or +inf score (with the log-sum-exp at -inf), and nothing of the key for a -inf score. It has to be so whichever unit takes the key's
exponential: of 16 keys in a row the last two go to the FMA pipe, the others to the special-function unit; and in a tile that the diagonal
or a padding mask cuts as in one that all rows see. Rows that don't see the key keep their bits."""
import numpy as np
import pytest
import torch

from luma_b200 import ffi, low
from oracle import binding as ob
from tests import helpers as H

pytestmark = pytest.mark.gpu
B, S, HQ, HKV = 2, 300, 4, 2


def _call(q, k, v, dt, mask, path):
    d = q.shape[-1]
    o, lse = torch.full(q.shape, 7.0, device="cuda", dtype=H.TORCH_DT[dt]), torch.full((B, HQ, S), 7.0, device="cuda")
    low.flash_attn(H.to_dev(q, dt), H.to_dev(k, dt), H.to_dev(v, dt), o, B, S, S, HQ, HKV, d, 0, 1.0 / np.sqrt(d), mask, None, lse)
    torch.cuda.synchronize()
    assert ffi.last_path() == path
    return H.to_np(o), lse.cpu().numpy()


@pytest.mark.parametrize("dt,d,padded", [("bf16", 128, False), ("f16", 64, False), ("bf16", 64, True)])
@pytest.mark.parametrize("at", [0, 13, 14, 15, 16, 127, 128, 142, 271])
@pytest.mark.parametrize("what", ["k nan", "k inf", "k -inf", "q nan"])
def test_rows_that_see_it(what, at, dt, d, padded):
    q, k, v = (H.round_to(H.normal((B, S, h, d), i), dt) for i, h in ((1, HQ), (2, HKV), (3, HKV)))
    mask = None
    if padded:
        mask = torch.ones(B, S, dtype=torch.uint8, device="cuda")
        mask[:, 5] = 0
    q[1, :, :, 3] = np.abs(q[1, :, :, 3]) + 0.125    # an infinity in K gives infinite scores of its own sign
    clean = _call(q, k, v, dt, mask, "prefill_tcgen05")
    x = {"q": q, "k": k}[what[0]]
    x[1, at, 0, 3] = {"-inf": -np.inf, "inf": np.inf, "nan": np.nan}[what.split()[1]]
    o, lse = _call(q, k, v, dt, mask, "prefill_tcgen05")
    hit = np.zeros((B, S, HQ), dtype=bool)           # rows that see the value: of one batch element, from its position on, the heads of its KV head
    if what == "q nan":
        hit[1, at, 0] = True
    else:
        hit[1, at:, :HQ // HKV] = True
    assert np.array_equal(o[~hit], clean[0][~hit]) and np.array_equal(lse.transpose(0, 2, 1)[~hit], clean[1].transpose(0, 2, 1)[~hit])
    if what == "k -inf" and at == 0:                 # row 0 sees nothing but a score of -inf; (the scalar kernel's first step is -inf minus -inf)
        assert np.isfinite(o[1, 6:]).all() and np.isfinite(lse[1, :, 6:]).all()
        return
    ffi.lib.flash_attn_set_option(b"force_generic", 1)
    try:
        want, lse_want = _call(q, k, v, dt, mask, "tile_simt")
    finally:
        ffi.lib.flash_attn_set_option(b"force_generic", 0)
    if what == "k -inf":
        assert np.isfinite(o).all()
        H.assert_bf16_close(o, want, f"{what} at {at}")
    else:
        assert np.isnan(want[hit]).all() and np.isnan(o[hit]).all()
        assert np.isfinite(o[~hit]).all()
    np.testing.assert_array_equal(np.isneginf(lse), np.isneginf(lse_want))
    np.testing.assert_allclose(lse, lse_want, rtol=0, atol=1e-3)
