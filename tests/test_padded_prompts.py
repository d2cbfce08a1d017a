"""Prompts with a key-padding mask on the tensor-core prefill kernel: K/V tiles behind the last key that counts are not walked, query tiles that sit in
padding see none (csrc/prefill_tcgen05.cu). Lengths at the edges of tiles and of the 512 keys that the search takes at a time, padding at either end, in the
middle, everywhere; query tokens behind start_pos. NaN in K of padded rows (which the mask takes out), output and log-sum-exp against the f64 oracle."""
import numpy as np
import pytest
import torch

from luma_b200 import ffi, low
from oracle import binding as ob
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hq,hkv,d,dt", [(4, 2, 128, "bf16"), (2, 2, 64, "f16"), (3, 1, 32, "bf16")])
@pytest.mark.parametrize("sq,skv,sp", [(700, 700, 0), (1300, 1300, 0), (200, 1111, 911), (129, 600, 100)])
def test_padding_anywhere(hq, hkv, d, dt, sq, skv, sp):
    lengths = [skv, skv - 1, 1, 0, 127, 128, 129, 511, 512, 513, 640]
    b = len(lengths) + 4
    mask = np.zeros((b, skv), dtype=np.uint8)
    for i, n in enumerate(lengths):
        mask[i, :n] = 1
    mask[-4, skv // 2:] = 1                       # padding in front
    mask[-3, 300] = 1                             # one key
    mask[-2] = np.arange(skv) % 200 < 60          # holes
    mask[-1, [0, skv - 1]] = 1                    # the ends
    q, k, v = (H.round_to(H.normal(s, x), dt) for s, x in (((b, sq, hq, d), 1), ((b, skv, hkv, d), 2), ((b, skv, hkv, d), 3)))
    want, lse_want = ob.attn_f64_batch(q, k, v, start_pos=sp, mask=mask, return_lse=True)
    k[mask == 0] = np.nan
    qd = H.to_dev(q, dt)
    o, lse = torch.full_like(qd, float("nan")), torch.full((b, hq, sq), float("nan"), device="cuda")
    low.flash_attn(qd, H.to_dev(k, dt), H.to_dev(v, dt), o, b, sq, skv, hq, hkv, d, sp, 1.0 / np.sqrt(d), torch.from_numpy(mask).cuda(), None, lse)
    torch.cuda.synchronize()
    assert ffi.last_path() == "prefill_tcgen05" and ffi.device_status() == 0
    H.assert_bf16_close(H.to_np(o), want, "padded")
    got, there = lse.cpu().numpy(), np.isfinite(lse_want)
    assert np.array_equal(np.isfinite(got), there) and np.abs(got[there] - lse_want[there]).max() <= 1e-3
