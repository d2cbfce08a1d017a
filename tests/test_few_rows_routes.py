"""Which kernel takes calls of a few rows from more than four sequences: by estimates of both, the prefill kernel's with the heads of a group in one tile and
clusters for the keys (csrc/decode_splitk.cu). Results on both sides of the line against the f64 oracle."""
import numpy as np
import pytest
import torch

from luma_b200 import ffi, low
from oracle import binding as ob
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,s,kv,hq,hkv,d,path", [
    (16, 4, 216, 64, 8, 128, "prefill_tcgen05"), (32, 12, 133, 32, 8, 128, "prefill_tcgen05"), (12, 8, 1700, 64, 4, 128, "prefill_tcgen05"), (32, 32, 885, 8, 8, 128, "prefill_tcgen05"),
    (25, 1, 1205, 8, 2, 64, "decode_splitk"), (16, 2, 400, 8, 8, 64, "decode_splitk"), (8, 2, 1010, 32, 8, 128, "decode_splitk"), (12, 8, 1700, 16, 2, 128, "decode_splitk"),
    (4, 1, 544, 32, 8, 64, "prefill_tcgen05"),      # up to 64 pairs, counted by heads
])
def test_sides_of_the_line(b, s, kv, hq, hkv, d, path):
    dt = "bf16"
    q, k, v = (H.round_to(H.normal(x, y), dt) for x, y in (((b, s, hq, d), 1), ((b, kv, hkv, d), 2), ((b, kv, hkv, d), 3)))
    want, lse_want = ob.attn_f64_batch(q, k, v, start_pos=kv - s, return_lse=True)
    qd = H.to_dev(q, dt)
    o, lse = torch.full_like(qd, float("nan")), torch.full((b, hq, s), float("nan"), device="cuda")
    low.flash_attn(qd, H.to_dev(k, dt), H.to_dev(v, dt), o, b, s, kv, hq, hkv, d, kv - s, 1.0 / np.sqrt(d), None, None, lse)
    torch.cuda.synchronize()
    assert ffi.last_path() == path and ffi.device_status() == 0
    H.assert_bf16_close(H.to_np(o), want, path)
    assert np.abs(lse.cpu().numpy() - lse_want).max() <= 1e-3
