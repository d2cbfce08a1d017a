"""The two units that take the prefill kernel's exponentials, seen through the log-sum-exp. Scores are exact here (one nonzero product each),
so that LSE = ln(1 + 2^-x), x < 1, shows the errors of the second key's 2^-x and of the first one's 2^0 alone. The bound is the one that CUDA documents for
ex2.approx whichever unit takes them, in tiles that the diagonal cuts and in others: 2^-22 relative, 2.4e-7 in the logarithm. To it come the
rounding of the argument (half an ulp below 1, times ln 2: 2.1e-8) and of the scale in log2 units (7.3e-8 of x, times ln 2, at half the weight: 2.5e-8), of
the sum (half an ulp above 1: 6e-8), of log2f (an ulp below 1, times ln 2: 4.1e-8) and of the product with ln 2 (3e-8): 4.2e-7."""
import numpy as np
import pytest
import torch

from luma_b200 import ffi, low
from tests import helpers as H

pytestmark = pytest.mark.gpu
BOUND = 4.2e-7


@pytest.mark.parametrize("dt,d", [("bf16", 128), ("f16", 64)])
@pytest.mark.parametrize("start", [0, 256])          # the key tile is cut by the diagonal; every row sees all of it
def test_log_sum_exp_of_two_keys(start, dt, d):
    n, s, kv = 256, 80, 128 if start else 80          # one batch element for each of n scores in [0, 1); the row that is looked at is the 16th
    q = np.zeros((n, s, 1, d), np.float32)
    q[..., 0] = 1.0
    q[..., 1] = (np.arange(n) / n).reshape(n, 1, 1)   # at most 8 bits: exact in both types
    scale = 0.6931471824645996                        # f32(ln 2): scores of (almost) whole powers of two
    worst = 0.0
    for top, other in ((0, 15), (14, 15), (15, 3), (14, 1)):
        k = np.zeros((n, kv, 1, d), np.float32)
        k[..., 0] = -256.0                            # no weight
        k[:, top, 0, 0] = 0.0
        k[:, other, 0, 0], k[:, other, 0, 1] = 0.0, -1.0
        v = np.zeros((n, kv, 1, d), np.float32)
        o, lse = torch.empty(n, s, 1, d, device="cuda", dtype=H.TORCH_DT[dt]), torch.empty(n, 1, s, device="cuda")
        low.flash_attn(H.to_dev(q, dt), H.to_dev(k, dt), H.to_dev(v, dt), o, n, s, kv, 1, 1, d, start, scale, None, None, lse)
        torch.cuda.synchronize()
        assert ffi.last_path() == "prefill_tcgen05"
        got = lse.cpu().numpy().astype(np.float64)[:, 0, 15]
        want = np.log1p(np.exp(-scale * np.arange(n) / n))
        worst = max(worst, np.abs(got - want).max())
    assert worst <= BOUND, worst
