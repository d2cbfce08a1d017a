"""The cut of few-row calls into equal shares counts what a sequence costs beside its units of 64 tokens (csrc/decode_splitk.cu): shares that begin or end in that
cost, whole columns in it, sequences without tokens between others, more sequences than a warp looks at in one go (128), totals on both sides of the line below which there is
no cost; one to 16 rows, through the three entry points. Against the f64 oracle, twice: the arrival counts are as the first call found them."""
import numpy as np
import pytest
import torch

from luma_b200 import ffi, low
from oracle import binding as ob
from tests import helpers as H

pytestmark = pytest.mark.gpu


def _lengths(kind, n, rng):
    if kind == "even":
        return [64 * 9] * n
    if kind == "short":
        return rng.integers(1, 130, size=n).tolist()
    if kind == "holes":
        return [int(x) if i % 3 else 0 for i, x in enumerate(rng.integers(1, 900, size=n))]
    return [int(x) for x in np.exp(rng.uniform(0, np.log(6000), size=n))]


@pytest.mark.parametrize("kind", ["even", "short", "holes", "mixed"])
@pytest.mark.parametrize("n,new,hq,hkv,d", [(3, 1, 8, 8, 128), (17, 1, 4, 1, 64), (130, 1, 2, 2, 32), (300, 1, 2, 1, 128), (9, 4, 4, 1, 128)])
def test_lengths_of_a_paged_cache(kind, n, new, hq, hkv, d):
    rng = np.random.Generator(np.random.Philox(n + d))
    lens, bs, dt = _lengths(kind, n, rng), 16, "bf16"
    if new > 1:
        lens = [8000] + [max(x, new) for x in lens[1:]]      # (long enough in all for this kernel)
    kc, vc, table = H.make_paged_cache(lens, bs, hkv, d, seed=n)
    kc, vc, q = H.round_to(kc, dt), H.round_to(vc, dt), H.round_to(H.normal((n, new, hq, d), 5), dt)
    want = ob.attn_f64_kvcache(q, kc, vc, lens, table)
    o = torch.empty((n, new, hq, d), device="cuda", dtype=torch.bfloat16)
    args = (H.to_dev(q, dt), H.to_dev(kc, dt), H.to_dev(vc, dt), o, torch.from_numpy(table).cuda(), torch.tensor(lens, dtype=torch.int32, device="cuda"), n, new, hq, hkv, d, bs,
            table.shape[1], 1.0 / np.sqrt(d))
    first = None
    for _ in range(2):
        o.fill_(float("nan"))
        low.flash_attn_with_kvcache(*args)
        torch.cuda.synchronize()
        assert ffi.last_path() == "decode_splitk"
        H.assert_bf16_close(H.to_np(o), want, f"{kind}, {n}")
        assert first is None or torch.equal(first, o)
        first = o.clone()


@pytest.mark.parametrize("b,sq,skv,hq,hkv,d", [(5, 1, 1700, 4, 4, 128), (40, 1, 1601, 8, 8, 64), (7, 4, 2049, 8, 2, 128), (200, 1, 64, 32, 32, 64)])
def test_contiguous(b, sq, skv, hq, hkv, d):
    dt = "f16"
    q, k, v = (H.round_to(H.normal(s, x), dt) for s, x in (((b, sq, hq, d), 1), ((b, skv, hkv, d), 2), ((b, skv, hkv, d), 3)))
    want, lse_want = ob.attn_f64_batch(q, k, v, start_pos=skv - sq, return_lse=True)
    qd = H.to_dev(q, dt)
    o, lse = torch.full_like(qd, float("nan")), torch.full((b, hq, sq), float("nan"), device="cuda")
    low.flash_attn(qd, H.to_dev(k, dt), H.to_dev(v, dt), o, b, sq, skv, hq, hkv, d, skv - sq, 1.0 / np.sqrt(d), None, None, lse)
    torch.cuda.synchronize()
    assert ffi.last_path() == "decode_splitk"
    H.assert_bf16_close(H.to_np(o), want, "contiguous")
    assert np.abs(lse.cpu().numpy() - lse_want).max() <= 1e-3


@pytest.mark.parametrize("decoding", [12, 150])
def test_decoding_sequences_between_prompts(decoding):
    rng = np.random.Generator(np.random.Philox(decoding))
    hq, hkv, d, bs, dt = 4, 1, 128, 16, "bf16"
    kl = [2000, 300] + rng.integers(0, 2000, size=decoding).tolist()
    ql = [400, 300] + [min(1, x) for x in kl[2:]]
    order = rng.permutation(len(kl))
    kl, ql = [int(kl[i]) for i in order], [int(ql[i]) for i in order]
    cu_q, cu_k = (np.concatenate([[0], np.cumsum(x)]).astype(np.int32) for x in (ql, kl))
    kc, vc, table = H.make_paged_cache(kl, bs, hkv, d, seed=3)
    kc, vc, q = H.round_to(kc, dt), H.round_to(vc, dt), H.round_to(H.normal((sum(ql), hq, d), 4), dt)
    want = ob.attn_f64_varlen(q, kc, vc, cu_q, cu_k, block_table=table)
    qd = H.to_dev(q, dt)
    o = torch.full_like(qd, float("nan"))
    low.flash_attn_varlen(qd, H.to_dev(kc, dt), H.to_dev(vc, dt), o, torch.from_numpy(cu_q).cuda(), torch.from_numpy(cu_k).cuda(), len(ql), max(ql), max(kl), hq, hkv, d,
                          1.0 / np.sqrt(d), block_tables=torch.from_numpy(table).cuda(), block_size=bs)
    torch.cuda.synchronize()
    assert ffi.last_path() == "prefill_tcgen05" and ffi.last_launches() == 2 and ffi.device_status() == 0
    H.assert_bf16_close(H.to_np(o), want, "between prompts")
