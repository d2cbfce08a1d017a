"""A CTA of the tensor-core prefill kernel works on one tile pair after the other, with the next one's Q, K and V and its first scores under way while the
last one's rows are written (csrc/prefill_tcgen05.cu). Every row has the same bits as in a call of its own sequence alone, where no CTA has more than one
pair: pairs of one, two and three steps in any succession, tiles without a partner (odd groups), tiles that see no key, sequences that end inside a
tile and on its edge, empty sequences, several pairs for every SM."""
import numpy as np
import pytest
import torch

from luma_b200 import ffi, high, low
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hq,hkv,d,dt", [(4, 4, 128, "bf16"), (6, 2, 64, "f16"), (8, 1, 128, "f16"), (3, 3, 32, "bf16")])
@pytest.mark.parametrize("totals", [True, False])
def test_rows_of_packed_sequences_are_those_of_each_alone(hq, hkv, d, dt, totals):
    rng = np.random.Generator(np.random.Philox(hq * d))
    n = 1600 // hq
    q_lens = rng.choice([0, 1, 17, 127, 128, 129, 200, 256, 257, 383, 500], size=n).tolist()
    k_lens = [max(0, x + int(rng.choice([0, 0, 0, 1, 130, -100]))) for x in q_lens]
    cu_q, cu_k = (torch.tensor(np.concatenate([[0], np.cumsum(x)]), dtype=torch.int32, device="cuda") for x in (q_lens, k_lens))
    g = torch.Generator(device="cuda").manual_seed(d)
    q, k, v = (torch.randn((sum(x), h, d), generator=g, device="cuda", dtype=H.TORCH_DT[dt]) for x, h in ((q_lens, hq), (k_lens, hkv), (k_lens, hkv)))
    o = torch.full_like(q, float("nan"))
    low.flash_attn_varlen(q, k, v, o, cu_q, cu_k, n, max(q_lens), max(k_lens), hq, hkv, d, 1.0 / np.sqrt(d),
                          total_q=q.shape[0] if totals else None, total_k=k.shape[0] if totals else None)
    torch.cuda.synchronize()
    assert ffi.last_path() == "prefill_tcgen05" and ffi.device_status() == 0
    at_q = at_k = 0
    for a, b in zip(q_lens, k_lens):
        unseen = max(0, a - b)                     # rows before the first key
        assert not bool(o[at_q:at_q + unseen].any())
        if a > unseen:
            alone = high.flash_attn_func(q[None, at_q + unseen:at_q + a], k[None, at_k:at_k + b], v[None, at_k:at_k + b], start_pos=max(0, b - a))
            got = o[at_q + unseen:at_q + a]
            if a * (hq // hkv) > 16:
                assert torch.equal(alone[0], got), (a, b)
            else:                                  # (which may be the few-row kernel's: other sums, one rounding of weights and result)
                assert float((alone[0].float() - got.float()).abs().max()) <= 2e-2, (a, b)
        at_q, at_k = at_q + a, at_k + b
    assert ffi.device_status() == 0


@pytest.mark.parametrize("d", [128, 64])
@pytest.mark.parametrize("b,s,hq,hkv", [(40, 130, 8, 8), (9, 900, 12, 4), (2, 1500, 32, 8)])
def test_rows_of_a_batch_are_those_of_each_element_alone(b, s, hq, hkv, d):
    g = torch.Generator(device="cuda").manual_seed(s)
    q, k, v = (torch.randn((b, s, h, d), generator=g, device="cuda", dtype=torch.bfloat16) for h in (hq, hkv, hkv))
    mask = torch.ones((b, s), dtype=torch.uint8, device="cuda")
    mask[:, s - s // 3:] = 0
    for m in (None, mask):
        o, lse = torch.full_like(q, float("nan")), torch.full((b, hq, s), float("nan"), device="cuda")
        low.flash_attn(q, k, v, o, b, s, s, hq, hkv, d, 0, 1.0 / np.sqrt(d), m, None, lse)
        torch.cuda.synchronize()
        assert ffi.last_path() == "prefill_tcgen05" and ffi.device_status() == 0
        for i in range(b):
            per = hq // hkv
            for h in range(hkv):                   # one KV head: at most a few pairs
                o1, l1 = torch.empty_like(o[i:i + 1, :, :per]), torch.empty((1, per, s), device="cuda")
                low.flash_attn(q[i:i + 1, :, h * per:(h + 1) * per].contiguous(), k[i:i + 1, :, h:h + 1].contiguous(), v[i:i + 1, :, h:h + 1].contiguous(), o1, 1, s, s, per, 1, d, 0,
                               1.0 / np.sqrt(d), None if m is None else m[i:i + 1], None, l1)
                assert torch.equal(o1, o[i:i + 1, :, h * per:(h + 1) * per]) and torch.equal(l1, lse[i:i + 1, h * per:(h + 1) * per])


@pytest.mark.parametrize("d", [128, 64])
def test_rows_to_several_buffers(d):
    # the head-sharded epilogue with two buffers of this GPU: a shard's heads in both, the others' left alone
    b, s, hq, hkv, first, total = 2, 700, 16, 4, 8, 32
    g = torch.Generator(device="cuda").manual_seed(d)
    q, k, v = (torch.randn((b, s, h, d), generator=g, device="cuda", dtype=torch.bfloat16) for h in (hq, hkv, hkv))
    outs = [torch.full((b, s, total, d), -7.0, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
    low.flash_attn_allgather(q, k, v, [x.data_ptr() for x in outs], total, first, b, s, s, hq, hkv, d, 0, 1.0 / np.sqrt(d))
    torch.cuda.synchronize()
    want = high.flash_attn_func(q, k, v)
    for x in outs:
        assert torch.equal(x[:, :, first:first + hq], want)
        assert bool((x[:, :, :first] == -7.0).all()) and bool((x[:, :, first + hq:] == -7.0).all())
    assert ffi.device_status() == 0


@pytest.mark.parametrize("d", [128, 64])
@pytest.mark.parametrize("paged", [False, True])
@pytest.mark.parametrize("s", [100, 256, 700])
def test_a_grid_of_one_wave_and_one_with_a_tile_pair_more(s, paged, d):
    # as many CTAs as the device has SMs, each on its own pair, and one pair more, which somebody takes over: the same bits for what they have in common
    sms, page = torch.cuda.get_device_properties(0).multi_processor_count, 16
    per_seq = -(-s // 256)                         # without GQA a pair is two row blocks of one head
    g = torch.Generator(device="cuda").manual_seed(s + d)
    width = -(-s // page)
    most = sms // per_seq + 1
    q = torch.randn((most, s, 1, d), generator=g, device="cuda", dtype=torch.bfloat16)
    k, v = (torch.randn((most * width, page, 1, d) if paged else (most, s, 1, d), generator=g, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    table = torch.randperm(most * width, generator=g, device="cuda").to(torch.int32).view(most, width)
    outs = []
    for b in (sms // per_seq, most):
        o = torch.full_like(q[:b], float("nan"))
        if paged:
            lens = torch.full((b,), s, dtype=torch.int32, device="cuda")
            low.flash_attn_with_kvcache(q[:b], k, v, o, table[:b], lens, b, s, 1, 1, d, page, width, 1.0 / np.sqrt(d))
        else:
            low.flash_attn(q[:b], k[:b], v[:b], o, b, s, s, 1, 1, d, 0, 1.0 / np.sqrt(d))
        torch.cuda.synchronize()
        assert ffi.last_path() == "prefill_tcgen05" and ffi.device_status() == 0
        outs.append(o)
    assert torch.equal(outs[0], outs[1][:len(outs[0])])
    kk, vv = ((x[table[-1].long()].reshape(1, -1, 1, d)[:, :s] if paged else x[-1:]) for x in (k, v))
    assert torch.equal(outs[1][-1:], high.flash_attn_func(q[-1:], kk.contiguous(), vv.contiguous()))
