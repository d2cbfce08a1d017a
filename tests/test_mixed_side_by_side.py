"""The few-row sequences of a packed batch on part of the SMs, in CTAs of eight warps ahead of the prefill kernel, which does not wait for them but ends behind them
(csrc/decode_splitk.cu, prefill_tcgen05.cu). Contexts around the 128 tokens of a wide CTA's unit, empty sequences, one and several rows, what follows in the stream reads both kernels'
rows, call behind call and in a graph with other values. Against the f64 oracle; the sizes are on the side of the rule that launches ahead."""
import numpy as np
import pytest
import torch

from luma_b200 import ffi, low
from oracle import binding as ob
from tests import helpers as H

pytestmark = pytest.mark.gpu


def _batch(seed, decoding, prompts, longest, hq, hkv, d, dt, page=16, several=False):
    rng = np.random.Generator(np.random.Philox(seed))
    kl = [longest] * prompts + [127, 128, 129, 1, longest, 0] + rng.integers(1, longest, size=decoding - 6).tolist()
    ql = [200] * prompts + [min(int(rng.integers(1, 16 // (hq // hkv) + 1)) if several else 1, x) for x in kl[prompts:]]
    order = rng.permutation(len(kl))
    kl, ql = [int(kl[i]) for i in order], [int(ql[i]) for i in order]
    cu_q, cu_k = (np.concatenate([[0], np.cumsum(x)]).astype(np.int32) for x in (ql, kl))
    kc, vc, table = H.make_paged_cache(kl, page, hkv, d, seed=seed)
    kc, vc, q = H.round_to(kc, dt), H.round_to(vc, dt), H.round_to(H.normal((sum(ql), hq, d), seed), dt)
    want = ob.attn_f64_varlen(q, kc, vc, cu_q, cu_k, block_table=table)
    dev = [H.to_dev(x, dt) for x in (q, kc, vc)]
    o = torch.full_like(dev[0], float("nan"))
    args = (o, torch.from_numpy(cu_q).cuda(), torch.from_numpy(cu_k).cuda(), len(ql), max(ql), max(kl), hq, hkv, d, 1.0 / np.sqrt(d), torch.from_numpy(table).cuda(), page)
    return dev, o, args, want


@pytest.mark.parametrize("decoding,prompts,longest,hq,hkv,d,dt,several", [
    (200, 1, 1500, 8, 2, 128, "bf16", False), (200, 1, 1500, 8, 2, 128, "f16", True), (80, 2, 1300, 8, 2, 64, "bf16", False), (120, 3, 1100, 8, 8, 128, "bf16", True), (300, 2, 700, 8, 2, 128, "f16", False),
    (40, 3, 200, 32, 32, 128, "bf16", False), (16, 1, 260, 32, 8, 64, "bf16", False),   # the ends of short sequences: fewer or more SMs than the keys alone ask for
])
def test_rows_of_both_kernels(decoding, prompts, longest, hq, hkv, d, dt, several):
    dev, o, args, want = _batch(decoding, decoding, prompts, longest, hq, hkv, d, dt, several=several)
    first = None
    for _ in range(20):
        o.fill_(float("nan"))
        low.flash_attn_varlen(*dev, *args, total_q=dev[0].shape[0])
        seen = o.clone()                           # behind it in the stream
        assert ffi.last_path() == "prefill_tcgen05" and ffi.last_launches() == 2
        first = seen if first is None else first
        assert torch.equal(seen, first)
    assert ffi.device_status() == 0
    H.assert_bf16_close(H.to_np(first), want, f"{decoding} beside {prompts}")


def test_in_a_graph_with_other_values():
    dev, o, args, want = _batch(9, 200, 1, 1500, 8, 2, 128, "bf16")
    call = lambda: low.flash_attn_varlen(*dev, *args, total_q=dev[0].shape[0])
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        call()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=stream):
            call()
            seen = o + 0
    for scale in (1.0, -1.0, 0.5):
        keep = dev[2].clone()
        dev[2].mul_(scale)
        o.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert ffi.device_status() == 0
        H.assert_bf16_close(H.to_np(seen), want * scale, f"V times {scale}")
        dev[2].copy_(keep)
    del graph
