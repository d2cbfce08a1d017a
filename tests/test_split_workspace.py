"""The scratch memory of the split-K kernel: whose it is between its look-up and the launch, under stream capture, where
there is none to be had, and what a call leaves in it for the next."""
import threading

import pytest
import torch

from luma_b200 import ffi, high

pytestmark = pytest.mark.gpu


def _decode(lens, hq=32, hkv=8, d=128, page=16, new=1, seed=0, dtype=torch.bfloat16):
    """A paged call: (function, number of arguments that it needs kept alive is its closure's)."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    need = [-(-n // page) for n in lens]
    order = torch.randperm(sum(need), generator=torch.Generator().manual_seed(seed + 1)).int()
    table = torch.zeros(len(lens), max(need), dtype=torch.int32)
    at = 0
    for i, n in enumerate(need):
        table[i, :n] = order[at:at + n]
        at += n
    k = torch.randn(sum(need), page, hkv, d, generator=g, device="cuda").to(dtype)
    v = torch.randn(sum(need), page, hkv, d, generator=g, device="cuda").to(dtype)
    q = torch.randn(len(lens), new, hq, d, generator=g, device="cuda").to(dtype)
    cl = torch.tensor(lens, dtype=torch.int32, device="cuda")
    table = table.cuda()
    return lambda: high.flash_attn_with_kvcache(q, k, v, cl, table)


def test_two_threads_on_one_stream_with_sizes_that_grow():
    # one CTA slot's worth of partials to all of them, 1 to 300 sequences: every step of a thread may make the buffer
    # that the other thread is about to launch on too small. Results do not depend on timing, so they are compared bit for bit.
    calls = [_decode([300 + 700 * i] * n, hq=hq, hkv=hkv, new=new, seed=i)
             for i, (n, hq, hkv, new) in enumerate([(1, 8, 8, 1), (2, 32, 8, 1), (5, 32, 8, 4), (30, 32, 32, 1), (300, 8, 2, 1)])]
    want = [c() for c in calls]
    torch.cuda.synchronize()
    wrong = []

    def work(order):
        for _ in range(20):
            for i in order:
                if not torch.equal(calls[i](), want[i]):   # the same (default) stream in every thread
                    wrong.append(i)
    for _ in range(3):
        ffi.lib.flash_attn_release_workspaces()
        threads = [threading.Thread(target=work, args=(order,)) for order in ([0, 1, 2, 3, 4], [4, 2, 0, 3, 1], [1, 3, 0, 4, 2])]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    assert not wrong, f"calls {sorted(set(wrong))} differ from their single-threaded result"


def test_more_streams_than_workspaces_from_two_threads():
    # beyond 32 streams the least recently used buffer is released: never one that another thread is launching on
    call = _decode([2000, 600, 64], seed=9)
    want = call()
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(40)]
    wrong = []

    def work(mine):
        for _ in range(4):
            for st in mine:
                with torch.cuda.stream(st):
                    o = call()
                    st.synchronize()
                    if not torch.equal(o, want):
                        wrong.append(st)
    threads = [threading.Thread(target=work, args=(streams[i::2],)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
