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


def _dense(b, s, kv, hq=32, hkv=8, d=128, seed=0, dtype=torch.bfloat16):
    g = torch.Generator(device="cuda").manual_seed(seed)
    q, k, v = (torch.randn(b, n, h, d, generator=g, device="cuda").to(dtype) for n, h in ((s, hq), (kv, hkv), (kv, hkv)))
    return lambda: high.flash_attn_func(q, k, v, start_pos=kv - s)


def _mixed(ones, prompts, new, kv, hq=32, hkv=8, d=128, page=16, seed=0, dtype=torch.bfloat16):
    g = torch.Generator(device="cuda").manual_seed(seed)
    q_lens, k_lens = [new] * prompts + [1] * ones, [kv] * (prompts + ones)
    pages = -(-kv // page)
    k, v = (torch.randn(len(k_lens) * pages, page, hkv, d, generator=g, device="cuda").to(dtype) for _ in range(2))
    q = torch.randn(sum(q_lens), hq, d, generator=g, device="cuda").to(dtype)
    table = torch.randperm(len(k_lens) * pages, generator=torch.Generator().manual_seed(seed)).int().view(len(k_lens), pages).cuda()
    cu = [torch.tensor([0] + n, dtype=torch.int32).cumsum(0).int().cuda() for n in (q_lens, k_lens)]
    return lambda: high.flash_attn_varlen_func(q, k, v, *cu, new, kv, block_table=table)


def _capture(call, stream):
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        out = call()
    return graph, out


CAPTURED = {"decode": lambda seed: _decode([3000, 40, 700], seed=seed), "speculate": lambda seed: _decode([5000, 2600], new=4, seed=seed),
            "contiguous": lambda seed: _dense(3, 1, 4000, seed=seed), "mixed": lambda seed: _mixed(24, 3, 256, 3000, seed=seed)}


@pytest.mark.parametrize("kind", CAPTURED)
def test_graphs_captured_on_one_stream_without_a_call_before(kind):
    # the stream has no workspace yet; two graphs of it and plain calls there must not depend on each other, in any order,
    # nor on what becomes of the stream's own workspace
    first, second = CAPTURED[kind](1), CAPTURED[kind](2)
    want1, want2 = first(), second()
    torch.cuda.synchronize()
    ffi.lib.flash_attn_release_workspaces()
    st = torch.cuda.Stream()
    graph1, out1 = _capture(first, st)
    graph2, out2 = _capture(second, st)

    def check(graph, out, want):
        out.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
    check(graph2, out2, want2)          # before the first graph has ever run
    with torch.cuda.stream(st):
        got = second()
    torch.cuda.synchronize()
    assert torch.equal(got, want2)
    check(graph1, out1, want1)
    ffi.lib.flash_attn_release_workspaces()
    check(graph2, out2, want2)
    other = torch.cuda.Stream()         # side by side, again and again
    for o in (out1, out2):
        o.fill_(float("nan"))
    torch.cuda.synchronize()
    for _ in range(20):
        with torch.cuda.stream(other):
            graph1.replay()
        with torch.cuda.stream(st):
            graph2.replay()
    torch.cuda.synchronize()
    assert torch.equal(out1, want1) and torch.equal(out2, want2)
    del graph1, out1
    torch.cuda.synchronize()
    third, want3 = CAPTURED[kind](3), CAPTURED[kind](3)()
    graph3, out3 = _capture(third, st)  # may take what the first graph gave back
    check(graph2, out2, want2)
    check(graph3, out3, want3)
    check(graph2, out2, want2)


def test_buffers_of_graphs_come_back():
    call = _decode([4000] * 8, seed=4)
    call()
    st = torch.cuda.Stream()

    def cycle(n):
        for _ in range(n):
            graph, out = _capture(call, st)
            graph.replay()
            torch.cuda.synchronize()
            del graph, out
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]
    before = cycle(8)
    after = cycle(40)
    assert before - after < 64 << 20, "each of 40 graphs that are gone kept its buffer (about 6 MB each)"
    assert ffi.lib.flash_attn_release_workspaces() >= 1


@pytest.fixture
def no_pool_memory():
    """cudaMallocAsync finds less than 1 MiB: the device's current pool is a small one that is full."""
    from cuda.bindings import runtime as rt

    def ok(ret):
        assert int(ret[0]) == 0, ret
        return ret[1] if len(ret) > 1 else None
    dev = torch.cuda.current_device()
    torch.cuda.synchronize()
    ffi.lib.flash_attn_release_workspaces()
    before = ok(rt.cudaDeviceGetMemPool(dev))
    props = rt.cudaMemPoolProps()
    props.allocType = rt.cudaMemAllocationType.cudaMemAllocationTypePinned
    props.location.type = rt.cudaMemLocationType.cudaMemLocationTypeDevice
    props.location.id = dev
    props.maxSize = 32 << 20
    pool = ok(rt.cudaMemPoolCreate(props))
    ok(rt.cudaDeviceSetMemPool(dev, pool))
    held = []
    while len(held) < 4096:
        err, ptr = rt.cudaMallocAsync(1 << 20, 0)
        if int(err) != 0:
            rt.cudaGetLastError()
            break
        held.append(ptr)
    assert 0 < len(held) < 4096
    yield
    torch.cuda.synchronize()
    ffi.lib.flash_attn_release_workspaces()
    for ptr in held:
        ok(rt.cudaFreeAsync(ptr, 0))
    torch.cuda.synchronize()
    ok(rt.cudaDeviceSetMemPool(dev, before))
    ok(rt.cudaMemPoolDestroy(pool))


@pytest.mark.parametrize("kind", ["speculate", "contiguous", "mixed"])
def test_calls_that_have_another_kernel_run_without_a_workspace(kind, no_pool_memory):
    ffi.lib.flash_attn_set_option(b"force_generic", 1)
    try:
        want = CAPTURED[kind](5)().float()
    finally:
        ffi.lib.flash_attn_set_option(b"force_generic", 0)
    got = CAPTURED[kind](5)().float()
    assert ffi.last_path() == "prefill_tcgen05" and ffi.lib.flash_attn_last_launches() == 1
    assert ffi.last_error() == ""       # nothing went wrong
    torch.cuda.synchronize()
    diff = (got - want).abs()           # two bf16 results of the same f32 sums: the bar of bf16 outputs
    assert diff.max() <= 2e-2 and diff.mean() <= 2e-3


def test_decoding_without_a_workspace_says_so(no_pool_memory):
    from luma_b200 import error
    with pytest.raises(error.CudaError, match="flash_attn_with_kvcache: could not allocate"):
        CAPTURED["decode"](6)()


def _noalloc(lens, hq, hkv, d, seed, page=16):
    """(call on a stream, its output buffer, f64 result) of the allocation-free entry point."""
    import numpy as np
    from oracle import binding as ob
    from tests import helpers as H
    kc, vc, table = H.make_paged_cache(lens, page, hkv, d, seed=seed)
    q = H.normal((len(lens), 1, hq, d), seed + 3)
    dq, dk, dv = (H.to_dev(x, "bf16") for x in (q, kc, vc))
    bt, cl, o = torch.from_numpy(table).cuda(), torch.tensor(lens, dtype=torch.int32, device="cuda"), torch.empty_like(dq)
    scale = float(1.0 / np.sqrt(d))

    def call(stream=None):
        st = stream if stream is not None else torch.cuda.current_stream()
        rc = ffi.lib.flash_attn_decode_bf16_noalloc(dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), o.data_ptr(), bt.data_ptr(), cl.data_ptr(),
                                                    len(lens), hq, hkv, d, page, bt.shape[1], scale, st.cuda_stream)
        assert rc == 0, ffi.last_error()
    want = ob.attn_f64_kvcache(H.round_to(q, "bf16"), H.round_to(kc, "bf16"), H.round_to(vc, "bf16"), lens, table, scale=scale)

    def check(what):
        torch.cuda.synchronize()
        H.assert_bf16_close(H.to_np(o), want, what)
        o.fill_(float("nan"))
    return call, check


def test_allocation_free_calls_after_calls_that_overlapped():
    # the documented misuse, two calls at once on the shared array (in bounds, but their results are spoiled), must not reach the calls
    # that follow, plain or captured before
    problems = [_noalloc(lens, hq, hkv, d, 50 + i) for i, (lens, hq, hkv, d) in enumerate(
        [([9000, 300, 5000], 8, 2, 128), ([2500] * 7, 16, 4, 64), ([40000], 8, 8, 128), ([64, 1, 0, 700], 8, 2, 128)])]
    st = [torch.cuda.Stream(), torch.cuda.Stream()]
    for call, check in problems:
        call()
        check("before")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=st[0]):
        problems[0][0](st[0])
    for _ in range(50):
        for i, j in ((0, 1), (2, 0), (1, 2)):
            problems[i][0](st[0])
            problems[j][0](st[1])
    torch.cuda.synchronize()
    for _, check in problems:
        try:
            check("spoiled")
        except AssertionError:
            pass
    for _ in range(2):
        for n, (call, check) in enumerate(problems):
            call()
            check(f"problem {n} after overlapping calls")
        graph.replay()
        problems[0][1]("captured before, replayed after overlapping calls")


def test_the_per_thread_stream_is_another_stream_in_every_thread():
    # one handle value (2), a stream of its own per thread: the threads' kernels run side by side
    from luma_b200 import low
    import types
    per_thread = types.SimpleNamespace(cuda_stream=2)

    def problem(lens, hq, hkv, seed):
        g = torch.Generator(device="cuda").manual_seed(seed)
        n, pages = len(lens), -(-max(lens) // 16)
        k, v = (torch.randn(n * pages, 16, hkv, 128, generator=g, device="cuda").bfloat16() for _ in range(2))
        q = torch.randn(n, 1, hq, 128, generator=g, device="cuda").bfloat16()
        table = torch.randperm(n * pages, generator=torch.Generator().manual_seed(seed)).int().view(n, pages).cuda()
        cl = torch.tensor(lens, dtype=torch.int32, device="cuda")

        def call(outs, stream=None):
            for o in outs:
                low.flash_attn_with_kvcache(q, k, v, o, table, cl, n, 1, hq, hkv, 128, 16, pages, 0.1, stream)
            if stream is not None:   # nothing of the thread's stream is in flight when the thread ends
                torch.cuda.ExternalStream(stream.cuda_stream).synchronize()
        return call, q
    problems = [problem([20000, 300], 32, 8, 1), problem([9000] * 12, 32, 8, 2), problem([30000], 8, 8, 3)]
    want = []
    for call, q in problems:
        want.append(torch.empty_like(q))
        call([want[-1]])
    torch.cuda.synchronize()
    ffi.lib.flash_attn_release_workspaces()
    for _ in range(12):      # more threads in all than the table has entries
        outs = [[torch.full_like(q, float("nan")) for _ in range(8)] for _, q in problems]
        torch.cuda.synchronize()
        threads = [threading.Thread(target=call, args=(o, per_thread)) for (call, _), o in zip(problems, outs)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        torch.cuda.synchronize()
        for w, out in zip(want, outs):
            assert all(torch.equal(w, o) for o in out)
