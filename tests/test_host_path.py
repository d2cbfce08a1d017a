"""The native host path (csrc/host_fast.cpp) against the Python path beside it: which calls it takes, that both give the same,
and that what it does not take raises what the Python path raises."""
import pytest
import torch

from luma_b200 import error as E
from luma_b200 import low

gpu = pytest.mark.gpu


@gpu
def test_sizes_whose_product_does_not_fit_64_bits_are_too_large_for_any_buffer():
    # 2^16 * 2^16 * 2^25 * 2^7 = 2^64, which wraps to 0 elements
    t = torch.zeros(1024, dtype=torch.bfloat16, device="cuda")
    with pytest.raises(E.BufferTooSmall):
        low.flash_attn(t, t, t, t, 1 << 16, 1 << 16, 1 << 16, 1 << 25, 1 << 25, 128, 0, 1.0)
    i = torch.zeros(4, dtype=torch.int32, device="cuda")
    with pytest.raises(E.BufferTooSmall):
        low.kvcache_append(t, t, t, t, i, i, 1 << 16, 1 << 16, 1 << 25, 128, 16, 1)


def test_an_extension_of_another_installation_is_not_loaded(monkeypatch, tmp_path):
    # the file's name says which Python and which torch it was built for; without it the front end works, in Python
    import importlib.metadata
    import sysconfig

    from luma_b200 import build, host_path
    assert sysconfig.get_config_var("SOABI") in build.host_path_file().name and importlib.metadata.version("torch") in build.host_path_file().name
    assert host_path.PATH == build.host_path_file() and host_path._load() is not None
    monkeypatch.setattr(host_path, "PATH", tmp_path / "_host.other.so")
    with pytest.warns(RuntimeWarning, match="python -m luma_b200.build"):
        assert host_path._load() is None
    assert host_path._not_taken(1, 2, 3) is None


def test_the_extension_is_rebuilt_when_a_declaration_changes(monkeypatch, tmp_path):
    from luma_b200 import build
    asked = []
    monkeypatch.setattr(build, "_stale", lambda target, deps: asked.append((target, [d.name for d in deps])) or False)
    build.build()
    deps = dict(asked)[build.host_path_file()]
    assert {"host_fast.cpp", "flash_attn.h", "luma_nn_kernels.h"} <= set(deps)


def _paged(hkv=2, d=64, page=16, lens=(70, 300), dtype=torch.bfloat16):
    g = torch.Generator(device="cuda").manual_seed(7)
    pages = -(-max(lens) // page)
    kc, vc = (torch.randn(len(lens) * pages, page, hkv, d, generator=g, device="cuda").to(dtype) for _ in range(2))
    table = torch.randperm(len(lens) * pages, generator=torch.Generator().manual_seed(8)).int().view(len(lens), pages).cuda()
    return kc, vc, table, torch.tensor(lens, dtype=torch.int32, device="cuda")


def _calls(dtype):
    """name of the native function -> (its arguments, the entry point's call, the tensors that the call writes)"""
    from luma_b200 import high
    g = torch.Generator(device="cuda").manual_seed(3)

    def rnd(*shape):
        return torch.randn(*shape, generator=g, device="cuda").to(dtype)
    q, k, v = rnd(2, 37, 8, 64), rnd(2, 90, 2, 64), rnd(2, 90, 2, 64)
    kc, vc, table, lens = _paged(dtype=dtype)
    cu_q, cu_k = (torch.tensor(x, dtype=torch.int32, device="cuda") for x in ([0, 20, 37], [0, 70, 370]))
    qp, kp, vp, q1 = rnd(37, 8, 64), rnd(370, 2, 64), rnd(370, 2, 64), rnd(2, 3, 8, 64)
    new_k, new_v = rnd(2, 3, 2, 64), rnd(2, 3, 2, 64)
    o, lse = torch.empty_like(q), torch.empty(2, 8, 37, device="cuda")
    mask = (torch.rand(2, 90, generator=g, device="cuda") < 0.8).to(torch.uint8)
    low_args = (q, k, v, o, 2, 37, 90, 8, 2, 64, 53, 0.125)
    app = (new_k, new_v, kc, vc, table, lens, 2, 3, 2, 64, 16, table.shape[1])
    x = rnd(33, 257)
    return {
        "attn": ((q, k, v, None, 53, False), lambda: high.flash_attn_func(q, k, v, start_pos=53)),
        "attn lse": ((q, k, v, 0.2, 53, True), lambda: high.flash_attn_func(q, k, v, 0.2, start_pos=53, return_lse=True)),
        "low_attn": (low_args + (mask, lse), lambda: (low.flash_attn(*low_args, mask, None, lse), o.clone(), lse.clone())[1:]),
        "low_attn plain": (low_args + (None, None), lambda: (low.flash_attn(*low_args), o.clone())[1]),
        "varlen": ((qp, kp, vp, cu_q, cu_k, 20, 300, None, None), lambda: high.flash_attn_varlen_func(qp, kp, vp, cu_q, cu_k, 20, 300)),
        "varlen paged": ((qp, kc, vc, cu_q, cu_k, 20, 300, 0.1, table),
                         lambda: high.flash_attn_varlen_func(qp, kc, vc, cu_q, cu_k, 20, 300, 0.1, block_table=table)),
        "kvcache": ((q1, kc, vc, lens, table, None), lambda: high.flash_attn_with_kvcache(q1, kc, vc, lens, table)),
        "append": (app, lambda: (low.kvcache_append(*app), kc.clone(), vc.clone())[1:]),
        "softmax": ((x,), lambda: low.softmax_last_dim(x)),
    }


@gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
def test_native_and_python_path_agree_bit_for_bit(dtype, monkeypatch):
    from luma_b200 import host_path
    taken = _calls(dtype)
    native = {}
    for name, (args, entry) in taken.items():
        assert getattr(host_path, name.split()[0])(*args) is not None, f"{name}: plain arguments are not taken"
        native[name] = entry()
    for f in ("attn", "low_attn", "varlen", "kvcache", "append", "softmax"):
        monkeypatch.setattr(host_path, f, host_path._not_taken)
    python = {name: entry() for name, (_, entry) in _calls(dtype).items()}      # the same seeds, buffers of its own
    for name in taken:
        a, b = (x if isinstance(x, tuple) else (x,) for x in (native[name], python[name]))
        assert len(a) == len(b) and all(torch.equal(x, y) for x, y in zip(a, b)), name


@gpu
def test_what_the_native_path_leaves_to_python():
    from luma_b200 import high, host_path
    calls = _calls(torch.bfloat16)
    for name, (args, _) in calls.items():
        f = getattr(host_path, name.split()[0])
        t = args[0]
        strided = torch.empty(*t.shape[:-1], 2 * t.shape[-1], dtype=t.dtype, device="cuda")[..., ::2]
        for first in (t.cpu(), strided, None, 3):
            assert f(first, *args[1:]) is None, (name, type(first))
        if name != "append":      # (which copies bytes: the C ABI checks the element size)
            assert f(t.double(), *args[1:]) is None, name
            assert len(args) == 1 or f(t, args[1].float(), *args[2:]) is None, name
        assert f(*args[:-1]) is None, name
    (q, k, v, *_), _ = calls["attn"]
    assert host_path.attn(q, k, v, 1, 53, False) is None              # an integer scale: float() is Python's business
    assert host_path.attn(q, k, v, None, True, False) is None
    assert host_path.attn(q, k, v, None, -1, False) is None
    # ... and raises there what it always raised
    with pytest.raises(E.InvalidStartPos):
        high.flash_attn_func(q, k, v, start_pos=-1)
    with pytest.raises(E.Unsupported):
        high.flash_attn_func(q.double(), k.double(), v.double())
    with pytest.raises(E.Unsupported):
        high.flash_attn_func(q, k.float(), v)
    with pytest.raises(E.Unsupported):
        high.flash_attn_func(q, k, v, causal=False)
    with pytest.raises(E.InvalidShape):
        high.flash_attn_func(q[:, :, :7].contiguous(), k, v)          # 7 heads over 2
    with pytest.raises(E.InvalidShape):
        high.flash_attn_func(q, k[:1].contiguous(), v[:1].contiguous())
    with pytest.raises(E.InvalidHeadSize):
        high.flash_attn_func(q[..., :48].contiguous(), k[..., :48].contiguous(), v[..., :48].contiguous())
    o = torch.empty_like(q)
    with pytest.raises(E.BufferTooSmall):
        low.flash_attn(q, k, v, o[:1], 2, 37, 90, 8, 2, 64, 53, 0.125)
    with pytest.raises(E.BufferTooSmall):
        low.flash_attn(q, k, v, o, 2, 37, 90, 8, 2, 64, 53, 0.125, torch.ones(2, 89, dtype=torch.uint8, device="cuda"))
    strided = torch.cat([q, q], dim=-1)[..., :64]
    assert torch.equal(high.flash_attn_func(strided, k, v, start_pos=53), high.flash_attn_func(q, k, v, start_pos=53))
