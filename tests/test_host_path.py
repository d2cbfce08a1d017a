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
