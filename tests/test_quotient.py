"""The f32 kernel divides a row by its sum with a product, its remainder and one correction (csrc/tile_f32.cuh): compiled for the host, against the division rounded to nearest,
over sums of 1 to 2^24 weights, with mantissas at the ends of their range."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np

from luma_b200.build import find_nvcc


def test_rounded_to_nearest(tmp_path):
    out = tmp_path / "quotient.so"
    subprocess.run([find_nvcc(), "-std=c++17", "-O2", "-shared", "-Xcompiler", "-fPIC,-ffp-contract=off", "-gencode", "arch=compute_100a,code=sm_100a", str(Path(__file__).parent / "cpp" / "quotient.cu"), "-o", str(out)], check=True)
    lib = ctypes.CDLL(str(out))
    rng = np.random.default_rng(1)
    n = 4_000_000
    y = (2.0 ** rng.uniform(0, 24, n)).astype(np.float32)
    x = (rng.standard_normal(n) * y * 2.0 ** rng.uniform(-8, 4, n)).astype(np.float32)
    for k, a in enumerate((x, y)):                                            # mantissas of few bits, of ones, and next to a power of two
        bits = a.view(np.uint32)
        bits[k * 1000:n // 4] &= 0xfffff000
        bits[n // 4:n // 4 + 200_000] |= 0x007fffff
        bits[n // 4 + 100_000 * (1 + k):n // 4 + 300_000] &= 0xff800003
    got = np.empty_like(x)
    lib.quotients(x.ctypes.data_as(ctypes.c_void_p), y.ctypes.data_as(ctypes.c_void_p), got.ctypes.data_as(ctypes.c_void_p), ctypes.c_longlong(n))
    want = x / y
    there = np.abs(want) > 2.0 ** -100
    assert there.sum() > 0.99 * n and np.array_equal(got[there], want[there])
