"""Row softmax of the math path: the oracle (luma-cpu's online softmax) against an f64 formula on
CPU, and the CUDA kernels through the C ABI against the oracle — row lengths that take the
warp-per-row, CTA-per-row and two-pass kernels, unaligned lengths, -inf entries, an all -inf row,
in-place operation, f32 / f16 / bf16."""
import numpy as np
import pytest
import torch

from oracle import binding as ob
from tests import helpers as H


def _ref64(x):
    x = x.astype(np.float64)
    e = np.exp(x - x.max(axis=-1, keepdims=True))
    return e / e.sum(axis=-1, keepdims=True)


def test_oracle_softmax_matches_f64_formula():
    x = H.normal((37, 513), 5) * 3.0
    np.testing.assert_allclose(ob.softmax_last_dim_f32(x), _ref64(x), rtol=5e-6, atol=1e-9)   # f32 running sum of 513 terms
    x[3, 10:] = -np.inf   # masked tail, as the causal mask produces
    got = ob.softmax_last_dim_f32(x)
    assert np.all(got[3, 10:] == 0.0) and abs(got[3].sum() - 1.0) < 1e-6


# (rows, row_size): up to 1024 -> warp kernel; up to 32768 -> CTA kernel; beyond -> two-pass
SHAPES = [(64, 8), (33, 256), (5, 1000), (17, 2048), (9, 4096), (3, 16384), (2, 40000), (7, 1001), (4, 77), (2, 33000)]


@pytest.mark.gpu
@pytest.mark.parametrize("dt", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("shape", SHAPES, ids=[str(s) for s in SHAPES])
def test_softmax_kernel_matches_oracle(shape, dt):
    from luma_b200 import ffi, low
    rows, n = shape
    x = H.round_to(H.normal((rows, n), 11 + n) * 2.5, dt)
    if n > 20:
        x[0, n // 2:] = -np.inf   # a causally masked row
    want = ob.softmax_last_dim_f32(x)
    xd = H.to_dev(x, dt)
    got = low.softmax_last_dim(xd)
    torch.cuda.synchronize()
    assert ffi.last_path().startswith("softmax_")
    g = H.to_np(got)
    if dt == "f32":
        np.testing.assert_allclose(g, want, rtol=2e-5, atol=1e-9)   # f32 sums in a different order, ex2.approx
    else:
        # one rounding of the result to 8 (bf16) or 11 (f16) significant bits
        rel = 2.0 ** -8 if dt == "bf16" else 2.0 ** -11
        atol = 4e-8 if dt == "f16" else 1e-9   # f16 results below 6.1e-5 are subnormal: spacing 6e-8
        assert np.all(np.abs(g - want) <= (rel + 2e-5) * want + atol), np.abs(g - want).max()
    assert np.all(g[0, n // 2:] == 0.0) if n > 20 else True
    # in place gives the same bits
    y = xd.clone()
    low.softmax_last_dim(y, out=y)
    torch.cuda.synchronize()
    assert torch.equal(y, got)


@pytest.mark.gpu
@pytest.mark.parametrize("dt", ["f32", "bf16", "f16"])
def test_softmax_rows_that_begin_anywhere(dt):
    """Rows that begin on no 16-byte boundary: odd and even sizes at both sides of every kernel's longest row, bases off the boundary by one
    element, by two and more, input and output alike or not. Guard elements around both stay as they are, the NaN around the input reaches no
    row, and a row's own NaN reaches its whole row."""
    from luma_b200 import low
    V = 4 if dt == "f32" else 8
    sizes = sorted({1, 2, 3, 7, 162, 1413} | {n + o for n in (128, 256, 512, 1024, 2048, 4096, 8192, 16384, 16400, 18432, 20480, 32768) for o in (-1, 0, 1, 2)})
    for n in sizes:
        rows = 9 if n < 5000 else 3
        for off_in, off_out in ((0, 0), (1, 1), (V - 1, V - 1), (0, 1), (3, 0)):
            x = H.round_to(H.normal((rows, n), 7 + n) * 2.5, dt)
            x[0, n // 2 + 1:] = -np.inf
            if n > 40:
                x[-1, n - 1] = np.nan
                x[1, 1:] = -np.inf
                x[1, n - 1] = np.nan      # with nothing but -inf beside it
            src = torch.full((rows * n + 2 * V,), float("nan"), device="cuda", dtype=H.to_dev(x[:1, :1], dt).dtype)
            dst = torch.full_like(src, -3.0)
            xd, yd = src[off_in:off_in + rows * n].view(rows, n), dst[off_out:off_out + rows * n].view(rows, n)
            xd.copy_(H.to_dev(x, dt))
            low.softmax_last_dim(xd, out=yd)
            torch.cuda.synchronize()
            g = H.to_np(yd)
            want = _ref64(np.nan_to_num(x, nan=0.0, neginf=-np.inf))
            if n > 40:
                want[[1, -1]] = np.nan
            # f32: sums of n terms in another order, ex2.approx, an argument rounded at |x| up to 12; 16 bits: one rounding of the result
            rel, atol = {"f32": (1e-5, 1e-9), "bf16": (2.0 ** -8 + 1e-5, 1e-9), "f16": (2.0 ** -11 + 1e-5, 4e-8)}[dt]
            np.testing.assert_allclose(g, want, rtol=rel, atol=atol, err_msg=f"{n} {off_in} {off_out}")
            around = torch.cat([dst[:off_out], dst[off_out + rows * n:]])
            assert bool((around == -3.0).all()), (n, off_in, off_out)


@pytest.mark.gpu
@pytest.mark.parametrize("dt", ["f32", "bf16", "f16"])
@pytest.mark.parametrize("n", [162, 1413, 4099, 16383, 32761, 33001])
def test_softmax_in_place_of_rows_that_begin_anywhere(n, dt):
    """A row's first and last words also hold its neighbours' ends, which other CTAs write meanwhile: the same bits as into another tensor."""
    from luma_b200 import low
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn((1500, n), generator=g, device="cuda", dtype=H.TORCH_DT[dt])
    want = low.softmax_last_dim(x)
    for _ in range(3):
        y = x.clone()
        low.softmax_last_dim(y, out=y)
        assert torch.equal(y, want)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2 ** 31 - 8, 2 ** 31 - 2])
def test_softmax_of_a_row_near_the_longest(n):
    """The largest row sizes of the signature, on and off the 16-byte grid: they are read twice like any long row, and a column counter passes 2^31."""
    from luma_b200 import ffi, low
    x = torch.zeros((1, n), device="cuda", dtype=torch.bfloat16)
    tall = [0, 1, n // 2 + 1, n - 4097, n - 1]
    x[0, tall] = 10.0
    y = low.softmax_last_dim(x, out=x)
    torch.cuda.synchronize()
    assert ffi.last_path() == "softmax_stream"
    total = len(tall) + (n - len(tall)) * np.exp(-10.0)
    got = y[0, tall].double().cpu().numpy()
    np.testing.assert_allclose(got, 1.0 / total, rtol=2.0 ** -8 + 1e-4)       # one rounding to 8 bits; whole counts below 2^24 in each thread's sum
    y[0, tall] = float(y[0, 2])
    assert bool((y == y[0, 2]).all())
    np.testing.assert_allclose(float(y[0, 2]), np.exp(-10.0) / total, rtol=2.0 ** -8 + 1e-4)


@pytest.mark.gpu
def test_softmax_all_minus_inf_row_and_errors():
    import luma_b200 as L
    from luma_b200 import low
    x = torch.full((3, 64), float("-inf"), device="cuda")
    x[1] = 0.0
    y = low.softmax_last_dim(x)
    torch.cuda.synchronize()
    assert torch.isnan(y[0]).all() and torch.isnan(y[2]).all()      # as the reference's arithmetic gives
    assert torch.allclose(y[1], torch.full((64,), 1.0 / 64, device="cuda"))
    with pytest.raises(L.Unsupported):
        low.softmax_last_dim(torch.zeros(4, 8, device="cuda").t())
