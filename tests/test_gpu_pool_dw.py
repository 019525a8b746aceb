"""Parity of pooling and depthwise convolution against the CPU oracle."""
import numpy as np
import pytest

from oracle import exb_oracle as O
from tests.util import kernels_of, dev, host, rng, f16_round, to_nhwc, to_nchw

pytestmark = pytest.mark.gpu


def _capi():
    from excalibur_b200 import capi
    return capi


POOL_CASES = [
    # N, C, H, W, type, k, s, pad, pad_mode, cip
    (2, 64, 112, 112, 0, 3, 2, 1, 1, 0),     # ResNet stem pool
    (1, 256, 20, 20, 0, 5, 1, 2, 1, 0),      # SPPF pool
    (3, 16, 7, 9, 0, 2, 2, 0, 0, 0),         # ceil mode, ragged
    (2, 8, 13, 13, 1, 3, 2, 1, 1, 0),        # avg, exclude pad
    (2, 8, 13, 13, 1, 3, 2, 1, 1, 1),        # avg, include pad
    (1, 24, 10, 10, 1, 2, 2, 0, 0, 1),       # avg, ceil
    (1, 8, 5, 5, 1, 3, 1, 1, 0, 1),
]


@pytest.mark.parametrize("case", POOL_CASES)
@pytest.mark.parametrize("dtype", ["f16", "f32"])
def test_pool(ctx, case, dtype):
    capi = _capi()
    N, Cc, H, W, type_, k, s, pad, pad_mode, cip = case
    x = rng(sum(case)).standard_normal((N, Cc, H, W)).astype(np.float32)
    if dtype == "f16":
        x = f16_round(x)
    ref = O.pool2d_f32(x, type_, k, s, pad, False, pad_mode, cip)
    d = capi.make_pool_desc(N, H, W, Cc, type_, k, s, pad, False, pad_mode, cip,
                            capi.EXB_F16 if dtype == "f16" else capi.EXB_F32)
    xd = dev(to_nhwc(x).astype(np.float16 if dtype == "f16" else np.float32))
    y, _ = capi.pool2d(ctx, d, xd)
    ctx.sync_check()
    y = to_nchw(host(y).astype(np.float32))
    assert y.shape == ref.shape
    if type_ == 0:
        np.testing.assert_array_equal(y, ref)
    elif dtype == "f32":
        np.testing.assert_allclose(y, ref, rtol=1e-6, atol=1e-6)
    else:
        np.testing.assert_allclose(y, ref, rtol=1e-3, atol=1e-3)


@pytest.mark.parametrize("type_", [0, 1])
@pytest.mark.parametrize("shape", [(4, 512, 7, 7), (2, 1280, 7, 7), (1, 64, 56, 56), (3, 8, 1, 1)])
def test_global_pool(ctx, type_, shape):
    capi = _capi()
    N, Cc, H, W = shape
    x = f16_round(rng(N + Cc).standard_normal(shape))
    ref = O.pool2d_f32(x, type_, global_pool=True)
    d = capi.make_pool_desc(N, H, W, Cc, type_, global_pool=True, dtype=capi.EXB_F16)
    y, _ = capi.pool2d(ctx, d, dev(to_nhwc(x).astype(np.float16)))
    ctx.sync_check()
    y = to_nchw(host(y).astype(np.float32))
    assert y.shape == ref.shape == (N, Cc, 1, 1)
    if type_ == 0:
        np.testing.assert_array_equal(y, ref)
    else:
        np.testing.assert_allclose(y, ref, rtol=2e-3, atol=1e-3)


def test_pool_int8_and_second_output(ctx):
    capi = _capi()
    N, Cc, H, W = 2, 64, 30, 30
    r = rng(77)
    xq = r.integers(-128, 128, (N, Cc, H, W)).astype(np.int8)
    d = capi.make_pool_desc(N, H, W, Cc, 0, 3, 2, 1, dtype=capi.EXB_I8)
    y, _ = capi.pool2d(ctx, d, dev(to_nhwc(xq)))
    ref = O.pool2d_f32(xq.astype(np.float32), 0, 3, 2, 1)
    np.testing.assert_array_equal(to_nchw(host(y)).astype(np.float32), ref)
    # fp16 max pool that also emits the int8 tensor the next int8 conv consumes
    x = f16_round(np.abs(r.standard_normal((N, Cc, H, W))) * 3)
    s = np.float32(127.0 / x.max())
    d = capi.make_pool_desc(N, H, W, Cc, 0, 3, 2, 1, dtype=capi.EXB_F16, out2_dtype=capi.EXB_I8, out2_scale=s)
    y, y2 = capi.pool2d(ctx, d, dev(to_nhwc(x).astype(np.float16)))
    ctx.sync_check()
    ref = O.pool2d_f32(x, 0, 3, 2, 1)
    np.testing.assert_array_equal(to_nchw(host(y).astype(np.float32)), ref)
    np.testing.assert_array_equal(to_nchw(host(y2)), O.requantize_rne(ref, s))


DW_CASES = [
    # N, C, H, W, k, s, pad, bias, act
    (2, 32, 112, 112, 3, 1, 1, True, 103),
    (2, 96, 56, 56, 3, 2, 1, True, 103),
    (1, 144, 57, 31, 3, 1, 1, False, 1),
    (1, 144, 57, 31, 3, 2, 1, True, 0),
    (3, 8, 9, 9, 5, 1, 2, True, 0),
    (1, 16, 4, 4, 4, 1, 0, True, 0),
    (2, 24, 15, 15, 3, 2, 0, True, 104),
]


@pytest.mark.parametrize("case", DW_CASES)
def test_dwconv_f16(ctx, case):
    capi = _capi()
    N, Cc, H, W, k, s, pad, has_bias, act = case
    r = rng(sum(case[:7]))
    x = f16_round(r.standard_normal((N, Cc, H, W)))
    w = (r.standard_normal((Cc, 1, k, k)) * 0.3).astype(np.float32)
    b = (r.standard_normal(Cc) * 0.1).astype(np.float32) if has_bias else None
    ref = O.dwconv2d_f32(x, w, b, s, pad, act)
    d = capi.make_dw_desc(N, H, W, Cc, k, s, pad, act=act)
    wp = capi.DwWeights(ctx, d, w, b)
    y = capi.dwconv2d(ctx, d, dev(to_nhwc(x).astype(np.float16)), wp)
    ctx.sync_check()
    y = to_nchw(host(y).astype(np.float32))
    assert y.shape == ref.shape
    np.testing.assert_allclose(y, ref, rtol=2e-3, atol=2e-3)


def test_dwconv_int8_in_out(ctx):
    capi = _capi()
    N, Cc, H, W = 2, 64, 28, 28
    r = rng(123)
    xq = r.integers(-128, 128, (N, Cc, H, W)).astype(np.int8)
    in_scale = np.float32(1.0 / 31.0)
    w = (r.standard_normal((Cc, 1, 3, 3)) * 0.3).astype(np.float32)
    b = (r.standard_normal(Cc) * 0.1).astype(np.float32)
    v = O.dwconv2d_f32(xq.astype(np.float32) * in_scale, w, b, 1, 1, 103)
    out_scale = np.float32(127.0 / 6.0)
    ref = O.requantize_rne(v, out_scale).astype(np.int32)
    d = capi.make_dw_desc(N, H, W, Cc, 3, 1, 1, capi.EXB_I8, capi.EXB_I8, 103, in_scale, out_scale)
    wp = capi.DwWeights(ctx, d, w, b)
    y = to_nchw(host(capi.dwconv2d(ctx, d, dev(to_nhwc(xq)), wp))).astype(np.int32)
    ctx.sync_check()
    # fp32 summation order differs from the oracle's double accumulation: at most 1 LSB where the
    # pre-rounding value sits on a rounding boundary.
    assert np.abs(y - ref).max() <= 1
    assert (y != ref).mean() < 1e-3


# Edges of the streaming 3x3 kernel: maps smaller than a thread's four columns, one row, ragged column groups, channel
# counts that do not fill (8, 24) or do not fit (264, 1240) one CTA, rows that end inside a stage, no padding; fp16 and
# int8 results.
DW_STREAM_CASES = [
    # N, C, H, W, stride, pad, act
    (1, 8, 1, 1, 1, 1, 103), (2, 8, 3, 3, 1, 0, 0), (3, 24, 5, 2, 1, 1, 1), (1, 264, 9, 33, 1, 1, 103), (2, 1240, 7, 6, 1, 1, 104),
    (1, 8, 2, 2, 2, 1, 103), (1, 16, 3, 4, 2, 1, 1), (2, 264, 13, 12, 2, 1, 103), (1, 40, 31, 257, 2, 1, 0), (5, 96, 40, 11, 2, 0, 103),
    (37, 32, 30, 31, 1, 1, 1), (64, 144, 14, 14, 1, 1, 103),
]


@pytest.mark.parametrize("out_i8", [False, True])
@pytest.mark.parametrize("case", DW_STREAM_CASES)
def test_dwconv_stream_edges(ctx, case, out_i8):
    capi = _capi()
    N, Cc, H, W, s, pad, act = case
    r = rng(sum(case))
    x = f16_round(r.standard_normal((N, Cc, H, W)))
    w = (r.standard_normal((Cc, 1, 3, 3)) * 0.3).astype(np.float32)
    b = (r.standard_normal(Cc) * 0.1).astype(np.float32)
    ref = O.dwconv2d_f32(x, w, b, s, pad, act)
    scale = np.float32(127.0 / 6.0)
    d = capi.make_dw_desc(N, H, W, Cc, 3, s, pad, capi.EXB_F16, capi.EXB_I8 if out_i8 else capi.EXB_F16, act, out_scale=scale)
    y = capi.dwconv2d(ctx, d, dev(to_nhwc(x).astype(np.float16)), capi.DwWeights(ctx, d, w, b))
    ctx.sync_check()
    y = to_nchw(host(y).astype(np.float32))
    assert y.shape == ref.shape
    if out_i8:
        diff = np.abs(y - O.requantize_rne(ref, scale).astype(np.float32))
        assert diff.max() <= 1 and (diff != 0).mean() < 1e-2
    else:
        np.testing.assert_allclose(y, ref, rtol=2e-3, atol=2e-3)


# CTAs of several tiles and slabs: the int8 kernel of stride 1 keeps the place of the next tile elsewhere than the others.  Whole
# numbers, whose fp16 result is exact.
@pytest.mark.parametrize("case", [(64, 160, 56, 56, 1, 1), (130, 192, 28, 28, 1, 1), (300, 528, 9, 21, 1, 0), (1100, 16, 17, 30, 1, 1), (64, 96, 57, 40, 2, 1)])
def test_dwconv_stream_of_many_tiles(ctx, case):
    import torch
    capi = _capi()
    N, Cc, H, W, s, pad = case
    g = torch.Generator("cuda").manual_seed(sum(case))
    x = torch.randint(-4, 5, (N, H, W, Cc), generator=g, device="cuda").half()
    r = rng(sum(case))
    w, b = r.integers(-2, 3, (Cc, 1, 3, 3)).astype(np.float32), r.integers(-9, 10, Cc).astype(np.float32)
    y = []
    for out in (capi.EXB_F16, capi.EXB_I8):
        d = capi.make_dw_desc(N, H, W, Cc, 3, s, pad, capi.EXB_F16, out, 1, out_scale=1.0)
        run = lambda p=capi.DwWeights(ctx, d, w, b): capi.dwconv2d(ctx, d, x, p)
        (name, _, _), = kernels_of(run)
        assert "dw3x3_stream_kernel" in name
        y.append(run())
    ctx.sync_check()
    assert torch.equal(y[0].clamp(max=127).to(torch.int8), y[1])
    ref = O.dwconv2d_f32(to_nchw(host(x[-1:].float())), w, b, s, pad, 1)
    np.testing.assert_array_equal(to_nchw(host(y[0][-1:].float())), ref)


# Edges of the streaming pooling kernel: windows hanging over every border of maps smaller than a thread's four columns,
# negative values next to padding (a maximum must not see the fill), channel counts around one CTA's, ceil mode, the
# int8 second output; below 32 channels stride 2 takes the other kernel.
POOL_STREAM_CASES = [
    # N, C, H, W, type, k, s, pad, pad_mode, cip
    (1, 8, 1, 1, 0, 5, 1, 2, 1, 0), (2, 264, 6, 3, 0, 5, 1, 2, 1, 0), (3, 40, 27, 33, 1, 5, 1, 2, 1, 1), (1, 520, 9, 5, 1, 3, 1, 1, 1, 0),
    (2, 24, 5, 7, 0, 3, 1, 1, 1, 0), (2, 32, 2, 2, 0, 3, 2, 1, 1, 0), (1, 72, 37, 41, 0, 3, 2, 1, 0, 0), (2, 64, 30, 9, 1, 3, 2, 1, 0, 1),
    (1, 32, 3, 5, 0, 2, 2, 0, 0, 0), (2, 136, 29, 31, 1, 2, 2, 0, 1, 0), (40, 64, 20, 20, 0, 5, 1, 2, 1, 0), (1, 16, 9, 9, 0, 3, 2, 1, 1, 0),
]


@pytest.mark.parametrize("case", POOL_STREAM_CASES)
def test_pool_stream_edges(ctx, case):
    capi = _capi()
    N, Cc, H, W, type_, k, s, pad, pad_mode, cip = case
    x = f16_round(rng(sum(case)).standard_normal((N, Cc, H, W)) - 3)
    ref = O.pool2d_f32(x, type_, k, s, pad, False, pad_mode, cip)
    q = np.float32(9.0)
    d = capi.make_pool_desc(N, H, W, Cc, type_, k, s, pad, False, pad_mode, cip, capi.EXB_F16, capi.EXB_I8, q)
    y, y2 = capi.pool2d(ctx, d, dev(to_nhwc(x).astype(np.float16)))
    ctx.sync_check()
    y = to_nchw(host(y).astype(np.float32))
    assert y.shape == ref.shape
    if type_ == 0:
        np.testing.assert_array_equal(y, ref)
        np.testing.assert_array_equal(to_nchw(host(y2)), O.requantize_rne(ref, q))
    else:
        np.testing.assert_allclose(y, ref, rtol=1e-3, atol=1e-3)


# A map split over a cluster of CTAs, and channel counts that leave lanes of the last CTA without work.
@pytest.mark.parametrize("type_", [0, 1])
@pytest.mark.parametrize("shape", [(1, 8, 112, 111), (3, 264, 33, 29), (1, 64, 40, 40), (70, 272, 9, 9)])
def test_global_pool_split(ctx, type_, shape):
    test_global_pool(ctx, type_, shape)


def _averages(ctx, capi, x, k, s, pad, pad_mode, cip, dtype, out2_scale=None):
    N, Cc, H, W = x.shape
    d = capi.make_pool_desc(N, H, W, Cc, 1, k, s, pad, False, pad_mode, cip, capi.EXB_F16 if dtype == np.float16 else capi.EXB_F32,
                            *(() if out2_scale is None else (capi.EXB_I8, out2_scale)))
    y, y2 = capi.pool2d(ctx, d, dev(to_nhwc(x).astype(dtype)))
    ctx.sync_check()
    return host(y), None if y2 is None else host(y2)


# Averages of small windows (row stream) against the kernel with a thread per output vector, which an fp32 map takes: small
# integers, so that the sums are exact in any order and only the division is left, with every divisor that the window
# can have at the borders, and infinities, NaN and zeros among the values.
@pytest.mark.parametrize("cip", [0, 1])
@pytest.mark.parametrize("window", [(5, 1, 2, 1), (5, 1, 0, 1), (3, 1, 1, 1), (3, 2, 1, 0), (3, 2, 0, 0), (2, 2, 0, 0), (2, 2, 1, 1)])
def test_pool_stream_average_is_a_division(ctx, window, cip):
    capi = _capi()
    k, s, pad, pad_mode = window
    r = rng(sum(window) + cip)
    x = r.integers(-1000, 1001, (3, 40, 14, 17)).astype(np.float32)
    x[0, :8] = 0
    for v, at in ((np.inf, 8), (-np.inf, 16), (np.nan, 24)):
        x[:, at:at + 8][r.random((3, 8, 14, 17)) < 0.02] = v
    x[1, 8, 3, 3], x[1, 8, 3, 4] = np.inf, -np.inf
    y, _ = _averages(ctx, capi, x, k, s, pad, pad_mode, cip, np.float16)
    ref, _ = _averages(ctx, capi, x, k, s, pad, pad_mode, cip, np.float32)
    assert np.isinf(ref).any() and np.isnan(ref).any()
    np.testing.assert_array_equal(y, ref.astype(np.float16))


# Windows that lie wholly in the padding (ceil mode on odd sides, padding as wide as the window) or hold nothing but NaN:
# the row stream gives what the kernel with a thread per output vector gives, whatever kernel the channel count selects.
@pytest.mark.parametrize("type_", [0, 1])
@pytest.mark.parametrize("case", [(1, 32, 3, 5, 2, 2, 1, 0), (2, 40, 3, 3, 2, 2, 1, 0), (1, 32, 4, 6, 2, 2, 2, 1), (2, 64, 7, 5, 3, 2, 3, 1), (1, 24, 5, 9, 3, 1, 4, 1),
                                  (1, 8, 6, 4, 5, 1, 6, 1), (1, 264, 2, 2, 5, 1, 5, 0)])
def test_pool_stream_windows_without_values(ctx, case, type_):
    import torch
    capi = _capi()
    N, Cc, H, W, k, s, pad, pad_mode = case
    x = rng(sum(case)).integers(-30, -2, (N, Cc, H, W)).astype(np.float32)
    x[:, 1] = np.nan
    x[:, 2, :2] = np.nan
    got = []
    for dt in (np.float16, np.float32):
        d = capi.make_pool_desc(N, H, W, Cc, type_, k, s, pad, False, pad_mode, 0, capi.EXB_F16 if dt == np.float16 else capi.EXB_F32,
                                *((capi.EXB_I8, np.float32(2.5)) if type_ == 0 else ()))
        y, y2 = capi.pool2d(ctx, d, dev(to_nhwc(x).astype(dt)))
        ctx.sync_check()
        got.append((y.to(torch.float16), y2))
    assert not torch.isfinite(got[1][0][..., 0]).all(), "no window without values"
    np.testing.assert_array_equal(host(got[0][0]), host(got[1][0]))
    if type_ == 0:
        np.testing.assert_array_equal(host(got[0][1]), host(got[1][1]))


# The int8 second output of an average is the rounded fp32 average (a value rounded to fp16 first lands on the other side of
# a half in a few per mille): integers whose sums are exact, against the kernel that an fp32 map takes.
@pytest.mark.parametrize("window", [(5, 1, 2, 1), (3, 1, 1, 1), (3, 2, 1, 0), (2, 2, 0, 0)])
def test_pool_stream_average_quantised_from_fp32(ctx, window):
    capi = _capi()
    k, s, pad, pad_mode = window
    x = rng(sum(window)).integers(-1000, 1001, (8, 64, 28, 31)).astype(np.float32)
    x[:, 3][rng(1).random((8, 28, 31)) < 0.05] = np.nan
    scale = np.float32(0.28)
    _, q = _averages(ctx, capi, x, k, s, pad, pad_mode, 0, np.float16, scale)
    _, ref = _averages(ctx, capi, x, k, s, pad, pad_mode, 0, np.float32, scale)
    np.testing.assert_array_equal(q, ref)


# More tiles than the row stream counts (2^30 images of one pixel, 17 GB each way): the kernels for other windows take them.
@pytest.mark.parametrize("op", ["dwconv", "pool"])
def test_row_stream_tile_limit(ctx, op):
    import torch
    capi = _capi()
    N, Cc = (1 << 30) + 5, 8
    if torch.cuda.mem_get_info()[0] < 48 << 30:
        pytest.skip("needs 48 GB of device memory")
    x = torch.empty((N, 1, 1, Cc), device="cuda", dtype=torch.float16).fill_(2)
    x[7], x[-1] = 3, -5
    if op == "dwconv":
        w = np.zeros((Cc, 1, 3, 3), np.float32)
        w[:, 0, 1, 1] = 1.5
        d = capi.make_dw_desc(N, 1, 1, Cc, 3, 1, 1, capi.EXB_F16, capi.EXB_F16, 0)
        y = capi.dwconv2d(ctx, d, x, capi.DwWeights(ctx, d, w, np.zeros(Cc, np.float32)))
        k = 1.5
    else:
        y, _ = capi.pool2d(ctx, capi.make_pool_desc(N, 1, 1, Cc, 0, 5, 1, 2, False, 1, 0, capi.EXB_F16), x)
        k = 1.0
    ctx.sync_check()
    for i, v in ((0, 2), (7, 3), (8, 2), (1 << 29, 2), (N - 2, 2), (N - 1, -5)):
        assert (y[i].float() == v * k).all(), i
    del x, y
    torch.cuda.empty_cache()


# The shapes of the edge tests run in the kernels they are there for (below 32 channels stride 2 takes the other one).
def test_stream_cases_take_the_stream_kernels(ctx):
    import torch
    capi = _capi()
    for N, Cc, H, W, s, pad, act in DW_STREAM_CASES:
        d = capi.make_dw_desc(N, H, W, Cc, 3, s, pad, capi.EXB_F16, capi.EXB_F16, act)
        w = capi.DwWeights(ctx, d, np.zeros((Cc, 1, 3, 3), np.float32), np.zeros(Cc, np.float32))
        x = torch.zeros((N, H, W, Cc), device="cuda", dtype=torch.float16)
        names = [n for n, _, _ in kernels_of(lambda: capi.dwconv2d(ctx, d, x, w))]
        assert any("dw3x3_stream_kernel" in n for n in names), ((N, Cc, H, W, s), names)
    for N, Cc, H, W, type_, k, s, pad, pad_mode, cip in POOL_STREAM_CASES:
        d = capi.make_pool_desc(N, H, W, Cc, type_, k, s, pad, False, pad_mode, cip, capi.EXB_F16)
        x = torch.zeros((N, H, W, Cc), device="cuda", dtype=torch.float16)
        names = [n for n, _, _ in kernels_of(lambda: capi.pool2d(ctx, d, x))]
        assert any("pool_stream_kernel" in n for n in names) == (s == 1 or Cc >= 32), ((N, Cc, H, W, k, s), names)
    ctx.sync_check()
