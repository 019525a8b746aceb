"""Parity of the dense convolution (tcgen05 implicit GEMM and the direct kernel) against the CPU
oracle: int32 accumulators bit-exact, dequantised fp32 bit-exact, requantised int8 bit-exact
against the oracle's half-even rule and within 1 LSB of the reference's half-away rule, fp16
within 1e-2 relative of the fp32 result."""
import re

import numpy as np
import pytest

from oracle import exb_oracle as O
from tests.util import kernels_of, dev, host, rng, f16_round, to_nhwc, to_nchw, assert_close_f16, quant_weights

pytestmark = pytest.mark.gpu


def _capi():
    from excalibur_b200 import capi
    return capi


def run_conv_i8(ctx, xq, wq, bias, ws, fs, stride, pad, out_dtype, act=0, impl=0, res=None, out_scale=1.0,
                out2_dtype=-1, out2_scale=1.0, group=1):
    capi = _capi()
    N, Cin, H, W = xq.shape
    Cout, _, kh, kw = wq.shape
    d = capi.make_conv_desc(N, H, W, Cin, Cout, (kh, kw), stride, pad, capi.EXB_I8, out_dtype, out2_dtype,
                            res is not None, act, out_scale, out2_scale, group=group, impl=impl)
    wp = capi.ConvWeights(ctx, d, wq, bias, ws, fs)
    resd = dev(to_nhwc(res).astype(np.float16)) if res is not None else None
    y, y2 = capi.conv2d(ctx, d, dev(to_nhwc(xq)), wp, resd)
    ctx.sync_check()
    return (to_nchw(host(y)), to_nchw(host(y2)) if y2 is not None else None,
            capi.lib().exb_conv2d_uses_tensor_cores(d))


I8_CASES = [
    # N, Cin, H, W, Cout, k, stride, pad
    (1, 64, 8, 8, 64, 3, 1, 1),
    (2, 64, 56, 56, 64, 3, 1, 1),       # ResNet stage 1
    (3, 64, 56, 56, 128, 3, 2, 1),      # stage 2 entry
    (3, 64, 56, 56, 128, 1, 2, 0),      # projection shortcut
    (2, 128, 28, 28, 128, 3, 1, 1),
    (5, 256, 14, 14, 256, 3, 1, 1),
    (20, 512, 7, 7, 512, 3, 1, 1),      # box spans 18 images + ragged tail
    (2, 32, 13, 11, 48, 3, 1, 1),       # odd sizes, 32-byte K blocks, Cout not multiple of 32
    (2, 96, 9, 9, 40, 1, 1, 0),         # 1x1, 32-byte K blocks, ragged Cout
    (1, 128, 15, 15, 64, 3, 2, 1),      # odd input, stride 2
    (1, 64, 12, 12, 320, 3, 1, 1),      # two Cout tiles
    (2, 64, 10, 10, 32, 5, 1, 2),       # 5x5
    (1, 32, 9, 9, 16, 3, 2, 0),         # stride 2 without padding
    (3, 256, 10, 13, 128, 3, 1, 1),     # row-box loop: two channel blocks per kernel row, weights streamed, ragged width
    (5, 128, 6, 5, 64, 3, 1, 1),        # row-box loop: map narrower than the 8-pixel tile, several images per tile
    (1, 192, 12, 12, 64, 2, 1, 0),      # row-box loop with two taps per row (2x2 kernel, no padding), three channel blocks
    (9, 128, 12, 12, 128, 3, 1, 1),     # row-box loop on CTA pairs (resident weights, halves per CTA), odd number of image groups
    (7, 256, 14, 14, 256, 3, 1, 1),     # tap loop on CTA pairs, odd number of image groups (last pair half empty)
]


@pytest.mark.parametrize("impl", [0, 1], ids=["tc", "direct"])
@pytest.mark.parametrize("case", I8_CASES)
def test_conv_i8_accumulators_bit_exact(ctx, case, impl):
    capi = _capi()
    N, Cin, H, W, Cout, k, stride, pad = case
    r = rng(sum(case))
    xq = r.integers(-128, 128, (N, Cin, H, W)).astype(np.int8)
    wq = r.integers(-127, 128, (Cout, Cin, k, k)).astype(np.int8)
    ref = O.conv2d_i8_acc(xq, wq, stride, pad)
    y, _, tc = run_conv_i8(ctx, xq, wq, None, np.ones(Cout, np.float32), 1.0, stride, pad, capi.EXB_I32, impl=impl)
    assert tc == (1 if impl == 0 else 0)
    assert y.shape == ref.shape
    np.testing.assert_array_equal(y, ref)


@pytest.mark.parametrize("case", I8_CASES[:6])
def test_conv_i8_dequant_and_requant(ctx, case):
    """The fused epilogue: fp32 result equals the reference formula acc*1/(ws*fs)+bias bit for bit;
    the int8 result equals the half-even requantisation of it, and is within 1 LSB of quantising
    with the reference's half-away rule."""
    capi = _capi()
    N, Cin, H, W, Cout, k, stride, pad = case
    r = rng(sum(case) + 1)
    x = r.uniform(-1, 1, (N, Cin, H, W)).astype(np.float32)
    w = (r.standard_normal((Cout, Cin, k, k)) * np.sqrt(2.0 / (Cin * k * k))).astype(np.float32)
    b = (r.standard_normal(Cout) * 0.01).astype(np.float32)
    wq, ws = quant_weights(w)
    fs = np.float32(127.0 / np.abs(x).max())
    xq = O.quantize_f32_i8(x, [fs])
    ref = O.conv2d_i8(x, wq, b, ws, fs, stride, pad, act=1)          # the reference's forward_cpu_i8
    y, _, _ = run_conv_i8(ctx, xq, wq, b, ws, fs, stride, pad, capi.EXB_F32, act=1)
    np.testing.assert_array_equal(y, ref)
    nxt = np.float32(127.0 / max(float(ref.max()), 1e-6))
    q, h16, _ = run_conv_i8(ctx, xq, wq, b, ws, fs, stride, pad, capi.EXB_I8, act=1, out_scale=nxt,
                            out2_dtype=capi.EXB_F16)
    np.testing.assert_array_equal(q, O.requantize_rne(ref, nxt))
    assert np.abs(q.astype(np.int32) - O.quantize_f32_i8(ref, [nxt]).astype(np.int32)).max() <= 1
    np.testing.assert_array_equal(h16.astype(np.float32), f16_round(ref))


def test_conv_i8_residual_relu_dual_output(ctx):
    """Second conv of a basic block: conv + skip (fp16) + ReLU, written as fp16 and as int8."""
    capi = _capi()
    N, Cc, H, W = 2, 64, 28, 28
    r = rng(4242)
    x = r.uniform(-1, 1, (N, Cc, H, W)).astype(np.float32)
    w = (r.standard_normal((Cc, Cc, 3, 3)) * np.sqrt(2.0 / (Cc * 9))).astype(np.float32)
    b = (r.standard_normal(Cc) * 0.01).astype(np.float32)
    skip = f16_round(r.uniform(-1, 1, (N, Cc, H, W)))
    wq, ws = quant_weights(w)
    fs = np.float32(127.0 / np.abs(x).max())
    xq = O.quantize_f32_i8(x, [fs])
    v = O.activation(O.conv2d_i8(x, wq, b, ws, fs, 1, 1, act=0) + skip, 1)
    nxt = np.float32(127.0 / v.max())
    y16, q, _ = run_conv_i8(ctx, xq, wq, b, ws, fs, 1, 1, capi.EXB_F16, act=1, res=skip,
                            out2_dtype=capi.EXB_I8, out2_scale=nxt)
    np.testing.assert_array_equal(y16.astype(np.float32), f16_round(v))
    np.testing.assert_array_equal(q, O.requantize_rne(v, nxt))


F16_CASES = [
    (1, 64, 56, 56, 64, 3, 1, 1),       # the single-layer benchmark configuration's shape
    (2, 16, 37, 41, 64, 7, 2, 3),       # stem-like (3 channels padded to 16)
    (2, 64, 28, 28, 128, 3, 2, 1),
    (2, 128, 14, 14, 256, 1, 1, 0),
    (4, 512, 7, 7, 512, 3, 1, 1),
    (1, 32, 40, 40, 255, 1, 1, 0),      # detect head width
    (2, 16, 30, 30, 32, 6, 2, 2),       # 6x6/2 stem
    (2, 32, 21, 19, 32, 3, 1, 1),       # row-box loop on 64-byte K rows, ragged map
    (2, 64, 11, 9, 64, 3, 1, 1),        # row-box loop, weights streamed with two CTAs per SM (73 KB slice)
    (1, 128, 12, 12, 64, 5, 1, 2),      # row-box loop with five taps per row, two channel blocks
    (9, 64, 12, 12, 128, 3, 1, 1),      # row-box loop on CTA pairs, fp16
    (3, 128, 14, 14, 256, 3, 2, 1),     # stride-2 tap loop on CTA pairs, fp16
]


@pytest.mark.parametrize("impl", [0, 1], ids=["tc", "direct"])
@pytest.mark.parametrize("case", F16_CASES)
def test_conv_f16(ctx, case, impl):
    capi = _capi()
    N, Cin, H, W, Cout, k, stride, pad = case
    r = rng(sum(case) + 7)
    x = f16_round(r.uniform(-1, 1, (N, Cin, H, W)))
    w = f16_round(r.standard_normal((Cout, Cin, k, k)) * np.sqrt(2.0 / (Cin * k * k)))
    b = (r.standard_normal(Cout) * 0.01).astype(np.float32)
    ref = O.conv2d_f32(x, w, b, stride, pad, act=1)
    d = capi.make_conv_desc(N, H, W, Cin, Cout, k, stride, pad, capi.EXB_F16, capi.EXB_F32, act=1, impl=impl)
    wp = capi.ConvWeights(ctx, d, w, b)
    y, _ = capi.conv2d(ctx, d, dev(to_nhwc(x).astype(np.float16)), wp)
    ctx.sync_check()
    assert capi.lib().exb_conv2d_uses_tensor_cores(d) == (1 if impl == 0 else 0)
    y = to_nchw(host(y))
    # fp32 accumulation of exactly representable products: only the summation order differs
    np.testing.assert_allclose(y, ref, rtol=1e-4, atol=1e-4)
    d16 = capi.make_conv_desc(N, H, W, Cin, Cout, k, stride, pad, capi.EXB_F16, capi.EXB_F16, act=1, impl=impl)
    y16, _ = capi.conv2d(ctx, d16, dev(to_nhwc(x).astype(np.float16)), wp)
    ctx.sync_check()
    assert_close_f16(to_nchw(host(y16).astype(np.float32)), ref, what="fp16 conv")


def test_conv_f16_config1_against_unrounded_fp32(ctx):
    """The single-layer benchmark configuration: fp32 data, fp16 kernel, 1e-2 relative of the fp32 result."""
    capi = _capi()
    r = rng(1000)
    x = r.uniform(-1, 1, (1, 64, 56, 56)).astype(np.float32)
    w = (r.standard_normal((64, 64, 3, 3)) * np.sqrt(2.0 / 576)).astype(np.float32)
    b = (r.standard_normal(64) * 0.01).astype(np.float32)
    ref = O.conv2d_f32(x, w, b, 1, 1, act=1)
    d = capi.make_conv_desc(1, 56, 56, 64, 64, 3, 1, 1, capi.EXB_F16, capi.EXB_F16, act=1)
    wp = capi.ConvWeights(ctx, d, w, b)
    xh = capi.nchw_f32_to_nhwc(ctx, dev(x), capi.EXB_F16)
    y, _ = capi.conv2d(ctx, d, xh, wp)
    out = host(capi.nhwc_to_nchw_f32(ctx, y))
    ctx.sync_check()
    assert_close_f16(out, ref, what="config 1")


def test_conv_silu_and_padded_channels(ctx):
    capi = _capi()
    N, Cin, H, W, Cout = 2, 24, 20, 20, 40
    cin_s, cout_s = 32, 48
    r = rng(31)
    x = f16_round(r.uniform(-1, 1, (N, Cin, H, W)))
    w = f16_round(r.standard_normal((Cout, Cin, 3, 3)) * 0.1)
    b = (r.standard_normal(Cout) * 0.1).astype(np.float32)
    ref = O.conv2d_f32(x, w, b, 1, 1, act=O.ACT_SILU)
    d = capi.make_conv_desc(N, H, W, Cin, Cout, 3, 1, 1, capi.EXB_F16, capi.EXB_F16, act=capi.ACT_SILU,
                            cin_stride=cin_s, cout_stride=cout_s)
    wp = capi.ConvWeights(ctx, d, w, b)
    y, _ = capi.conv2d(ctx, d, dev(to_nhwc(x, cin_s).astype(np.float16)), wp)
    ctx.sync_check()
    yh = host(y).astype(np.float32)
    assert not yh[..., Cout:].any(), "padding channels must be written as zero"
    assert_close_f16(to_nchw(yh, Cout), ref, what="silu")


def test_conv_grouped_direct(ctx):
    capi = _capi()
    N, Cin, H, W, Cout, g = 2, 16, 9, 9, 24, 4
    r = rng(8)
    x = f16_round(r.uniform(-1, 1, (N, Cin, H, W)))
    w = f16_round(r.standard_normal((Cout, Cin // g, 3, 3)) * 0.2)
    ref = O.conv2d_f32(x, w, None, 1, 1, group=g)
    d = capi.make_conv_desc(N, H, W, Cin, Cout, 3, 1, 1, capi.EXB_F16, capi.EXB_F32, group=g)
    assert capi.lib().exb_conv2d_uses_tensor_cores(d) == 0
    wp = capi.ConvWeights(ctx, d, w, None)
    y, _ = capi.conv2d(ctx, d, dev(to_nhwc(x).astype(np.float16)), wp)
    ctx.sync_check()
    np.testing.assert_allclose(to_nchw(host(y)), ref, rtol=1e-4, atol=1e-4)


def test_conv_full_size_tc_equals_direct(ctx):
    """Batch-256 stage-1 layer: the tensor-core kernel against the direct kernel on the device, bit for bit over the
    whole batch, and two images of that same launch against the CPU oracle."""
    capi = _capi()
    import torch
    N, Cc, H, W = 256, 64, 56, 56
    g = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randint(-128, 128, (N, H, W, Cc), generator=g, device="cuda", dtype=torch.int32).to(torch.int8)
    r = rng(55)
    wq = r.integers(-127, 128, (Cc, Cc, 3, 3)).astype(np.int8)
    outs = []
    for impl in (0, 1):
        d = capi.make_conv_desc(N, H, W, Cc, Cc, 3, 1, 1, capi.EXB_I8, capi.EXB_I32, impl=impl)
        wp = capi.ConvWeights(ctx, d, wq, None, np.ones(Cc, np.float32), 1.0)
        y, _ = capi.conv2d(ctx, d, x, wp)
        ctx.sync_check()
        outs.append(y)
    assert torch.equal(outs[0], outs[1])
    # two images of the same launch (the first and the last) against the CPU oracle's accumulators
    for n in (0, N - 1):
        xn = to_nchw(host(x[n:n + 1]))
        ref = O.conv2d_i8_acc(xn, wq, 1, 1)
        np.testing.assert_array_equal(to_nchw(host(outs[0][n:n + 1])), ref)
    # linearity: conv(2x) == 2*conv(x) on the accumulators
    d = capi.make_conv_desc(N, H, W, Cc, Cc, 3, 1, 1, capi.EXB_I8, capi.EXB_I32)
    wp = capi.ConvWeights(ctx, d, wq, None, np.ones(Cc, np.float32), 1.0)
    xh = (x.to(torch.int32) // 2).to(torch.int8)
    y1, _ = capi.conv2d(ctx, d, xh, wp)
    y2, _ = capi.conv2d(ctx, d, (xh.to(torch.int32) * 2).to(torch.int8), wp)
    ctx.sync_check()
    assert torch.equal(y1 * 2, y2)


def test_conv_empty_batch_and_errors(ctx):
    capi = _capi()
    d = capi.make_conv_desc(0, 8, 8, 64, 64, 3, 1, 1, capi.EXB_I8, capi.EXB_I32)
    wq = np.zeros((64, 64, 3, 3), np.int8)
    wp = capi.ConvWeights(ctx, d, wq, None, np.ones(64, np.float32), 1.0)
    assert capi.lib().exb_conv2d_fwd(ctx.handle, d, None, wp.handle, None, None, None, None) == 0
    bad = capi.make_conv_desc(1, 2, 2, 64, 64, 3, 1, 0, capi.EXB_I8, capi.EXB_I32)   # window > input
    assert capi.lib().exb_conv2d_fwd(ctx.handle, bad, None, wp.handle, None, None, None, None) == capi.EXB_ERR_BAD_ARG
    assert "window" in capi.last_error()


STEM_CASES = [
    # N, H, W, Cout, k, stride, pad, w_pad
    (2, 64, 64, 64, 7, 2, 3, 4),      # ResNet stem
    (3, 37, 41, 32, 3, 2, 1, 4),      # MobileNet stem, odd sizes
    (2, 48, 40, 32, 6, 2, 2, 4),      # YOLOv5 stem
    (1, 224, 224, 64, 7, 2, 3, 4),
]


@pytest.mark.parametrize("impl", [0, 1], ids=["tc", "direct"])
@pytest.mark.parametrize("case", STEM_CASES)
def test_stem_conv_folded_rows(ctx, case, impl):
    """3-channel stem: fp32 NCHW image -> padded NHWC4 fp16 rows -> conv with kw taps folded into K."""
    capi = _capi()
    N, H, W, Cout, k, stride, pad, w_pad = case
    r = rng(sum(case))
    x = r.uniform(0, 1, (N, 3, H, W)).astype(np.float32)
    w = f16_round(r.standard_normal((Cout, 3, k, k)) * np.sqrt(2.0 / (3 * k * k)))
    b = (r.standard_normal(Cout) * 0.01).astype(np.float32)
    ref = O.conv2d_f32(f16_round(x), w, b, stride, pad, act=1)
    w_pitch = (W + w_pad + 8 + 7) // 8 * 8
    xp = capi.nchw_f32_to_nhwc_padded(ctx, dev(x), capi.EXB_F16, 4, w_pad, w_pitch)
    xh = host(xp).astype(np.float32)
    np.testing.assert_array_equal(xh[:, :, w_pad:w_pad + W, :3], f16_round(np.transpose(x, (0, 2, 3, 1))))
    assert not xh[:, :, :w_pad].any() and not xh[:, :, w_pad + W:].any() and not xh[..., 3].any()
    d = capi.make_conv_desc(N, H, W, 3, Cout, k, stride, pad, capi.EXB_F16, capi.EXB_F32, act=1, cin_stride=4,
                            impl=impl, x_w_pitch=w_pitch, x_w_pad=w_pad)
    assert capi.lib().exb_conv2d_uses_tensor_cores(d) == (1 if impl == 0 else 0)
    wp = capi.ConvWeights(ctx, d, w, b)
    y, _ = capi.conv2d(ctx, d, xp, wp)
    ctx.sync_check()
    np.testing.assert_allclose(to_nchw(host(y)), ref, rtol=1e-4, atol=1e-4)


POOL_STEM_CASES = [
    # N, H, W, k, pad
    (2, 64, 64, 7, 3),
    (3, 37, 41, 7, 3),      # odd conv output (19 x 21) -> pooled 10 x 11, ragged last tiles
    (2, 48, 40, 6, 2),      # YOLO-style 6x6/2 stem
    (1, 224, 224, 7, 3),
    (2, 30, 26, 5, 2),
]


@pytest.mark.parametrize("case", POOL_STEM_CASES)
@pytest.mark.parametrize("with_i8", [False, True], ids=["f16", "f16+i8"])
def test_stem_conv_with_fused_max_pool(ctx, case, with_i8):
    """Stem conv + ReLU + 3x3/2 pad-1 max pooling in one kernel equals conv -> fp16 -> pool of the
    oracle (bit-exact given the conv's fp16 result: max of rounded values, then the int8 copy)."""
    capi = _capi()
    N, H, W, k, pad = case
    r = rng(sum(case) + 7)
    x = r.uniform(0, 1, (N, 3, H, W)).astype(np.float32)
    w = f16_round(r.standard_normal((64, 3, k, k)) * np.sqrt(2.0 / (3 * k * k)))
    b = (r.standard_normal(64) * 0.1).astype(np.float32)
    w_pad = 4
    w_pitch = (W + w_pad + 8 + 7) // 8 * 8
    xp = capi.nchw_f32_to_nhwc_padded(ctx, dev(x), capi.EXB_F16, 4, w_pad, w_pitch)
    q = 25.0
    kw = dict(act=1, cin_stride=4, x_w_pitch=w_pitch, x_w_pad=w_pad)
    d0 = capi.make_conv_desc(N, H, W, 3, 64, k, 2, pad, capi.EXB_F16, capi.EXB_F16, **kw)
    d1 = capi.make_conv_desc(N, H, W, 3, 64, k, 2, pad, capi.EXB_F16, capi.EXB_F16,
                             capi.EXB_I8 if with_i8 else -1, out2_scale=q, fuse_pool=1, **kw)
    assert capi.lib().exb_conv2d_pool_fusable(d0) == 1
    wp = capi.ConvWeights(ctx, d0, w, b)
    y0, _ = capi.conv2d(ctx, d0, xp, wp)                     # the plain kernel's fp16 conv output
    y1, y2 = capi.conv2d(ctx, d1, xp, wp)
    ctx.sync_check()
    conv16 = to_nchw(host(y0).astype(np.float32))
    ref_conv = O.conv2d_f32(f16_round(x), w, b, 2, pad, act=1)
    np.testing.assert_allclose(conv16, ref_conv, rtol=2e-3, atol=2e-3)
    ref_pool = O.pool2d_f32(conv16, 0, 3, 2, 1)
    got = to_nchw(host(y1).astype(np.float32))
    assert got.shape == ref_pool.shape
    np.testing.assert_array_equal(got, ref_pool)
    if with_i8:
        np.testing.assert_array_equal(to_nchw(host(y2).astype(np.float32)), O.requantize_rne(ref_pool, q))


def test_fused_max_pool_is_refused_where_it_cannot_run(ctx):
    capi = _capi()
    d = capi.make_conv_desc(1, 16, 16, 32, 64, 3, 1, 1, capi.EXB_I8, capi.EXB_F16, act=1)
    assert capi.lib().exb_conv2d_pool_fusable(d) == 0
    d.fuse_pool = 1
    w = capi.ConvWeights(ctx, d, np.zeros((64, 32, 3, 3), np.int8), np.zeros(64, np.float32), np.ones(64, np.float32), 1.0)
    x = dev(np.zeros((1, 16, 16, 32), np.int8))
    with pytest.raises(capi.ExbError):
        capi.conv2d(ctx, d, x, w)


RES_DUAL_CASES = [
    # N, Cin, H, W, Cout, k, stride, pad
    (2, 64, 56, 56, 64, 3, 1, 1),       # two CTAs per SM, one 64-channel block
    (3, 128, 28, 28, 128, 3, 1, 1),     # two blocks
    (5, 256, 14, 14, 256, 3, 1, 1),     # one CTA per SM, the two halves of a lane quarter on two warps
    (20, 512, 7, 7, 512, 3, 1, 1),      # two Cout tiles of 256, 7x1x18 boxes with a ragged tail
    (3, 64, 56, 56, 128, 1, 2, 0),      # projection shortcut (fp16 output only)
    (2, 32, 13, 11, 48, 3, 1, 1),       # ragged tiles, 48 channels: the thread-per-pixel epilogue
    (1, 64, 12, 12, 320, 3, 1, 1),      # two Cout tiles of 160 channels: thread-per-pixel epilogue
    (2, 64, 9, 7, 192, 3, 1, 1),        # three blocks, tiles ragged in both directions
]


@pytest.mark.parametrize("case", RES_DUAL_CASES)
def test_conv_i8_residual_dual_output_shapes(ctx, case):
    """conv + fp16 skip + ReLU written as fp16 and int8 (the second convolution of a residual block) on every tile /
    channel-block configuration of the tensor-core kernel's two epilogues, against the CPU oracle, bit for bit."""
    capi = _capi()
    N, Cin, H, W, Cout, k, stride, pad = case
    r = rng(sum(case) + 11)
    x = r.uniform(-1, 1, (N, Cin, H, W)).astype(np.float32)
    w = (r.standard_normal((Cout, Cin, k, k)) * np.sqrt(2.0 / (Cin * k * k))).astype(np.float32)
    b = (r.standard_normal(Cout) * 0.01).astype(np.float32)
    wq, ws = quant_weights(w)
    fs = np.float32(127.0 / np.abs(x).max())
    xq = O.quantize_f32_i8(x, [fs])
    pre = O.conv2d_i8(x, wq, b, ws, fs, stride, pad, act=0)
    with_res = k == 3
    skip = f16_round(r.uniform(-1, 1, pre.shape)) if with_res else None
    v = O.activation(pre + skip, 1) if with_res else pre
    nxt = np.float32(127.0 / max(float(np.abs(v).max()), 1e-6))
    if with_res:
        y16, q, tc = run_conv_i8(ctx, xq, wq, b, ws, fs, stride, pad, capi.EXB_F16, act=1, res=skip,
                                 out2_dtype=capi.EXB_I8, out2_scale=nxt)
        np.testing.assert_array_equal(q, O.requantize_rne(v, nxt))
    else:
        y16, _, tc = run_conv_i8(ctx, xq, wq, b, ws, fs, stride, pad, capi.EXB_F16)
    assert tc == 1
    np.testing.assert_array_equal(y16.astype(np.float32), f16_round(v))
    # int8 first, fp16 second (the order the first convolution of the next block's producer uses)
    q2, h2, _ = run_conv_i8(ctx, xq, wq, b, ws, fs, stride, pad, capi.EXB_I8, act=1 if with_res else 0, res=skip,
                            out_scale=nxt, out2_dtype=capi.EXB_F16)
    np.testing.assert_array_equal(q2, O.requantize_rne(v, nxt))
    np.testing.assert_array_equal(h2.astype(np.float32), f16_round(v))


# The kernel for problems of few tiles: reductions of fewer K blocks than CTAs, K blocks that do not divide evenly, more of
# them than the ring holds, channel counts that end inside a tile (multiples of 8), both strides, one pixel, maps
# narrower than a box, every output form.  int8 equals the persistent kernel bit for bit, fp16 the oracle.
SPLIT_CASES = [
    # N, Cin, H, W, Cout, k, stride
    (1, 512, 7, 7, 512, 3, 1), (1, 32, 1, 1, 8, 1, 1), (1, 64, 9, 5, 72, 3, 2), (2, 96, 14, 13, 40, 3, 1), (1, 512, 1, 1, 1000, 1, 1),
    (3, 160, 7, 6, 264, 1, 1), (1, 256, 15, 15, 64, 3, 2), (1, 64, 56, 56, 64, 3, 1), (1, 1024, 4, 4, 32, 3, 1), (5, 32, 20, 3, 16, 5, 1),
]


@pytest.mark.parametrize("case", SPLIT_CASES)
def test_conv_split_kernel(ctx, case):
    import torch
    capi = _capi()
    N, Cin, H, W, Cout, k, s = case
    r = rng(sum(case) + 3)
    xq = r.integers(-128, 128, (N, H, W, Cin)).astype(np.int8)
    wq = r.integers(-127, 128, (Cout, Cin, k, k)).astype(np.int8)
    b = r.standard_normal(Cout).astype(np.float32)
    ws = r.uniform(500, 900, Cout).astype(np.float32)
    got = {}
    for impl in (0, 2):
        for out, out2, res in ((capi.EXB_I8, -1, False), (capi.EXB_F16, capi.EXB_I8, True), (capi.EXB_F32, -1, False)):
            d = capi.make_conv_desc(N, H, W, Cin, Cout, k, s, k // 2, capi.EXB_I8, out, out2, res=res, act=1, out_scale=9.0, out2_scale=9.0,
                                    impl=impl)
            oh, ow = capi.conv_out_dims(d)
            skip = dev(rng(5).standard_normal((N, oh, ow, Cout)).astype(np.float16)) if res else None
            ys = capi.conv2d(ctx, d, dev(xq), capi.ConvWeights(ctx, d, wq, b, ws, 40.0), residual=skip)
            ctx.sync_check()
            for i, y in enumerate(ys):
                if y is not None:
                    got.setdefault((out, i), []).append(y)
    for key, (a, c) in got.items():
        assert torch.equal(a, c), key
    x = f16_round(r.uniform(-1, 1, (N, Cin, H, W)))
    w = f16_round(r.standard_normal((Cout, Cin, k, k)) * np.sqrt(2.0 / (Cin * k * k)))
    ref = O.conv2d_f32(x, w, b, s, k // 2, act=1)
    d = capi.make_conv_desc(N, H, W, Cin, Cout, k, s, k // 2, capi.EXB_F16, capi.EXB_F32, act=1)
    y, _ = capi.conv2d(ctx, d, dev(to_nhwc(x).astype(np.float16)), capi.ConvWeights(ctx, d, w, b))
    ctx.sync_check()
    np.testing.assert_allclose(to_nchw(host(y)), ref, rtol=1e-4, atol=1e-4)


# The persistent kernel on the small shapes of the tests above, which the automatic choice now gives to the split kernel;
# channel counts that are multiples of 8 but not of 16 go through its two-halves epilogue.
@pytest.mark.parametrize("case", I8_CASES + [(2, 96, 14, 13, 40, 3, 1, 1), (3, 64, 20, 20, 408, 1, 1, 0)])
def test_conv_persistent_kernel_small(ctx, case):
    capi = _capi()
    N, Cin, H, W, Cout, k, stride, pad = case
    r = rng(sum(case) + 21)
    xq = r.integers(-128, 128, (N, Cin, H, W)).astype(np.int8)
    wq = r.integers(-127, 128, (Cout, Cin, k, k)).astype(np.int8)
    acc = O.conv2d_i8_acc(xq, wq, stride, pad).astype(np.float32)
    y, _, _ = run_conv_i8(ctx, xq, wq, None, np.ones(Cout, np.float32), 1.0, stride, pad, capi.EXB_F32, act=1, impl=2)
    np.testing.assert_array_equal(y, np.maximum(acc, 0))
    q, _, _ = run_conv_i8(ctx, xq, wq, None, np.ones(Cout, np.float32), 1.0, stride, pad, capi.EXB_I8, act=1, out_scale=np.float32(1e-3), impl=2)
    np.testing.assert_array_equal(q, O.requantize_rne(np.maximum(acc, 0), np.float32(1e-3)))


# CTA pairs of the persistent kernel: along the images (odd group counts) and, with one image, along the rows (odd tile
# rows); row-box and tap loops, both epilogues, two N tiles.  Integer values, so that every path is exact.
PAIR_CASES = [(3, 64, 115, 113, 64, 3, 1, "f16"), (1, 64, 200, 210, 64, 3, 1, "f16"),
              (1, 64, 401, 400, 64, 3, 2, "f16"), (3, 64, 230, 226, 128, 3, 2, "f16"),
              (1, 128, 401, 400, 96, 3, 2, "i8"), (2, 128, 300, 270, 64, 3, 2, "i8"),
              # more than 128 channels
              (5, 1184, 9, 7, 160, 1, 1, "i8"), (1, 160, 37, 9, 192, 3, 1, "i8"), (5, 608, 9, 7, 192, 1, 1, "f16"),
              (3, 160, 9, 9, 320, 3, 1, "i8"), (1, 96, 37, 9, 304, 3, 1, "f16"), (3, 96, 9, 9, 304, 3, 1, "f16"),
              (2, 128, 9, 9, 384, 3, 1, "f16"), (3, 256, 7, 7, 512, 3, 1, "i8")]
# N tiles of 128 channels or fewer, single
SINGLE_CASES = [(5, 512, 9, 7, 160, 1, 1, "i8"), (5, 256, 9, 7, 192, 1, 1, "f16"), (3, 64, 9, 9, 320, 3, 1, "i8"), (1, 64, 37, 9, 320, 3, 1, "f16"),
                (2, 128, 9, 9, 272, 1, 1, "i8"), (3, 64, 17, 9, 408, 3, 1, "f16")]


@pytest.mark.parametrize("case", PAIR_CASES + SINGLE_CASES)
def test_conv_pairs(ctx, case):
    capi = _capi()
    N, Cin, H, W, Cout, k, s, dtype = case
    r = rng(sum(case[:7]) + 22)
    xq = r.integers(-8, 9, (N, Cin, H, W)).astype(np.int8)
    wq = r.integers(-8, 9, (Cout, Cin, k, k)).astype(np.int8)
    ref = O.conv2d_i8_acc(xq, wq, s, k // 2)
    if dtype == "i8":
        q, _, _ = run_conv_i8(ctx, xq, wq, None, np.ones(Cout, np.float32), 1.0, s, k // 2, capi.EXB_I8, out_scale=np.float32(0.03), impl=2)
        np.testing.assert_array_equal(q, O.requantize_rne(ref.astype(np.float32), np.float32(0.03)))
    d = capi.make_conv_desc(N, H, W, Cin, Cout, k, s, k // 2, capi.EXB_I8 if dtype == "i8" else capi.EXB_F16, capi.EXB_F32, impl=2)
    if dtype == "i8":
        p = capi.ConvWeights(ctx, d, wq, None, np.ones(Cout, np.float32), 1.0)
    else:
        p = capi.ConvWeights(ctx, d, wq.astype(np.float32), np.zeros(Cout, np.float32))
    y, _ = capi.conv2d(ctx, d, dev(to_nhwc(xq).astype(np.int8 if dtype == "i8" else np.float16)), p)
    ctx.sync_check()
    np.testing.assert_array_equal(to_nchw(host(y)), ref.astype(np.float32))


# Residual read through a nearest resize by 2: one and several N tiles of the persistent kernel, the split kernel.
@pytest.mark.parametrize("case", [(2, 64, 30, 46, 256, "f16", 2), (1, 64, 16, 10, 32, "f16", 2), (2, 64, 14, 12, 384, "i8", 2), (4, 512, 16, 8, 512, "f16", 2),
                                  (3, 128, 8, 6, 64, "i8", 0), (1, 256, 14, 14, 96, "f16", 0), (300, 64, 14, 14, 128, "i8", 2)])
def test_conv_half_resolution_residual(ctx, case):
    capi = _capi()
    N, Cin, H, W, Cout, dtype, impl = case
    r = rng(sum(case[:5]) + 23)
    xq = r.integers(-4, 5, (N, Cin, H, W)).astype(np.int8)
    wq = r.integers(-3, 4, (Cout, Cin, 1, 1)).astype(np.int8)
    res = r.integers(-64, 65, (N, Cout, H // 2, W // 2)).astype(np.float32)
    ref = O.conv2d_i8_acc(xq, wq, 1, 0).astype(np.float32) + np.repeat(np.repeat(res, 2, 2), 2, 3)
    d = capi.make_conv_desc(N, H, W, Cin, Cout, 1, 1, 0, capi.EXB_I8 if dtype == "i8" else capi.EXB_F16, capi.EXB_F32, res=True, impl=impl)
    d.res_half = 1
    p = (capi.ConvWeights(ctx, d, wq, None, np.ones(Cout, np.float32), 1.0) if dtype == "i8"
         else capi.ConvWeights(ctx, d, wq.astype(np.float32), np.zeros(Cout, np.float32)))
    y, _ = capi.conv2d(ctx, d, dev(to_nhwc(xq).astype(np.int8 if dtype == "i8" else np.float16)), p, dev(to_nhwc(res).astype(np.float16)))
    ctx.sync_check()
    np.testing.assert_array_equal(to_nchw(host(y)), ref)


# Channel counts whose 256-channel tiles are not whole 32-channel blocks.
@pytest.mark.parametrize("case", [(1, 640, 50, 50, 1152, "f16", 2), (1, 640, 46, 48, 1920, "f16", 2)])
def test_conv_half_resolution_residual_of_many_channels(ctx, case):
    test_conv_half_resolution_residual(ctx, case)


# Depth-to-space in the epilogue: one and several N tiles, factors that differ.
@pytest.mark.parametrize("case", [(2, 64, 9, 7, 64, 2, 2), (1, 32, 20, 33, 32, 1, 3), (3, 128, 12, 11, 32, 2, 4), (2, 256, 60, 92, 128, 2, 2)])
def test_conv_depth_to_space(ctx, case):
    import torch
    capi = _capi()
    N, Cin, H, W, C, rh, rw = case
    r = rng(sum(case) + 24)
    Cout = rh * rw * C
    x = r.integers(-4, 5, (N, Cin, H, W)).astype(np.int8)
    wq = r.integers(-2, 3, (Cout, Cin, 1, 1)).astype(np.int8)
    b = r.integers(-9, 10, Cout).astype(np.float32)
    d = capi.make_conv_desc(N, H, W, Cin, Cout, 1, 1, 0, capi.EXB_F16, capi.EXB_F16, act=1)
    p = capi.ConvWeights(ctx, d, wq.astype(np.float32), b)
    d.d2s_h, d.d2s_w = rh, rw
    assert capi.lib().exb_conv2d_d2s_fusable(d) == 1
    y = torch.full((N, H * rh, W * rw, C), -1.0, device="cuda", dtype=torch.float16)
    capi.conv2d(ctx, d, dev(to_nhwc(x).astype(np.float16)), p, y=y)
    ctx.sync_check()
    acc = np.maximum(O.conv2d_i8_acc(x, wq, 1, 0) + b[None, :, None, None], 0)
    ref = acc.reshape(N, rh, rw, C, H, W).transpose(0, 4, 1, 5, 2, 3).reshape(N, H * rh, W * rw, C)
    np.testing.assert_array_equal(host(y).astype(np.float32), ref.astype(np.float16).astype(np.float32))


# There is no pair kernel with PReLU or a mapped residual: N tiles of such layers are not chosen as if they ran in pairs.
# 128-channel tiles, two CTAs of 320 threads per SM, took 65 us for the first one where 256-channel tiles take 60.
@pytest.mark.parametrize("case", [(256, 7, 7, 512, 512, "prelu"), (256, 8, 6, 512, 512, "half")])
def test_layers_without_a_pair_kernel_keep_wide_tiles(ctx, case):
    import torch
    capi = _capi()
    N, H, W, Cin, Cout, kind = case
    half = kind == "half"
    d = capi.make_conv_desc(N, H, W, Cin, Cout, 3, 1, 1, capi.EXB_F16, capi.EXB_F16, act=1 if half else 106, res=half, impl=2)
    d.res_half = int(half)
    p = capi.ConvWeights(ctx, d, (rng(3).standard_normal((Cout, Cin, 3, 3)) * 0.02).astype(np.float32), None)
    p.set_slopes(ctx, np.full(Cout, 0.1, np.float32))
    x = torch.zeros((N, H, W, Cin), device="cuda", dtype=torch.float16)
    res = torch.zeros((N, H // 2, W // 2, Cout), device="cuda", dtype=torch.float16) if half else None
    launches = kernels_of(lambda: capi.conv2d(ctx, d, x, p, res))
    ctx.sync_check()
    conv = [k for k in launches if "conv_tc_kernel" in k[0]]
    assert len(conv) == 1 and conv[0][2][0] == 576, launches


def _route(ctx, case, i8, out, impl):
    """The convolution kernels that a case launches, by their demangled names."""
    import torch
    capi = _capi()
    N, Cin, H, W, Cout, k, s = case
    d = capi.make_conv_desc(N, H, W, Cin, Cout, k, s, k // 2, capi.EXB_I8 if i8 else capi.EXB_F16, out, impl=impl)
    w = np.zeros((Cout, Cin, k, k), np.int8 if i8 else np.float32)
    p = capi.ConvWeights(ctx, d, w, None, np.ones(Cout, np.float32), 1.0) if i8 else capi.ConvWeights(ctx, d, w)
    x = torch.zeros((N, H, W, Cin), device="cuda", dtype=torch.int8 if i8 else torch.float16)
    names = [n for n, _, _ in kernels_of(lambda: capi.conv2d(ctx, d, x, p))]
    ctx.sync_check()
    return [n for n in names if "conv_" in n]


# The shapes above run in the kernels they are there for.
@pytest.mark.parametrize("case", SPLIT_CASES)
def test_split_cases_take_the_split_kernel(ctx, case):
    capi = _capi()
    for i8 in (True, False):
        names = _route(ctx, case, i8, capi.EXB_I8 if i8 else capi.EXB_F32, 0)
        assert len(names) == 1 and "conv_split_kernel" in names[0], names


@pytest.mark.parametrize("case", PAIR_CASES + SINGLE_CASES)
def test_pair_cases_take_the_pair_kernel(ctx, case):
    capi = _capi()
    i8 = case[7] == "i8"
    names = _route(ctx, case[:7], i8, capi.EXB_I8 if i8 else capi.EXB_F32, 2)
    paired = re.search(r"conv_tc_kernel<(true|false), \w+, \w+, false, true>", names[0]) is not None
    assert len(names) == 1 and paired == (case in PAIR_CASES), names


# N tiles of short reductions: 128 channels where the epilogue sets the pace (CTAs of 320 threads, two per SM), 256 where the
# activations that every tile reads again do (CTAs of 576): fp16 below 256 bytes of K, more than two tiles per SM.
@pytest.mark.parametrize("case,wide", [((64, 112, 28, 28, 320, 1, 1, "f16"), True), ((16, 48, 28, 28, 408, 3, 1, "f16"), True),
                                       ((32, 128, 14, 14, 1280, 3, 1, "i8"), True), ((100, 384, 10, 10, 256, 1, 1, "i8"), False),
                                       ((25, 96, 56, 56, 192, 3, 2, "i8"), False), ((32, 160, 28, 28, 320, 1, 1, "f16"), False)])
def test_n_tile_of_short_reductions(ctx, case, wide):
    import torch
    capi = _capi()
    N, Cin, H, W, Cout, k, s, dtype = case
    i8 = dtype == "i8"
    r = rng(sum(case[:7]))
    d = capi.make_conv_desc(N, H, W, Cin, Cout, k, s, k // 2, capi.EXB_I8 if i8 else capi.EXB_F16, capi.EXB_F32, impl=2)
    wq = r.integers(-8, 9, (Cout, Cin, k, k)).astype(np.int8)
    p = capi.ConvWeights(ctx, d, wq, None, np.ones(Cout, np.float32), 1.0) if i8 else capi.ConvWeights(ctx, d, wq.astype(np.float32))
    x = r.integers(-8, 9, (N, H, W, Cin)).astype(np.int8)
    xd = dev(x if i8 else x.astype(np.float16))
    launches = [l for l in kernels_of(lambda: capi.conv2d(ctx, d, xd, p)) if "conv_tc_kernel" in l[0]]
    assert len(launches) == 1 and launches[0][2][0] == (576 if wide else 320), launches
    y, _ = capi.conv2d(ctx, d, xd, p)
    ctx.sync_check()
    for n in (0, N - 1):
        np.testing.assert_array_equal(host(y[n]).transpose(2, 0, 1), O.conv2d_i8_acc(x[n:n + 1].transpose(0, 3, 1, 2), wq, s, k // 2)[0].astype(np.float32))


# 64-channel tiles keep their weights resident on one CTA per SM (576 threads, pairs) for K blocks of 128 bytes only: 96 fp16
# channels took 50.5 us that way at 100 x 44 x 44, 35.4 with two CTAs of 320 threads per SM.
@pytest.mark.parametrize("cin,threads", [(96, 320), (64, 576), (128, 576)])
def test_resident_weights_of_64_channel_tiles(ctx, cin, threads):
    import torch
    capi = _capi()
    d = capi.make_conv_desc(50, 44, 44, cin, 64, 3, 1, 1, capi.EXB_F16, capi.EXB_F32, impl=2)
    r = rng(cin)
    wq = r.integers(-8, 9, (64, cin, 3, 3)).astype(np.int8)
    x = r.integers(-8, 9, (50, 44, 44, cin)).astype(np.int8)
    p, xd = capi.ConvWeights(ctx, d, wq.astype(np.float32)), dev(x.astype(np.float16))
    launches = [l for l in kernels_of(lambda: capi.conv2d(ctx, d, xd, p)) if "conv_tc_kernel" in l[0]]
    assert len(launches) == 1 and launches[0][2][0] == threads, launches
    y, _ = capi.conv2d(ctx, d, xd, p)
    ctx.sync_check()
    for n in (0, 49):
        np.testing.assert_array_equal(host(y[n]).transpose(2, 0, 1), O.conv2d_i8_acc(x[n:n + 1].transpose(0, 3, 1, 2), wq, 1, 1)[0].astype(np.float32))


# Tiles of more than 128 channels do not run as pairs where that takes a round more: 125 tiles on 148 SMs, 75 pairs on 74.
@pytest.mark.parametrize("case,paired", [((2, 128, 40, 40, 1280, "f16"), False), ((2, 256, 40, 40, 1280, "i8"), False), ((2, 128, 40, 40, 1024, "f16"), True)])
def test_pairs_take_no_extra_round(ctx, case, paired):
    capi = _capi()
    N, Cin, H, W, Cout, dtype = case
    names = _route(ctx, (N, Cin, H, W, Cout, 3, 1), dtype == "i8", capi.EXB_I8 if dtype == "i8" else capi.EXB_F16, 2)
    assert len(names) == 1 and (re.search(r"conv_tc_kernel<(true|false), \w+, \w+, false, true>", names[0]) is not None) == paired, names


# The choice between the kernels: divided tiles where they do not fill the SMs, the persistent kernel for short int8 reductions
# of more tiles (96 -> 320 1x1 at 8 x 40 x 40 took 11.4 us divided, 8.1 not).
@pytest.mark.parametrize("case,split", [((8, 96, 40, 40, 320, 1, 1), False), ((8, 128, 56, 56, 96, 1, 1), False), ((8, 256, 7, 7, 960, 1, 1), True)])
def test_short_int8_reductions_are_divided_only_when_few(ctx, case, split):
    capi = _capi()
    names = _route(ctx, case, True, capi.EXB_I8, 0)
    assert len(names) == 1 and ("conv_split_kernel" in names[0]) == split, names


# Long reductions whose undivided tiles just fit the SMs: int8 ones are divided, fp16 ones keep the order of their sums.
@pytest.mark.parametrize("case,i8,kernel,ctas", [((5, 512, 56, 56, 32, 3, 1), False, "conv_split_kernel<false, false, true>", 133),
                                                 ((8, 288, 56, 56, 192, 3, 2), True, "conv_split_kernel<true, false, false>", 294)])
def test_long_reductions_of_one_tile_per_sm(ctx, case, i8, kernel, ctas):
    import torch
    capi = _capi()
    N, Cin, H, W, Cout, k, s = case
    d = capi.make_conv_desc(N, H, W, Cin, Cout, k, s, k // 2, capi.EXB_I8 if i8 else capi.EXB_F16, capi.EXB_F16, impl=0)
    r = rng(sum(case))
    wq = r.integers(-4, 5, (Cout, Cin, k, k)).astype(np.int8)
    x = r.integers(-2, 3, (N, H, W, Cin)).astype(np.int8)
    p = capi.ConvWeights(ctx, d, wq, None, np.ones(Cout, np.float32), 1.0) if i8 else capi.ConvWeights(ctx, d, wq.astype(np.float32))
    xd = dev(x if i8 else x.astype(np.float16))
    launches = [l for l in kernels_of(lambda: capi.conv2d(ctx, d, xd, p)) if "conv_" in l[0]]
    assert len(launches) == 1 and kernel in launches[0][0] and launches[0][1][0] == ctas, launches
    y, _ = capi.conv2d(ctx, d, xd, p)
    ctx.sync_check()
    want = O.conv2d_i8_acc(x[-1:].transpose(0, 3, 1, 2), wq, s, k // 2)[0].astype(np.float16)
    np.testing.assert_array_equal(host(y[-1]).transpose(2, 0, 1), want)


# Whichever kernel the plan picks, an fp16 layer's sums keep their order, to the last bit of an fp32 result: undivided tiles and the
# persistent kernel's tap loop (and its row boxes of one channel block) sum alike.
@pytest.mark.parametrize("case", [(1, 80, 66, 50, 400, 3, 1), (2, 48, 64, 50, 264, 3, 1), (9, 64, 13, 12, 384, 1, 1), (4, 320, 21, 77, 344, 1, 2), (20, 64, 30, 25, 128, 3, 1),
                                  (16, 32, 40, 40, 64, 3, 1)])
def test_undivided_sums_keep_their_order(ctx, case):
    import torch
    capi = _capi()
    N, Cin, H, W, Cout, k, s = case
    r = rng(sum(case))
    w = r.standard_normal((Cout, Cin, k, k)).astype(np.float32)
    x = dev(r.standard_normal((N, H, W, Cin)).astype(np.float16))
    desc = lambda impl: capi.make_conv_desc(N, H, W, Cin, Cout, k, s, k // 2, capi.EXB_F16, capi.EXB_F32, impl=impl)
    p = capi.ConvWeights(ctx, desc(0), w)
    names = [n for n, _, _ in kernels_of(lambda: capi.conv2d(ctx, desc(0), x, p)) if "conv_" in n]
    assert len(names) == 1 and re.search(r"conv_split_kernel<\w+, \w+, true>", names[0]), names
    assert torch.equal(capi.conv2d(ctx, desc(0), x, p)[0], capi.conv2d(ctx, desc(2), x, p)[0])
    ctx.sync_check()


# The lean quad epilogue (fp16 result, alone or with an int8 copy) against the same kernel's fp32 result, which is read from the
# general form: whole-number operands, so the sums are exact whatever their order, and scale, bias, residual, activation and
# rounding are repeated here in the same fp32 steps.  N tiles of one, two, three and five blocks, a tile that ends inside its
# last block, one CTA per SM and two, pairs, three and eight accumulators in flight; infinities and NaN.
LEAN_CASES = [(5, 32, 17, 13, 32, 1, 1), (3, 64, 9, 7, 72, 1, 1), (2, 32, 11, 13, 160, 1, 1), (40, 64, 28, 28, 96, 1, 1), (3, 96, 8, 8, 64, 3, 2),
              (50, 64, 24, 24, 64, 3, 1), (9, 32, 30, 30, 320, 1, 1)]


@pytest.mark.parametrize("i8", [True, False])
@pytest.mark.parametrize("case", LEAN_CASES)
def test_lean_quad_epilogue(ctx, case, i8):
    import torch
    capi = _capi()
    N, Cin, H, W, Cout, k, s = case
    r = rng(sum(case) + i8)
    wq = r.integers(-3, 4, (Cout, Cin, k, k)).astype(np.int8)
    bias = r.integers(-40, 40, Cout).astype(np.float32) / 8
    ws = np.exp2(r.integers(2, 6, Cout)).astype(np.float32)

    def desc(out, out2, act, res):
        return capi.make_conv_desc(N, H, W, Cin, Cout, k, s, k // 2, capi.EXB_I8 if i8 else capi.EXB_F16, out, out2, res=res, act=act,
                                   out_scale=0.7, out2_scale=0.7, impl=2)
    d0 = desc(capi.EXB_F32, -1, 0, False)
    p = capi.ConvWeights(ctx, d0, wq, bias, ws, 0.25) if i8 else capi.ConvWeights(ctx, d0, wq.astype(np.float32), bias)
    x = r.integers(-4, 5, (N, H, W, Cin)).astype(np.int8 if i8 else np.float16)
    if not i8:
        x[0, 0, 0, 0], x[-1, -1, -1, 1] = np.inf, np.nan
    xd = dev(x)
    v = capi.conv2d(ctx, d0, xd, p)[0]
    oh, ow = capi.conv_out_dims(d0)
    skip = dev(r.standard_normal((N, oh, ow, Cout)).astype(np.float16))
    for act in (0, 1, 103, 104):
        for res in (False, True):
            for out2 in (-1, capi.EXB_I8):
                y, y2 = capi.conv2d(ctx, desc(capi.EXB_F16, out2, act, res), xd, p, residual=skip if res else None)
                u = v + skip.float() if res else v
                if act == 104:
                    want = u * torch.sigmoid(u)
                    ok = torch.isfinite(want)
                    # the sigmoid is within 2 ulp of fp32: at most one fp16 rounding apart
                    assert ((y.float() - want.half().float()).abs()[ok] <= (want.abs() * 2.0 ** -10 + 2.0 ** -24)[ok]).all(), (act, res, out2)
                else:
                    # fmaxf / fminf: a NaN gives the bound
                    want = u if act == 0 else torch.where(u > 0, u, torch.zeros_like(u))
                    if act == 103:
                        want = torch.where(want < 6, want, torch.full_like(u, 6.0))
                    assert torch.equal(torch.nan_to_num(y, nan=12345.0), torch.nan_to_num(want.half(), nan=12345.0)), (act, res, out2)
                    if y2 is not None:
                        ok = ~torch.isnan(want)
                        assert torch.equal(y2[ok], (want * 0.7).round().clamp(-128, 127).to(torch.int8)[ok]), (act, res, out2)
    ctx.sync_check()


# The same where each case is sure to run in the quad epilogue (q; r: row epilogue) of so many warps, in pairs (p), fp16 and int8.
LEAN_KERNELS = [((5, 32, 17, 13, 32, 1, 1), "8q", "8q"), ((3, 64, 9, 7, 72, 1, 1), "8r", "8r"), ((2, 32, 11, 13, 160, 1, 1), "16q", "16q"),
                ((40, 64, 28, 28, 96, 1, 1), "8q", "8q"), ((3, 96, 8, 8, 64, 3, 2), "8q", "8q"), ((50, 64, 24, 24, 64, 3, 1), "8q", "8q"),
                ((9, 32, 30, 30, 320, 1, 1), "16q", "8r"),
                # channels that end inside the last block
                ((5, 32, 17, 13, 24, 1, 1), "8q", "8q"), ((3, 64, 9, 7, 56, 1, 1), "8q", "8q"), ((5, 64, 12, 9, 88, 3, 1), "8q", "8q"),
                # more tiles per CTA than its eight, three and four accumulators
                ((100, 32, 56, 56, 32, 1, 1), "8q", "8q"), ((19, 32, 56, 56, 160, 1, 1), "16q", "16q"), ((50, 64, 56, 56, 64, 1, 1), "8q", "8q"),
                # pairs: row boxes, tap loop, one and several tiles each
                ((50, 128, 28, 28, 64, 3, 1), "16qp", "16qp"), ((3, 64, 15, 15, 128, 3, 1), "16qp", "16qp"),
                ((2, 128, 9, 9, 384, 3, 1), "16qp", "8q"), ((40, 256, 14, 14, 512, 3, 1), "16qp", "16qp")]


@pytest.mark.parametrize("i8", [True, False])
@pytest.mark.parametrize("case,f16_kernel,i8_kernel", LEAN_KERNELS)
def test_lean_quad_kernels(ctx, case, f16_kernel, i8_kernel, i8):
    capi = _capi()
    N, Cin, H, W, Cout, k, s = case
    d = capi.make_conv_desc(N, H, W, Cin, Cout, k, s, k // 2, capi.EXB_I8 if i8 else capi.EXB_F16, capi.EXB_F16, act=1, impl=2)
    w = np.ones((Cout, Cin, k, k), np.int8 if i8 else np.float32)
    p = capi.ConvWeights(ctx, d, w, None, np.ones(Cout, np.float32), 1.0) if i8 else capi.ConvWeights(ctx, d, w)
    x = dev(np.zeros((N, H, W, Cin), np.int8 if i8 else np.float16))
    name = [n for n, _, _ in kernels_of(lambda: capi.conv2d(ctx, d, x, p)) if "conv_" in n][0]
    warps, epi, pair = re.search(r"conv_tc_kernel<\w+, (\d+), \D*(\d), \w+, (\w+)>", name).groups()
    assert warps + {"0": "r", "1": "q"}[epi] + ("p" if pair == "true" else "") == (i8_kernel if i8 else f16_kernel), name
    test_lean_quad_epilogue(ctx, case, i8)


# Reductions that are not divided, and the exchange of those that are, with boxes of fewer pixels than a tile has rows and rings
# smaller than the tile that takes their place; channel counts with and without whole 32-channel blocks.
@pytest.mark.parametrize("case", [(15, 32, 11, 11, 176, 1, 2), (15, 32, 11, 11, 192, 1, 2), (1, 64, 6, 6, 48, 1, 1), (3, 64, 5, 5, 64, 1, 1), (2, 512, 5, 7, 208, 3, 1),
                                  (1, 1024, 3, 3, 512, 1, 1), (7, 128, 9, 13, 128, 3, 1), (1, 256, 13, 11, 256, 3, 1)])
@pytest.mark.parametrize("i8", [True, False])
def test_split_tiles_of_few_pixels(ctx, case, i8):
    import torch
    capi = _capi()
    N, Cin, H, W, Cout, k, s = case
    names = _route(ctx, case, i8, capi.EXB_I8 if i8 else capi.EXB_F16, 0)
    assert len(names) == 1 and "conv_split_kernel" in names[0], names
    r = rng(sum(case) + i8)
    wq = r.integers(-4, 5, (Cout, Cin, k, k)).astype(np.int8)
    x = dev(r.integers(-4, 5, (N, H, W, Cin)).astype(np.int8 if i8 else np.float16))
    got = []
    for impl in (0, 2):        # whole numbers: exact whatever the order of the sums
        d = capi.make_conv_desc(N, H, W, Cin, Cout, k, s, k // 2, capi.EXB_I8 if i8 else capi.EXB_F16, capi.EXB_F16, capi.EXB_I8, res=True, act=1,
                                out2_scale=0.01, impl=impl)
        oh, ow = capi.conv_out_dims(d)
        skip = dev(rng(7).integers(-50, 50, (N, oh, ow, Cout)).astype(np.float16))
        p = capi.ConvWeights(ctx, d, wq, None, np.ones(Cout, np.float32), 1.0) if i8 else capi.ConvWeights(ctx, d, wq.astype(np.float32))
        got.append(capi.conv2d(ctx, d, x, p, residual=skip))
        ctx.sync_check()
    for a, b in zip(*got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("case,undivided", [((15, 32, 11, 11, 176, 1, 2), True), ((15, 32, 11, 11, 192, 1, 2), True), ((1, 64, 6, 6, 48, 1, 1), True),
                                            ((3, 64, 5, 5, 64, 1, 1), True), ((2, 512, 5, 7, 208, 3, 1), False), ((1, 1024, 3, 3, 512, 1, 1), False),
                                            ((7, 128, 9, 13, 128, 3, 1), False), ((1, 256, 13, 11, 256, 3, 1), False)])
@pytest.mark.parametrize("i8", [True, False])
def test_form_of_split_tiles_of_few_pixels(ctx, case, undivided, i8):
    capi = _capi()
    names = _route(ctx, case, i8, capi.EXB_I8 if i8 else capi.EXB_F16, 0)
    assert len(names) == 1 and re.search(r"conv_split_kernel<\w+, \w+, %s>" % ("true" if undivided else "false"), names[0]), names


# Undivided tiles, which go from TMEM to the result in a loop of their own: every activation, residual and output against the
# persistent kernel on whole-number operands.  Channel counts with and without whole 32-channel blocks, N tiles beyond the first,
# boxes of fewer pixels than a tile has rows; int8 alone behind a residual and no activation, PReLU and fp32 take the general form.
DIRECT_CASES = [(15, 32, 11, 11, 176, 1, 2), (1, 64, 12, 10, 256, 1, 1), (3, 64, 6, 4, 72, 1, 1), (40, 128, 14, 14, 96, 1, 1)]


@pytest.mark.parametrize("i8", [True, False])
@pytest.mark.parametrize("case", DIRECT_CASES)
def test_split_undivided_tiles(ctx, case, i8):
    import torch
    capi = _capi()
    N, Cin, H, W, Cout, k, s = case
    r = rng(sum(case) + i8)
    wq = r.integers(-3, 4, (Cout, Cin, k, k)).astype(np.int8)
    bias = r.integers(-40, 40, Cout).astype(np.float32) / 8
    x = dev(r.integers(-4, 5, (N, H, W, Cin)).astype(np.int8 if i8 else np.float16))
    slopes = r.integers(1, 8, Cout).astype(np.float32) / 8

    def desc(out, out2, act, res, impl):
        d = capi.make_conv_desc(N, H, W, Cin, Cout, k, s, k // 2, capi.EXB_I8 if i8 else capi.EXB_F16, out, out2, res=res != 0, act=act,
                                out_scale=0.7, out2_scale=0.3, impl=impl)
        d.res_half = int(res == 2)
        return d
    d0 = desc(capi.EXB_F16, -1, 0, 0, 0)
    p = capi.ConvWeights(ctx, d0, wq, bias, np.exp2(r.integers(2, 6, Cout)).astype(np.float32), 0.25) if i8 else \
        capi.ConvWeights(ctx, d0, wq.astype(np.float32), bias)
    p.set_slopes(ctx, slopes)
    oh, ow = capi.conv_out_dims(d0)
    full = dev(r.standard_normal((N, oh, ow, Cout)).astype(np.float16))
    half = dev(r.standard_normal((N, oh // 2, ow // 2, Cout)).astype(np.float16))
    halves = oh % 2 == 0 and ow % 2 == 0 and Cout % 32 == 0
    for act in (0, 1, 103, 104, capi.ACT_PRELU):
        for res in (0, 1, 2) if halves else (0, 1):
            for out, out2 in ((capi.EXB_F16, -1), (capi.EXB_F16, capi.EXB_I8), (capi.EXB_I8, -1), (capi.EXB_F32, -1)):
                if res == 2 and (out == capi.EXB_I8 or act == capi.ACT_PRELU):
                    continue
                run = lambda impl: capi.conv2d(ctx, desc(out, out2, act, res, impl), x, p, residual=(None, full, half)[res])
                if out == capi.EXB_F16:
                    names = [n for n, _, _ in kernels_of(lambda: run(0)) if "conv_" in n]
                    assert len(names) == 1 and re.search(r"conv_split_kernel<\w+, \w+, true>", names[0]), names
                (a, a2), (b, b2) = run(0), run(2)
                assert torch.equal(a, b), (act, res, out, out2)
                assert a2 is None or torch.equal(a2, b2), (act, res, out, out2)
    ctx.sync_check()
