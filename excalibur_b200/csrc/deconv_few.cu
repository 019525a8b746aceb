// Transposed convolution with kernel = stride, few outputs per input pixel and an fp32 NCHW result (a probability map at
// the end of a segmentation head: 64 channels -> 1, 2 x 2).
//
// It is a 1 x 1 convolution to rh * rw * C <= 4 values per pixel whose result is scattered, bound by reading the input
// once.  As a tcgen05 convolution it pads those to 16 channels, writes them as fp16 and takes a second pass to scatter them.
// Here a warp multiplies 16 pixels at a time by mma.sync, whose fragments come straight from global memory: the order of
// the reduction is free, so four lanes share a pixel and each reads 32 contiguous bytes of it.  (Eight lanes per pixel with
// FMAs and shuffles were bound by their instructions: 20.8 us.)  64 -> 1, 2 x 2, sigmoid at 4 x 240 x 368: two passes 32 us,
// this kernel 13 us.
#include "conv_common.cuh"

namespace exb {
namespace {

constexpr int kFewThreads = 256, kFewOutputs = 4, kFewChannels = 64, kFewUnroll = 2;
constexpr int kFewPixels = kFewThreads / 32 * 16 * kFewUnroll;      // pixels of a block's step

__global__ void __launch_bounds__(kFewThreads) deconv_few_kernel(const __half* __restrict__ x, const __half* __restrict__ w,
                                                                 const float* __restrict__ scale, const float* __restrict__ bias,
                                                                 const float* __restrict__ slope, float* __restrict__ y, int pixels,
                                                                 int H, int W, int rh, int rw, int C, int cs, int act) {
    // Lane l = 4 * g + j: rows (pixels) g and g + 8, channels 16 * j .. + 15 of the pixel, in K steps of four of them;
    // of the weights output g's; of the accumulators outputs 2 * j and 2 * j + 1.
    const int lane = threadIdx.x & 31, g = lane >> 2, j = lane & 3, outputs = rh * rw * C, OW = W * rw;
    uint4 wv[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        wv[i] = make_uint4(0u, 0u, 0u, 0u);
        if (g < outputs && j * 16 + i * 8 < cs) wv[i] = *reinterpret_cast<const uint4*>(w + g * cs + j * 16 + i * 8);
    }
    float qs[2], qb[2], neg[2];
    int at[2];          // of the output from its pixel's first
    int plane[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int q = 2 * j + k;
        const bool real = q < outputs;
        qs[k] = real ? scale[q] : 0.f;
        qb[k] = real ? bias[q] : 0.f;
        neg[k] = real && act == EXB_ACT_PRELU ? slope[q] : 0.f;
        const int t = q / C, a = t / rw;
        plane[k] = q - t * C;
        at[k] = a * OW + t - a * rw;
    }
    const bool adjacent = C == 1 && rw == 2 && 2 * j + 1 < outputs;      // both outputs side by side
    pdl_enter();
    const int first = (blockIdx.x * (kFewThreads / 32) + (threadIdx.x >> 5)) * 16 * kFewUnroll;
    for (int p0 = first; p0 < pixels; p0 += gridDim.x * kFewPixels) {
        __syncwarp();
        uint4 raw[kFewUnroll][2][2];       // [..][row half][8 channels]
#pragma unroll
        for (int u = 0; u < kFewUnroll; ++u)
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int p = p0 + u * 16 + r * 8 + g;
                    raw[u][r][i] = make_uint4(0u, 0u, 0u, 0u);
                    if (p < pixels && j * 16 + i * 8 < cs)
                        raw[u][r][i] = __ldg(reinterpret_cast<const uint4*>(x + (int64_t)p * cs + j * 16 + i * 8));
                }
        float sums[kFewUnroll][4] = {};
#pragma unroll
        for (int u = 0; u < kFewUnroll; ++u) {
            float (&acc)[4] = sums[u];
            auto mma = [&](uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
                asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                             : "+f"(acc[0]), "+f"(acc[1]), "+f"(acc[2]), "+f"(acc[3])
                             : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
            };
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const uint4 lo = raw[u][0][i], hi = raw[u][1][i];
                mma(lo.x, hi.x, lo.y, hi.y, wv[i].x, wv[i].y);
                mma(lo.z, hi.z, lo.w, hi.w, wv[i].z, wv[i].w);
            }
        }
        if (2 * j >= outputs) continue;
#pragma unroll
        for (int u = 0; u < kFewUnroll; ++u) {
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int p = p0 + u * 16 + r * 8 + g;
                if (p >= pixels) continue;
                const int row = p / W, ox = p - row * W;            // row of all images
                float v[2];
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    v[k] = fmaf(sums[u][2 * r + k], qs[k], qb[k]);
                    if (act == EXB_ACT_PRELU) v[k] = v[k] >= 0.f ? v[k] : v[k] * neg[k];
                    else if (act != EXB_ACT_NONE) v[k] = apply_act(v[k], act);
                }
                if (adjacent) {
                    *reinterpret_cast<float2*>(y + (int64_t)row * rh * OW + ox * rw + at[0]) = make_float2(v[0], v[1]);
                } else {
                    const int before = row / H * (C - 1);      // planes of H rows that come before, beside the rows themselves
#pragma unroll
                    for (int k = 0; k < 2; ++k)
                        if (2 * j + k < outputs)
                            y[((int64_t)(before + plane[k]) * H + row) * rh * OW + ox * rw + at[k]] = v[k];
                }
            }
        }
    }
}

}  // namespace
}  // namespace exb

using namespace exb;

extern "C" int exb_deconv_few_f32(exb_ctx* ctx, const void* x, const exb_conv_weights* w, float* y, int N, int H, int W, int rh, int rw,
                                  int C, int act, void* stream) {
    EXB_REQUIRE(ctx != nullptr && w != nullptr, "exb_deconv_few_f32: null argument");
    EXB_REQUIRE(N >= 0 && H > 0 && W > 0 && rh > 0 && rw > 0 && C > 0, "exb_deconv_few_f32: bad shape");
    EXB_REQUIRE(w->dtype == EXB_F16 && w->kh == 1 && w->kw == 1 && w->group == 1 && w->Cout == rh * rw * C,
                "exb_deconv_few_f32: weights are not those of a 1x1 fp16 convolution to %d channels", rh * rw * C);
    if (rh * rw * C > kFewOutputs || w->cin_pad > kFewChannels || w->cin_pad % 8)
        return fail(EXB_ERR_UNSUPPORTED, "exb_deconv_few_f32: up to %d outputs of up to %d channels, a multiple of 8", kFewOutputs, kFewChannels);
    EXB_REQUIRE(act != EXB_ACT_PRELU || w->d_slope != nullptr, "exb_deconv_few_f32: EXB_ACT_PRELU without slopes (exb_conv_weights_set_slopes)");
    EXB_REQUIRE(w->device == ctx->device, "exb_deconv_few_f32: weights live on device %d, context on %d", w->device, ctx->device);
    if (N == 0) return EXB_OK;
    EXB_REQUIRE(x && y && aligned16(x), "exb_deconv_few_f32: null or misaligned buffer");
    EXB_REQUIRE((int64_t)N * H * W < (1ll << 30), "exb_deconv_few_f32: map too large");
    EXB_REQUIRE(C != 1 || rw != 2 || (reinterpret_cast<uintptr_t>(y) & 7) == 0, "exb_deconv_few_f32: misaligned result");
    const int pixels = N * H * W;
    int grid = (pixels + kFewPixels - 1) / kFewPixels;
    if (grid > 4 * ctx->sm_count) grid = 4 * ctx->sm_count;      // what is resident: the weights are read once per block
    launch_overlapped(ctx, deconv_few_kernel, dim3((unsigned)grid), dim3(kFewThreads), static_cast<cudaStream_t>(stream),
                      static_cast<const __half*>(x), static_cast<const __half*>(w->d_w), w->d_scale, w->d_bias, w->d_slope, y, pixels, H, W,
                      rh, rw, C, w->cin_pad, act);
    return after_launch("exb_deconv_few_f32");
}
