// Depthwise convolution on NHWC tensors, fp32 math on fp16 or int8 activations.  Weights are kept tap-major [kh*kw][C] in
// fp32 so consecutive threads read consecutive channels.  Three kernels: 3x3 windows of fp16 maps run on the row stream
// (dw3x3_stream_kernel); 3x3 windows of int8 maps with a thread per 8 channels of a strip of TW output pixels, in which every
// input vector is loaded once per kernel row and reused by all taps that touch it (dw_strip_kernel); any other window with
// a thread per output vector (dw_generic_kernel).
#include <math.h>

#include <type_traits>

#include "common.cuh"
#include "row_stream.cuh"

struct exb_dw_weights {
    float* d_w;     // [kh*kw][cs]
    float* d_bias;  // [cs] (zeros when the layer has no bias)
    float* d_slope; // [cs] PReLU slopes, or null
    int C, cs, kh, kw;
    int device;
};

namespace exb {
namespace {

constexpr int V = 8;  // channels per thread

struct DwParams {
    int N, H, W, cs, OH, OW;
    int kh, kw, sh, sw, pt, pl;
    int act;
    float in_scale, out_scale;
    const float* slope;   // EXB_ACT_PRELU only: [cs]
};

__device__ __forceinline__ void load8(const __half* p, float (&v)[V], float) {
    uint4 r = *reinterpret_cast<const uint4*>(p);
    const __half2* h = reinterpret_cast<const __half2*>(&r);
#pragma unroll
    for (int i = 0; i < 4; ++i) { float2 f = __half22float2(h[i]); v[2 * i] = f.x; v[2 * i + 1] = f.y; }
}
__device__ __forceinline__ void load8(const int8_t* p, float (&v)[V], float scale) {
    alignas(8) int8_t b[8];
    *reinterpret_cast<uint2*>(b) = *reinterpret_cast<const uint2*>(p);
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = (float)b[i] * scale;
}
__device__ __forceinline__ void store8(__half* p, const float (&v)[V], float) {
    uint4 r;
    __half2* h = reinterpret_cast<__half2*>(&r);
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
    *reinterpret_cast<uint4*>(p) = r;
}
__device__ __forceinline__ void store8(int8_t* p, const float (&v)[V], float scale) {
    uint2 r;
    r.x = quant_pack4(v[0], v[1], v[2], v[3], scale);
    r.y = quant_pack4(v[4], v[5], v[6], v[7], scale);
    *reinterpret_cast<uint2*>(p) = r;
}
__device__ __forceinline__ void loadw(const float* p, float (&v)[V]);
// Activation of the 8 channels starting at c0.
__device__ __forceinline__ void dw_act(float (&v)[V], const DwParams& p, int c0) {
    if (p.act == EXB_ACT_PRELU) {
        float s[V];
        loadw(p.slope + c0, s);
#pragma unroll
        for (int k = 0; k < V; ++k) v[k] = v[k] >= 0.f ? v[k] : v[k] * s[k];
    } else {
        apply_act_vec(v, p.act);
    }
}
__device__ __forceinline__ void loadw(const float* p, float (&v)[V]) {
    float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

template <typename TIn, typename TOut, int K, int S, int TW>
__global__ void __launch_bounds__(128) dw_strip_kernel(const TIn* __restrict__ x, const float* __restrict__ w,
                                                       const float* __restrict__ bias, TOut* __restrict__ y,
                                                       DwParams p) {
    constexpr int IN_W = (TW - 1) * S + K;
    const int cvecs = p.cs / V;
    const int owb = (p.OW + TW - 1) / TW;
    const int64_t total = (int64_t)p.N * p.OH * owb * cvecs;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += stride) {
        const int cv = (int)(idx % cvecs);
        int64_t t = idx / cvecs;
        const int ob = (int)(t % owb); t /= owb;
        const int oh = (int)(t % p.OH);
        const int n = (int)(t / p.OH);
        const int ow0 = ob * TW;
        float acc[TW][V];
        {
            float b[V];
            loadw(bias + cv * V, b);
#pragma unroll
            for (int j = 0; j < TW; ++j)
#pragma unroll
                for (int k = 0; k < V; ++k) acc[j][k] = b[k];
        }
#pragma unroll
        for (int r = 0; r < K; ++r) {
            const int ih = oh * S - p.pt + r;
            if (ih < 0 || ih >= p.H) continue;
            float in[IN_W][V];
#pragma unroll
            for (int j = 0; j < IN_W; ++j) {
                const int iw = ow0 * S - p.pl + j;
                if (iw >= 0 && iw < p.W) {
                    load8(x + (((int64_t)n * p.H + ih) * p.W + iw) * p.cs + cv * V, in[j], p.in_scale);
                } else {
#pragma unroll
                    for (int k = 0; k < V; ++k) in[j][k] = 0.f;
                }
            }
#pragma unroll
            for (int s = 0; s < K; ++s) {
                float wv[V];
                loadw(w + (int64_t)(r * K + s) * p.cs + cv * V, wv);
#pragma unroll
                for (int j = 0; j < TW; ++j)
#pragma unroll
                    for (int k = 0; k < V; ++k) acc[j][k] = fmaf(in[j * S + s][k], wv[k], acc[j][k]);
            }
        }
#pragma unroll
        for (int j = 0; j < TW; ++j) {
            const int ow = ow0 + j;
            if (ow < p.OW) {
                dw_act(acc[j], p, cv * V);
                store8(y + (((int64_t)n * p.OH + oh) * p.OW + ow) * p.cs + cv * V, acc[j], p.out_scale);
            }
        }
    }
}

// 3x3, stride 1 or 2, fp16 input, on the row stream of row_stream.cuh.  A thread keeps its 9 x 4 weights in registers for
// the whole launch; an input row adds to the three output rows it belongs to (stride 2: one or two).  Products are packed
// fma.rn.f32x2, each lane the same fma, in the same order, as a scalar loop's.  144 channels @56, batch 256: 85 to 92 us
// from card to card, 77 to 83 % of the HBM copy rate (143 us with the window of rows in registers); 960 channels @7x6,
// batch 9: 3.7 us (22.6).
struct DwStreamParams : RowStreamParams {
    int act;
    float out_scale, clamp_hi;      // clamp_hi: upper bound of a ReLU / ReLU6 result (int8: of its multiple of out_scale)
    const float* slope;
};
constexpr int kDwStages = 3;
template <int S> constexpr RowStreamKind kDwKind = {S, S, 3, S == 1 ? 3 : 2, kDwStages, S == 1 ? 0 : 1, S == 1 ? 75.0 : 56.0};

// One output row of a thread: activation, conversion, store.  kClamp: ReLU or ReLU6.  Both are monotone with bounds that
// fp16 holds exactly, so an fp16 result is clamped after its rounding, two channels per instruction.
template <typename TOut, bool kClamp>
__device__ __forceinline__ void dw_store_row(const f32x2 (&acc)[kRowCols][2], TOut* y, int cs, int cols, const DwStreamParams& p, int c) {
    constexpr bool kHalf = std::is_same<TOut, __half>::value;
    if constexpr (kClamp && !kHalf) {
        // int8 behind ReLU / ReLU6: the bounds are applied to v * scale (a positive scale keeps the order, and both
        // forms round the same product), then 1.5 * 2^23 is added, which leaves the value rounded half to even in the
        // low byte: no float-to-integer conversions, whose quarter-rate pipe bounded this store (105 -> 91 us on 256
        // maps of 32 channels @112)
        const f32x2 s2 = pack2(p.out_scale, p.out_scale), magic = pack2(12582912.f, 12582912.f), one = pack2(1.f, 1.f), zero = pack2(-0.f, -0.f);
#pragma unroll
        for (int t = 0; t < kRowCols; ++t) {
            uint32_t u[4];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float a, b;
                asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(fma2(acc[t][h], s2, zero)));
                a = fminf(fmaxf(a, 0.f), p.clamp_hi);
                b = fminf(fmaxf(b, 0.f), p.clamp_hi);
                asm("mov.b64 {%0, %1}, %2;" : "=r"(u[2 * h]), "=r"(u[2 * h + 1]) : "l"(fma2(pack2(a, b), one, magic)));
            }
            if (t < cols)
                *reinterpret_cast<uint32_t*>(y + t * cs) = __byte_perm(__byte_perm(u[0], u[1], 0x0040), __byte_perm(u[2], u[3], 0x0040), 0x5410);
        }
        return;
    }
    float v[4 * kRowCols];
#pragma unroll
    for (int t = 0; t < kRowCols; ++t)
#pragma unroll
        for (int h = 0; h < 2; ++h) asm("mov.b64 {%0, %1}, %2;" : "=f"(v[4 * t + 2 * h]), "=f"(v[4 * t + 2 * h + 1]) : "l"(acc[t][h]));
    if constexpr (kClamp) {
        // bounds below
    } else if (p.act == EXB_ACT_PRELU) {
        const float4 s = __ldg(reinterpret_cast<const float4*>(p.slope + c));
        const float sl[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
        for (int k = 0; k < 4 * kRowCols; ++k) v[k] = v[k] >= 0.f ? v[k] : v[k] * sl[k & 3];
    } else {
        apply_act_vec(v, p.act);
    }
    if constexpr (kHalf) {
        const __half2 zero = __half2half2(__ushort_as_half(0)), hi = __float2half2_rn(p.clamp_hi);
#pragma unroll
        for (int t = 0; t < kRowCols; ++t) {
            __half2 a = __floats2half2_rn(v[4 * t], v[4 * t + 1]), b = __floats2half2_rn(v[4 * t + 2], v[4 * t + 3]);
            if constexpr (kClamp) {
                a = __hmin2(__hmax2(a, zero), hi);
                b = __hmin2(__hmax2(b, zero), hi);
            }
            if (t < cols)
                *reinterpret_cast<uint2*>(y + t * cs) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
        }
    } else {
#pragma unroll
        for (int t = 0; t < kRowCols; ++t)
            if (t < cols)
                *reinterpret_cast<uint32_t*>(y + t * cs) = quant_pack4(v[4 * t], v[4 * t + 1], v[4 * t + 2], v[4 * t + 3], p.out_scale);
    }
}

// acc = (first ? bias : acc) + the three taps of one kernel row on an input row
template <int S>
__device__ __forceinline__ void dw_taps(f32x2 (&acc)[kRowCols][2], int j, const f32x2 (&wv)[9][2], int krow, const f32x2 (&b2)[2],
                                        f32x2 v0, f32x2 v1) {
#pragma unroll
    for (int tc = 0; tc < kRowCols; ++tc) {
        const int sx = j - S * tc;
        if (sx < 0 || sx > 2) continue;
        const bool first = krow == 0 && sx == 0;
        acc[tc][0] = fma2(v0, wv[3 * krow + sx][0], first ? b2[0] : acc[tc][0]);
        acc[tc][1] = fma2(v1, wv[3 * krow + sx][1], first ? b2[1] : acc[tc][1]);
    }
}

template <typename TOut, int S, bool kClamp>
__global__ void __launch_bounds__(kRowThreads, 2)
    dw3x3_stream_kernel(const __grid_constant__ CUtensorMap map, const float* __restrict__ w, const float* __restrict__ bias,
                        TOut* __restrict__ y, const DwStreamParams p) {
    constexpr int RS = kDwKind<S>.RS, IN = (kRowCols - 1) * S + 3;
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full[kDwStages];
    __shared__ int abort_flag;
    uint8_t* ring = row_stream_init<kDwStages>(map, smem_raw, full, &abort_flag);
    const int c = (int)(blockIdx.x % p.slabs) * p.slab + (int)(threadIdx.x % p.units) * 4;
    f32x2 wv[9][2], b2[2];
    {
#pragma unroll
        for (int t = 0; t < 9; ++t) {
            const float4 f = __ldg(reinterpret_cast<const float4*>(w + (size_t)t * p.cs + c));
            wv[t][0] = pack2(f.x, f.y);
            wv[t][1] = pack2(f.z, f.w);
        }
        const float4 f = __ldg(reinterpret_cast<const float4*>(bias + c));
        b2[0] = pack2(f.x, f.y);
        b2[1] = pack2(f.z, f.w);
    }
    __syncthreads();
    pdl_wait();
    // stride 1: three output rows are in the making; stride 2: one
    f32x2 acc[S == 1 ? 3 : 1][kRowCols][2];
    const int64_t ypitch = (int64_t)p.OW * p.cs;
    RowTile t;
    TOut* yo = y;
    int o = 0;                          // output row that the next completed accumulator belongs to
    auto finish = [&](const f32x2 (&a)[kRowCols][2]) {
        if (o >= 0 && o < t.rows) dw_store_row<TOut, kClamp>(a, yo, p.cs, t.cols, p, c);
        ++o;
        yo += ypitch;
    };
    row_stream_run<S, 3, RS, kDwStages, S == 1 && std::is_same<TOut, int8_t>::value>(
        map, p, ring, full, &abort_flag,
        [&](const RowTile& tile) {
            t = tile;
            o = S == 1 ? -2 : -1;
            yo = y + (((int64_t)t.n * p.OH + t.oh0 + o) * p.OW + t.ow0) * p.cs + c;
#pragma unroll
            for (int a = 0; a < (S == 1 ? 3 : 1); ++a)
#pragma unroll
                for (int tc = 0; tc < kRowCols; ++tc) acc[a][tc][0] = b2[0], acc[a][tc][1] = b2[1];
        },
        [&](const int rr, const uint2 (&rv)[IN]) {
            if constexpr (S == 1) {
                // input row i = 3*st + rr is kernel row 0 of output row i, 1 of i - 1, 2 of i - 2 (which it completes)
#pragma unroll
                for (int j = 0; j < IN; ++j) {
                    const f32x2 v0 = cvt2(rv[j].x), v1 = cvt2(rv[j].y);
                    dw_taps<S>(acc[rr], j, wv, 0, b2, v0, v1);
                    dw_taps<S>(acc[(rr + 2) % 3], j, wv, 1, b2, v0, v1);
                    dw_taps<S>(acc[(rr + 1) % 3], j, wv, 2, b2, v0, v1);
                }
                finish(acc[(rr + 1) % 3]);
            } else if (rr == 0) {        // row 2k - 1: kernel row 1 of output row k - 1
#pragma unroll
                for (int j = 0; j < IN; ++j) dw_taps<S>(acc[0], j, wv, 1, b2, cvt2(rv[j].x), cvt2(rv[j].y));
            } else {                     // row 2k: kernel row 2 of output row k - 1, then kernel row 0 of row k
#pragma unroll
                for (int j = 0; j < IN; ++j) dw_taps<S>(acc[0], j, wv, 2, b2, cvt2(rv[j].x), cvt2(rv[j].y));
                finish(acc[0]);
#pragma unroll
                for (int j = 0; j < IN; ++j) dw_taps<S>(acc[0], j, wv, 0, b2, cvt2(rv[j].x), cvt2(rv[j].y));
            }
        });
}

template <typename TOut, int S>
int launch_stream(exb_ctx* ctx, const DwParams& d, const __half* x, const exb_dw_weights* w, TOut* y, cudaStream_t st) {
    const RowStreamKind& kind = kDwKind<S>;
    const RowStreamPlan pl = row_stream_plan(kind, ctx->sm_count, d.N, d.OH, d.OW, d.cs);
    DwStreamParams p;
    CUtensorMap map;
    size_t smem;
    const int grid = row_stream_setup(ctx, kind, pl, x, d.N, d.H, d.W, d.pt, d.pl, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE, p, map, smem);
    if (grid < 0) return grid;
    p.act = d.act; p.out_scale = d.out_scale; p.slope = d.slope;
    const bool half_out = std::is_same<TOut, __half>::value;
    const bool clamp = (d.act == EXB_ACT_RELU || d.act == EXB_ACT_RELU6) && (half_out || d.out_scale > 0.f);
    p.clamp_hi = d.act == EXB_ACT_RELU6 ? 6.f : INFINITY;
    if (!half_out) p.clamp_hi = fminf(p.clamp_hi * d.out_scale, 127.f);
    auto kern = clamp ? dw3x3_stream_kernel<TOut, S, true> : dw3x3_stream_kernel<TOut, S, false>;
    if (int rc = raise_smem_limit(ctx, kern)) return rc;
    return launch_pdl(ctx, "dw3x3_stream_kernel", kern, dim3((unsigned)grid), dim3((unsigned)pl.threads), smem, st, map, w->d_w, w->d_bias, y, p);
}

// Any window / stride: one output pixel x 8 channels per thread.
template <typename TIn, typename TOut>
__global__ void __launch_bounds__(128) dw_generic_kernel(const TIn* __restrict__ x, const float* __restrict__ w,
                                                         const float* __restrict__ bias, TOut* __restrict__ y,
                                                         DwParams p) {
    const int cvecs = p.cs / V;
    const int64_t total = (int64_t)p.N * p.OH * p.OW * cvecs;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += stride) {
        const int cv = (int)(idx % cvecs);
        int64_t t = idx / cvecs;
        const int ow = (int)(t % p.OW); t /= p.OW;
        const int oh = (int)(t % p.OH);
        const int n = (int)(t / p.OH);
        float acc[V];
        loadw(bias + cv * V, acc);
        for (int r = 0; r < p.kh; ++r) {
            const int ih = oh * p.sh - p.pt + r;
            if (ih < 0 || ih >= p.H) continue;
            for (int s = 0; s < p.kw; ++s) {
                const int iw = ow * p.sw - p.pl + s;
                if (iw < 0 || iw >= p.W) continue;
                float in[V], wv[V];
                load8(x + (((int64_t)n * p.H + ih) * p.W + iw) * p.cs + cv * V, in, p.in_scale);
                loadw(w + (int64_t)(r * p.kw + s) * p.cs + cv * V, wv);
#pragma unroll
                for (int k = 0; k < V; ++k) acc[k] = fmaf(in[k], wv[k], acc[k]);
            }
        }
        dw_act(acc, p, cv * V);
        store8(y + (((int64_t)n * p.OH + oh) * p.OW + ow) * p.cs + cv * V, acc, p.out_scale);
    }
}

template <typename TIn, typename TOut>
int launch(exb_ctx* ctx, const DwParams& p, const void* x, const exb_dw_weights* w, void* y, cudaStream_t st) {
    const TIn* xi = static_cast<const TIn*>(x);
    TOut* yo = static_cast<TOut*>(y);
    const int cvecs = p.cs / V;
    if (p.kh == 3 && p.kw == 3 && p.sh == p.sw && (p.sh == 1 || p.sh == 2)) {
        if constexpr (std::is_same<TIn, __half>::value) {
            const int rc = p.sh == 1 ? launch_stream<TOut, 1>(ctx, p, xi, w, yo, st) : launch_stream<TOut, 2>(ctx, p, xi, w, yo, st);
            if (rc != EXB_ERR_UNSUPPORTED) return rc;      // (more tiles than it counts: 2^30 and more tiny maps)
        } else {
            constexpr int TW = 4;
            const int64_t total = (int64_t)p.N * p.OH * ((p.OW + TW - 1) / TW) * cvecs;
            const int grid = stream_grid(ctx, total, 128, 16);
            if (p.sh == 1) dw_strip_kernel<TIn, TOut, 3, 1, TW><<<grid, 128, 0, st>>>(xi, w->d_w, w->d_bias, yo, p);
            else dw_strip_kernel<TIn, TOut, 3, 2, TW><<<grid, 128, 0, st>>>(xi, w->d_w, w->d_bias, yo, p);
            return after_launch("dw_strip_kernel");
        }
    }
    const int64_t total = (int64_t)p.N * p.OH * p.OW * cvecs;
    const int grid = stream_grid(ctx, total, 128, 16);
    dw_generic_kernel<TIn, TOut><<<grid, 128, 0, st>>>(xi, w->d_w, w->d_bias, yo, p);
    return after_launch("dw_generic_kernel");
}

int check_desc(const exb_dwconv_desc* d, int& cs, int& OH, int& OW) {
    EXB_REQUIRE(d != nullptr, "null depthwise descriptor");
    EXB_REQUIRE(d->N >= 0 && d->H > 0 && d->W > 0 && d->C > 0, "bad depthwise input shape");
    EXB_REQUIRE(d->kh > 0 && d->kw > 0 && d->stride_h > 0 && d->stride_w > 0, "bad depthwise window / stride");
    EXB_REQUIRE(d->pad_t >= 0 && d->pad_b >= 0 && d->pad_l >= 0 && d->pad_r >= 0, "negative pad");
    cs = d->c_stride ? d->c_stride : d->C;
    EXB_REQUIRE(cs >= d->C, "c_stride %d < C %d", cs, d->C);
    if (cs % V != 0) return fail(EXB_ERR_UNSUPPORTED, "depthwise conv needs the physical channel count (%d) to be a multiple of %d", cs, V);
    OH = (d->H + d->pad_t + d->pad_b - d->kh) / d->stride_h + 1;
    OW = (d->W + d->pad_l + d->pad_r - d->kw) / d->stride_w + 1;
    EXB_REQUIRE(OH > 0 && OW > 0, "depthwise window larger than the padded input");
    if (!act_supported(d->act) && d->act != EXB_ACT_PRELU)
        return fail(EXB_ERR_UNSUPPORTED, "activation type %d is not implemented", d->act);
    return EXB_OK;
}

}  // namespace
}  // namespace exb

using namespace exb;

extern "C" int exb_dw_weights_pack(exb_ctx* ctx, const exb_dwconv_desc* d, const float* w, const float* bias,
                                   exb_dw_weights** out) {
    EXB_REQUIRE(ctx && out && w, "exb_dw_weights_pack: null argument");
    *out = nullptr;
    int cs, OH, OW;
    if (int rc = check_desc(d, cs, OH, OW)) return rc;
    const int taps = d->kh * d->kw;
    float* hw = new float[(size_t)taps * cs]();
    float* hb = new float[cs]();
    for (int c = 0; c < d->C; ++c) {
        for (int t = 0; t < taps; ++t) hw[(size_t)t * cs + c] = w[(size_t)c * taps + t];
        if (bias) hb[c] = bias[c];
    }
    exb_dw_weights* pw = new exb_dw_weights();
    pw->C = d->C; pw->cs = cs; pw->kh = d->kh; pw->kw = d->kw; pw->device = ctx->device;
    pw->d_w = nullptr; pw->d_bias = nullptr; pw->d_slope = nullptr;
    cudaError_t e = cudaSetDevice(ctx->device);
    if (e == cudaSuccess) e = cudaMalloc(&pw->d_w, sizeof(float) * taps * cs);
    if (e == cudaSuccess) e = cudaMalloc(&pw->d_bias, sizeof(float) * cs);
    if (e == cudaSuccess) e = cudaMemcpy(pw->d_w, hw, sizeof(float) * taps * cs, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(pw->d_bias, hb, sizeof(float) * cs, cudaMemcpyHostToDevice);
    delete[] hw;
    delete[] hb;
    if (e != cudaSuccess) {
        exb_dw_weights_destroy(pw);
        return fail(EXB_ERR_CUDA, "exb_dw_weights_pack: %s", cudaGetErrorString(e));
    }
    *out = pw;
    return EXB_OK;
}

extern "C" int exb_dw_weights_destroy(exb_dw_weights* w) {
    if (!w) return EXB_OK;
    if (w->d_w) cudaFree(w->d_w);
    if (w->d_bias) cudaFree(w->d_bias);
    if (w->d_slope) cudaFree(w->d_slope);
    delete w;
    return EXB_OK;
}

extern "C" int exb_dwconv2d_fwd(exb_ctx* ctx, const exb_dwconv_desc* d, const void* x, const exb_dw_weights* w,
                                void* y, void* stream) {
    EXB_REQUIRE(ctx && w, "exb_dwconv2d_fwd: null argument");
    int cs, OH, OW;
    if (int rc = check_desc(d, cs, OH, OW)) return rc;
    EXB_REQUIRE(w->C == d->C && w->cs == cs && w->kh == d->kh && w->kw == d->kw,
                "exb_dwconv2d_fwd: packed weights do not match the descriptor");
    if (d->N == 0) return EXB_OK;
    EXB_REQUIRE(x && y && aligned16(x) && aligned16(y), "exb_dwconv2d_fwd: null or misaligned buffer");
    DwParams p;
    p.N = d->N; p.H = d->H; p.W = d->W; p.cs = cs; p.OH = OH; p.OW = OW;
    p.kh = d->kh; p.kw = d->kw; p.sh = d->stride_h; p.sw = d->stride_w; p.pt = d->pad_t; p.pl = d->pad_l;
    p.act = d->act; p.in_scale = d->in_scale; p.out_scale = d->out_scale;
    p.slope = w->d_slope;
    EXB_REQUIRE(p.act != EXB_ACT_PRELU || p.slope != nullptr, "exb_dwconv2d_fwd: EXB_ACT_PRELU without slopes (exb_dw_weights_set_slopes)");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (d->in_dtype == EXB_F16 && d->out_dtype == EXB_F16) return launch<__half, __half>(ctx, p, x, w, y, st);
    if (d->in_dtype == EXB_I8 && d->out_dtype == EXB_I8) return launch<int8_t, int8_t>(ctx, p, x, w, y, st);
    if (d->in_dtype == EXB_I8 && d->out_dtype == EXB_F16) return launch<int8_t, __half>(ctx, p, x, w, y, st);
    if (d->in_dtype == EXB_F16 && d->out_dtype == EXB_I8) return launch<__half, int8_t>(ctx, p, x, w, y, st);
    return fail(EXB_ERR_UNSUPPORTED, "depthwise conv dtypes in=%d out=%d", d->in_dtype, d->out_dtype);
}

extern "C" int exb_dw_weights_set_slopes(exb_ctx* ctx, exb_dw_weights* w, const float* slopes, int n) {
    EXB_REQUIRE(ctx != nullptr && w != nullptr && slopes != nullptr, "exb_dw_weights_set_slopes: null argument");
    EXB_REQUIRE(n == 1 || n == w->C, "exb_dw_weights_set_slopes: %d slopes for %d channels", n, w->C);
    float* h = new float[w->cs]();
    for (int c = 0; c < w->C; ++c) h[c] = slopes[n == 1 ? 0 : c];
    cudaError_t e = cudaSetDevice(w->device);
    if (e == cudaSuccess && !w->d_slope) e = cudaMalloc(&w->d_slope, sizeof(float) * w->cs);
    if (e == cudaSuccess) e = cudaMemcpy(w->d_slope, h, sizeof(float) * w->cs, cudaMemcpyHostToDevice);
    delete[] h;
    if (e != cudaSuccess) return fail(EXB_ERR_CUDA, "exb_dw_weights_set_slopes: %s", cudaGetErrorString(e));
    return EXB_OK;
}
