// Depthwise convolution on NHWC tensors, fp32 math on fp16 or int8 activations.
// A thread owns 8 consecutive channels of a strip of TW output pixels along W: every input
// vector of the strip is loaded once per kernel row and reused by all taps that touch it, and
// each weight vector is loaded once per strip.  Weights are kept tap-major [kh*kw][C] in fp32
// so consecutive threads read consecutive channels.
#include <math.h>

#include <type_traits>

#include "common.cuh"
#include "ptx_sm100.cuh"
#include "tensor_map.cuh"

namespace exb {
// How a streaming launch is cut: slab x column groups fill the threads of a CTA, R output rows are a tile.
struct DwStreamPlan {
    int N, OH, OW, S, sms;       // what it was made for
    int slab, groups, threads, tiles_w, R, ctas_per_sm;
};
}  // namespace exb

struct exb_dw_weights {
    float* d_w;     // [kh*kw][cs]
    float* d_bias;  // [cs] (zeros when the layer has no bias)
    float* d_slope; // [cs] PReLU slopes, or null
    int C, cs, kh, kw;
    int device;
    mutable std::mutex plan_mutex;
    mutable exb::DwStreamPlan plan;
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

// 3x3, stride 1 or 2, fp16 input: input rows stream through shared memory.
//
// A CTA owns a tile of 4 * groups output columns x R output rows x `slab` channels of one image.  One thread brings
// the input rows in with TMA, kStageRows at a time, two stages ahead of the arithmetic (zero fill outside the map is
// the padding); the ring runs on across the tiles of the persistent CTA.  A thread owns 4 channels x 4 output columns,
// keeps its 9 x 4 weights in registers for the whole launch and consumes an input row the moment it has read it: the
// row adds to the three output rows it belongs to (stride 2: one or two), so nothing but accumulators is carried from
// row to row.  Products are packed fma.rn.f32x2, each lane the same fma, in the same order, as a scalar loop's.
//
// Bound by HBM on large maps.  Loads that wait in registers (a thread keeping its own window of rows) left DRAM half
// idle: bytes in flight were limited by registers and stood still during the arithmetic.  Here 50-100 KB per SM are in
// flight whatever the threads do.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, const f32x2& c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 cvt2(uint32_t h) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h));
    return pack2(f.x, f.y);
}

constexpr int kDwCols = 4;          // output columns per thread
constexpr int kDwStages = 3;
constexpr int kDwThreads = 256;
template <int S> constexpr int kDwStageRows = S == 1 ? 3 : 2;
constexpr uint32_t kDwMaxSpins = 1u << 21;

struct DwStreamParams {
    int H, W, OH, OW, cs;
    int slab, units, groups;        // channels of a CTA, slab / 4, groups of kDwCols output columns
    int slabs, tiles_w, bands, tiles;
    int R, stages;                  // output rows per tile, stages per tile
    int in_w, row_bytes, slot_bytes;
    int pt, pl, act;
    float out_scale, clamp_hi;      // clamp_hi: upper bound of a ReLU / ReLU6 result (int8: of its multiple of out_scale)
    const float* slope;
    int* error;
};

// One output row of a thread: activation, conversion, store.  kClamp: ReLU or ReLU6.  Both are monotone with bounds that
// fp16 holds exactly, so an fp16 result is clamped after its rounding, two channels per instruction.
template <typename TOut, bool kClamp>
__device__ __forceinline__ void dw_store_row(const f32x2 (&acc)[kDwCols][2], TOut* y, int cs, int cols, const DwStreamParams& p, int c) {
    constexpr bool kHalf = std::is_same<TOut, __half>::value;
    if constexpr (kClamp && !kHalf) {
        // int8 behind ReLU / ReLU6: the bounds are applied to v * scale (a positive scale keeps the order, and both
        // forms round the same product), then 1.5 * 2^23 is added, which leaves the value rounded half to even in the
        // low byte: no float-to-integer conversions, whose quarter-rate pipe bounded this store (105 -> 91 us on 256
        // maps of 32 channels @112)
        const f32x2 s2 = pack2(p.out_scale, p.out_scale), magic = pack2(12582912.f, 12582912.f), one = pack2(1.f, 1.f), zero = pack2(-0.f, -0.f);
#pragma unroll
        for (int t = 0; t < kDwCols; ++t) {
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
    float v[4 * kDwCols];
#pragma unroll
    for (int t = 0; t < kDwCols; ++t)
#pragma unroll
        for (int h = 0; h < 2; ++h) asm("mov.b64 {%0, %1}, %2;" : "=f"(v[4 * t + 2 * h]), "=f"(v[4 * t + 2 * h + 1]) : "l"(acc[t][h]));
    if constexpr (kClamp) {
        // bounds below
    } else if (p.act == EXB_ACT_PRELU) {
        const float4 s = __ldg(reinterpret_cast<const float4*>(p.slope + c));
        const float sl[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
        for (int k = 0; k < 4 * kDwCols; ++k) v[k] = v[k] >= 0.f ? v[k] : v[k] * sl[k & 3];
    } else {
        apply_act_vec(v, p.act);
    }
    if constexpr (kHalf) {
        const __half2 zero = __half2half2(__ushort_as_half(0)), hi = __float2half2_rn(p.clamp_hi);
#pragma unroll
        for (int t = 0; t < kDwCols; ++t) {
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
        for (int t = 0; t < kDwCols; ++t)
            if (t < cols)
                *reinterpret_cast<uint32_t*>(y + t * cs) = quant_pack4(v[4 * t], v[4 * t + 1], v[4 * t + 2], v[4 * t + 3], p.out_scale);
    }
}

// acc = (first ? bias : acc) + the three taps of one kernel row on an input row
template <int S>
__device__ __forceinline__ void dw_taps(f32x2 (&acc)[kDwCols][2], int j, const f32x2 (&wv)[9][2], int krow, const f32x2 (&b2)[2],
                                        f32x2 v0, f32x2 v1) {
#pragma unroll
    for (int tc = 0; tc < kDwCols; ++tc) {
        const int sx = j - S * tc;
        if (sx < 0 || sx > 2) continue;
        const bool first = krow == 0 && sx == 0;
        acc[tc][0] = fma2(v0, wv[3 * krow + sx][0], first ? b2[0] : acc[tc][0]);
        acc[tc][1] = fma2(v1, wv[3 * krow + sx][1], first ? b2[1] : acc[tc][1]);
    }
}

template <typename TOut, int S, bool kClamp>
__global__ void __launch_bounds__(kDwThreads, 2)
    dw3x3_stream_kernel(const __grid_constant__ CUtensorMap map, const float* __restrict__ w, const float* __restrict__ bias,
                        TOut* __restrict__ y, const DwStreamParams p) {
    constexpr int RS = kDwStageRows<S>, IN = (kDwCols - 1) * S + 3;
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full[kDwStages];
    __shared__ int abort_flag;
    uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
    const int tid = threadIdx.x;
    pdl_launch_dependents();
    if (tid == 0) {
        abort_flag = 0;
        for (int i = 0; i < kDwStages; ++i) ptx::mbar_init(&full[i], 1);
        ptx::fence_mbar_init();
        ptx::tma_prefetch_desc(&map);
    }
    // the grid is a multiple of the slab count: a CTA keeps its channels, and a thread its weights, from tile to tile
    const int slab0 = (int)(blockIdx.x % p.slabs) * p.slab;
    const int u = tid % p.units, g = tid / p.units;
    const bool active = g < p.groups;
    const int c = slab0 + u * 4;
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

    // thread 0: next stage to request
    int it_tile = (int)blockIdx.x, it_stage = 0;
    auto request = [&](int slot) {
        if (it_tile >= p.tiles) return;
        int t = it_tile / p.slabs;
        const int tw = t % p.tiles_w;
        t /= p.tiles_w;
        const int band = t % p.bands, n = t / p.bands;
        const uint32_t bar = ptx::smem_u32(&full[slot]);
        ptx::mbar_arrive_expect_tx_u32(bar, (uint32_t)(RS * p.row_bytes));
        // stride 2: a stage is the rows (2k - 1, 2k) of the tile, the first row of stage 0 is never used
        ptx::tma_load_4d_u32(ptx::smem_u32(ring + (size_t)slot * p.slot_bytes), reinterpret_cast<uint64_t>(&map), bar, slab0,
                             tw * p.groups * kDwCols * S - p.pl, band * p.R * S - p.pt + it_stage * RS - (S == 2 ? 1 : 0), n);
        if (++it_stage == p.stages) {
            it_stage = 0;
            it_tile += gridDim.x;
        }
    };
    if (tid == 0)
        for (int i = 0; i < kDwStages - 1; ++i) request(i);

    const uint8_t* src0 = ring + ((size_t)g * kDwCols * S * p.slab + u * 4) * 2;
    const uint32_t px_bytes = (uint32_t)p.slab * 2;
    int slot = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int tile = (int)blockIdx.x; tile < p.tiles && ok; tile += gridDim.x) {
        int t = tile / p.slabs;
        const int tw = t % p.tiles_w;
        t /= p.tiles_w;
        const int band = t % p.bands, n = t / p.bands;
        const int oh0 = band * p.R, ow0 = (tw * p.groups + g) * kDwCols;
        const int cols = active ? min(kDwCols, p.OW - ow0) : 0;
        const int rows = min(p.R, p.OH - oh0);
        TOut* yo = y + (((int64_t)n * p.OH + oh0) * p.OW + ow0) * p.cs + c;
        const int64_t ypitch = (int64_t)p.OW * p.cs;
        // stride 1: three output rows are in the making; stride 2: one
        f32x2 acc[S == 1 ? 3 : 1][kDwCols][2];
#pragma unroll
        for (int a = 0; a < (S == 1 ? 3 : 1); ++a)
#pragma unroll
            for (int tc = 0; tc < kDwCols; ++tc) acc[a][tc][0] = b2[0], acc[a][tc][1] = b2[1];
        int o = S == 1 ? -2 : -1;           // output row that the next completed accumulator belongs to
        yo += o * ypitch;
        for (int st = 0; st < p.stages; ++st) {
            if (tid == 0) request(slot == 0 ? kDwStages - 1 : slot - 1);      // the slot read in the previous stage
            const bool got = ptx::mbar_wait_bounded(&full[slot], phase, &abort_flag, kDwMaxSpins);
            if (got && cols > 0) {
                const uint8_t* src = src0 + (size_t)slot * p.slot_bytes;
#pragma unroll
                for (int rr = 0; rr < RS; ++rr) {
                    uint2 rv[IN];
#pragma unroll
                    for (int j = 0; j < IN; ++j) rv[j] = *reinterpret_cast<const uint2*>(src + j * px_bytes);
                    src += p.row_bytes;
                    if constexpr (S == 1) {
                        // input row i = 3*st + rr is kernel row 0 of output row i, 1 of i - 1, 2 of i - 2 (which it completes)
#pragma unroll
                        for (int j = 0; j < IN; ++j) {
                            const f32x2 v0 = cvt2(rv[j].x), v1 = cvt2(rv[j].y);
                            dw_taps<S>(acc[rr], j, wv, 0, b2, v0, v1);
                            dw_taps<S>(acc[(rr + 2) % 3], j, wv, 1, b2, v0, v1);
                            dw_taps<S>(acc[(rr + 1) % 3], j, wv, 2, b2, v0, v1);
                        }
                        if (o >= 0 && o < rows) dw_store_row<TOut, kClamp>(acc[(rr + 1) % 3], yo, p.cs, cols, p, c);
                        ++o;
                        yo += ypitch;
                    } else if (rr == 0) {        // row 2k - 1: kernel row 1 of output row k - 1
#pragma unroll
                        for (int j = 0; j < IN; ++j) dw_taps<S>(acc[0], j, wv, 1, b2, cvt2(rv[j].x), cvt2(rv[j].y));
                    } else {                     // row 2k: kernel row 2 of output row k - 1, then kernel row 0 of row k
#pragma unroll
                        for (int j = 0; j < IN; ++j) dw_taps<S>(acc[0], j, wv, 2, b2, cvt2(rv[j].x), cvt2(rv[j].y));
                        if (o >= 0 && o < rows) dw_store_row<TOut, kClamp>(acc[0], yo, p.cs, cols, p, c);
                        ++o;
                        yo += ypitch;
#pragma unroll
                        for (int j = 0; j < IN; ++j) dw_taps<S>(acc[0], j, wv, 0, b2, cvt2(rv[j].x), cvt2(rv[j].y));
                    }
                }
            }
            // everybody has read the slot (it is requested again at the top of the next stage); a wait that ran out
            // takes all threads out together
            if (!__syncthreads_and(got)) {
                ok = false;
                break;
            }
            if (++slot == kDwStages) {
                slot = 0;
                phase ^= 1u;
            }
        }
    }
    if (!ok && tid == 0) {
        atomicExch(p.error, 4);
        for (int i = 0; i < 2000; ++i) __nanosleep(100);      // copies in flight land before the shared memory is handed on
    }
}

// The cut with the least modelled time, in SM cycles: what the whole SM has to issue and to move, plus twice the chain of
// the busiest CTA - rows one after the other, each a load, nine dependent fmas and a store, slower the more warps share
// the SM.  Constants fitted to 21 layers (batch 1 to 256, 7 x 7 to 112 x 112, 16 to 960 channels), about 80 cuts of each:
// the pick is within 3 % of the best cut on average, 19 % at worst.  Large maps get whole pixels (slab = all channels),
// small ones many small CTAs.  Rows of less than 128 bytes cost TMA and L2 about double.
template <int S>
DwStreamPlan dw_stream_plan(int sms, int N, int OH, int OW, int cs) {
    static const int kRows[2][8] = {{1, 4, 7, 10, 13, 16, 19, 28}, {1, 2, 3, 4, 7, 10, 14, 14}};   // stride 1: (R + 2) % 3 == 0
    DwStreamPlan best = {N, OH, OW, S, sms, 0, 0, 0, 0, 0, 0};
    double best_t = 1e30;
    const int cols = (OW + kDwCols - 1) / kDwCols;
    for (int slab = cs <= 256 ? cs : 256 / 8 * 8; slab >= 8; slab -= 8) {
        if (cs % slab) continue;
        const int units = slab / 4;
        const int gmax = kDwThreads / units < cols ? kDwThreads / units : cols;
        int prev_groups = 0;
        for (int tiles_w = (cols + gmax - 1) / gmax; tiles_w <= cols; ++tiles_w) {
            const int groups = (cols + tiles_w - 1) / tiles_w;
            const int in_w = (groups * kDwCols - 1) * S + 3;
            if (groups == prev_groups || in_w > 256) continue;
            prev_groups = groups;
            const int threads = (groups * units + 31) / 32 * 32;
            const int slot = (kDwStageRows<S> * in_w * slab * 2 + 127) / 128 * 128;
            const int smem = kDwStages * slot + 1024 + 256;
            int per_sm = 512 / threads;          // 128 registers per thread
            if (per_sm > 227 * 1024 / smem) per_sm = 227 * 1024 / smem;
            if (per_sm > 8) per_sm = 8;
            if (per_sm < 1) continue;
            for (int R : kRows[S - 1]) {
                const double bands = (OH + R - 1) / R;
                if (R > 1 && R >= OH + 3) break;
                const double rows = S == 1 ? R + 2 : 2 * (R + 1);
                const double tiles = (double)N * (cs / slab) * tiles_w * bands;
                const double per = tiles / sms;
                const double waves = ceil(per / per_sm);
                const double issue = per * rows * (S == 1 ? 75.0 : 56.0) * (threads / 32);
                const double mem = per * rows * slab * 2 * (in_w * (slab < 64 ? 2 : 1) + groups * kDwCols / (double)S) / 40.0;
                const double resident = per < 1 ? 1 : (per < per_sm ? per : per_sm);
                const double chain = waves * (rows * (300.0 + 7.0 * resident * (threads / 32)) + 800.0);
                const double t = (issue > mem ? issue : mem) + 2.0 * chain;
                if (t < best_t) {
                    best_t = t;
                    best.slab = slab; best.groups = groups; best.threads = threads; best.tiles_w = tiles_w; best.R = R;
                    best.ctas_per_sm = per_sm;
                }
            }
        }
    }
    return best;
}

template <typename TOut, int S>
int launch_stream(exb_ctx* ctx, const DwParams& d, const __half* x, const exb_dw_weights* w, TOut* y, cudaStream_t st) {
    auto encode = tensor_map_encoder();
    if (!encode) return fail(EXB_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    DwStreamPlan pl;
    {       // the cut for one shape is found once
        std::lock_guard<std::mutex> lock(w->plan_mutex);
        DwStreamPlan& k = w->plan;
        if (k.N != d.N || k.OH != d.OH || k.OW != d.OW || k.S != S || k.sms != ctx->sm_count) k = dw_stream_plan<S>(ctx->sm_count, d.N, d.OH, d.OW, d.cs);
        pl = k;
    }
    if (!pl.slab) return fail(EXB_ERR_UNSUPPORTED, "depthwise tile does not fit shared memory");
    DwStreamParams p;
    p.H = d.H; p.W = d.W; p.OH = d.OH; p.OW = d.OW; p.cs = d.cs;
    p.slab = pl.slab; p.units = pl.slab / 4; p.groups = pl.groups; p.slabs = d.cs / pl.slab; p.tiles_w = pl.tiles_w;
    p.R = pl.R; p.bands = (d.OH + pl.R - 1) / pl.R;
    p.stages = S == 1 ? (pl.R + 2) / 3 : pl.R + 1;
    const int64_t tiles = (int64_t)d.N * p.bands * p.tiles_w * p.slabs;
    if (tiles > INT32_MAX / 2) return fail(EXB_ERR_UNSUPPORTED, "depthwise tensor too large");
    p.tiles = (int)tiles;
    p.in_w = (pl.groups * kDwCols - 1) * S + 3;
    p.row_bytes = p.in_w * p.slab * 2;
    p.slot_bytes = (kDwStageRows<S> * p.row_bytes + 127) / 128 * 128;
    p.pt = d.pt; p.pl = d.pl; p.act = d.act; p.out_scale = d.out_scale; p.slope = d.slope; p.error = ctx->d_error;
    const bool half_out = std::is_same<TOut, __half>::value;
    const bool clamp = (d.act == EXB_ACT_RELU || d.act == EXB_ACT_RELU6) && (half_out || d.out_scale > 0.f);
    p.clamp_hi = d.act == EXB_ACT_RELU6 ? 6.f : INFINITY;
    if (!half_out) p.clamp_hi = fminf(p.clamp_hi * d.out_scale, 127.f);
    CUtensorMap map;
    cuuint64_t dims[4] = {(cuuint64_t)d.cs, (cuuint64_t)d.W, (cuuint64_t)d.H, (cuuint64_t)d.N};
    cuuint64_t strides[3] = {(cuuint64_t)d.cs * 2, (cuuint64_t)d.W * d.cs * 2, (cuuint64_t)d.H * d.W * d.cs * 2};
    cuuint32_t box[4] = {(cuuint32_t)p.slab, (cuuint32_t)p.in_w, (cuuint32_t)kDwStageRows<S>, 1};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    const CUresult r = encode(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<__half*>(x), dims, strides, box, estr,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(EXB_ERR_CUDA, "cuTensorMapEncodeTiled(depthwise) failed with %d", (int)r);
    auto kern = clamp ? dw3x3_stream_kernel<TOut, S, true> : dw3x3_stream_kernel<TOut, S, false>;
    if (int rc = raise_smem_limit(ctx, kern)) return rc;
    int grid = ctx->sm_count * pl.ctas_per_sm / p.slabs * p.slabs;
    if (grid < p.slabs) grid = p.slabs;
    if (grid > p.tiles) grid = p.tiles;
    return launch_pdl(ctx, "dw3x3_stream_kernel", kern, dim3((unsigned)grid), dim3((unsigned)pl.threads), (size_t)kDwStages * p.slot_bytes + 128, st,
                      map, w->d_w, w->d_bias, y, p);
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
            return p.sh == 1 ? launch_stream<TOut, 1>(ctx, p, xi, w, yo, st) : launch_stream<TOut, 2>(ctx, p, xi, w, yo, st);
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
    pw->plan = DwStreamPlan{};
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
