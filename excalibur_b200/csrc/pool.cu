// Max / average / global pooling on NHWC tensors.  Small square windows on fp16 maps stream input rows through shared
// memory; any other window or type takes the kernel in which one thread produces one 16-byte channel vector of one output
// pixel (8 fp16, 16 int8 or 4 fp32 channels).  Global pooling splits the map across the threads of a CTA, and across a
// cluster where that leaves SMs idle.
#include "common.cuh"
#include "host/known_divisor.hpp"
#include "row_stream.cuh"

#include <cooperative_groups.h>
#include <float.h>

#include <array>
#include <type_traits>

namespace exb {
namespace {

struct PoolParams {
    int N, H, W, C, cs;  // cs = physical channels
    int PH, PW;
    int type, kh, kw, sh, sw, pt, pb, pl, pr;
    int count_include_pad;
    float out2_scale;
};

template <typename T> struct PV;
template <> struct PV<__half> {
    static constexpr int N = 8;
    __device__ static void load(const __half* p, float (&v)[8]) {
        uint4 r = *reinterpret_cast<const uint4*>(p);
        const __half2* h = reinterpret_cast<const __half2*>(&r);
#pragma unroll
        for (int i = 0; i < 4; ++i) { float2 f = __half22float2(h[i]); v[2 * i] = f.x; v[2 * i + 1] = f.y; }
    }
    __device__ static void store(__half* p, const float (&v)[8]) {
        uint4 r;
        __half2* h = reinterpret_cast<__half2*>(&r);
#pragma unroll
        for (int i = 0; i < 4; ++i) h[i] = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
        *reinterpret_cast<uint4*>(p) = r;
    }
};
template <> struct PV<float> {
    static constexpr int N = 4;
    __device__ static void load(const float* p, float (&v)[4]) {
        float4 r = *reinterpret_cast<const float4*>(p);
        v[0] = r.x; v[1] = r.y; v[2] = r.z; v[3] = r.w;
    }
    __device__ static void store(float* p, const float (&v)[4]) {
        *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    }
};
template <> struct PV<int8_t> {
    static constexpr int N = 16;
    __device__ static void load(const int8_t* p, float (&v)[16]) {
        alignas(16) int8_t b[16];
        *reinterpret_cast<uint4*>(b) = *reinterpret_cast<const uint4*>(p);
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = (float)b[i];
    }
    __device__ static void store(int8_t* p, const float (&v)[16]) {
        alignas(16) int8_t b[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) b[i] = (int8_t)(int)v[i];
        *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(b);
    }
};

// Second output: int8 copy of V consecutive channels, q = sat8(rne(v * scale)).
template <int V>
__device__ __forceinline__ void store_q8(int8_t* p, const float (&v)[V], float scale) {
    alignas(16) int8_t b[V];
#pragma unroll
    for (int i = 0; i < V; ++i) b[i] = (int8_t)quant_rne(v[i] * scale);
    if (V == 8) *reinterpret_cast<uint2*>(p) = *reinterpret_cast<const uint2*>(b);
    else if (V == 4) *reinterpret_cast<uint32_t*>(p) = *reinterpret_cast<const uint32_t*>(b);
    else *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(b);
}

template <typename T, bool kOut2>
__global__ void __launch_bounds__(256) pool_kernel(const T* __restrict__ x, T* __restrict__ y,
                                                   int8_t* __restrict__ y2, PoolParams p) {
    constexpr int V = PV<T>::N;
    const int cvecs = p.cs / V;
    const int64_t total = (int64_t)p.N * p.PH * p.PW * cvecs;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    pdl_wait();
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += stride) {
        int cv, pw, ph, n;
        if (total <= 0xffffffffll) {      // 32-bit divisions cost a fifth of 64-bit ones
            uint32_t t = (uint32_t)idx;
            cv = (int)(t % (uint32_t)cvecs); t /= (uint32_t)cvecs;
            pw = (int)(t % (uint32_t)p.PW); t /= (uint32_t)p.PW;
            ph = (int)(t % (uint32_t)p.PH);
            n = (int)(t / (uint32_t)p.PH);
        } else {
            cv = (int)(idx % cvecs);
            int64_t t = idx / cvecs;
            pw = (int)(t % p.PW); t /= p.PW;
            ph = (int)(t % p.PH);
            n = (int)(t / p.PH);
        }
        int hs = ph * p.sh - p.pt, ws = pw * p.sw - p.pl;
        float acc[V];
        if (p.type == 0) {
            const int he = min(hs + p.kh, p.H), we = min(ws + p.kw, p.W);
            hs = max(hs, 0); ws = max(ws, 0);
#pragma unroll
            for (int k = 0; k < V; ++k) acc[k] = -FLT_MAX;
            for (int h = hs; h < he; ++h)
                for (int w = ws; w < we; ++w) {
                    float v[V];
                    PV<T>::load(x + (((int64_t)n * p.H + h) * p.W + w) * p.cs + cv * V, v);
#pragma unroll
                    for (int k = 0; k < V; ++k) acc[k] = fmaxf(acc[k], v[k]);
                }
        } else {
            int he = min(hs + p.kh, p.H + p.pb), we = min(ws + p.kw, p.W + p.pr);
            int pool_size = (he - hs) * (we - ws);
            hs = max(hs, 0); ws = max(ws, 0);
            he = min(he, p.H); we = min(we, p.W);
            if (p.count_include_pad == 0) pool_size = (he - hs) * (we - ws);
#pragma unroll
            for (int k = 0; k < V; ++k) acc[k] = 0.f;
            for (int h = hs; h < he; ++h)
                for (int w = ws; w < we; ++w) {
                    float v[V];
                    PV<T>::load(x + (((int64_t)n * p.H + h) * p.W + w) * p.cs + cv * V, v);
#pragma unroll
                    for (int k = 0; k < V; ++k) acc[k] += v[k];
                }
            const float div = (float)pool_size;
#pragma unroll
            for (int k = 0; k < V; ++k) acc[k] = acc[k] / div;
        }
        const int64_t o = (((int64_t)n * p.PH + ph) * p.PW + pw) * p.cs + cv * V;
        PV<T>::store(y + o, acc);
        if (kOut2) store_q8<V>(y2 + o, acc, p.out2_scale);
    }
}

// Global pooling: grid = (blocks of cw channel vectors, N, splits of the map), 256 threads = cw vectors x rows of pixels.
// A thread keeps eight loads in flight (one at a time, 3 maps of 32 channels @100x90 took 205 us, now 6: every load a round trip to HBM); the rows
// meet in shared memory, the splits - a cluster, used when image count and channels alone leave SMs idle - in the first
// CTA's, through distributed shared memory.
template <typename T, bool kOut2>
__global__ void __launch_bounds__(256, 4) global_pool_kernel(const T* __restrict__ x, T* __restrict__ y,
                                                          int8_t* __restrict__ y2, PoolParams p, int cw, int splits) {
    constexpr int V = PV<T>::N, kUnroll = 8;
    __shared__ float part[256][V + 1];
    pdl_launch_dependents();
    const int cvecs = p.cs / V;
    const int tid = threadIdx.x, row = tid / cw, rows = 256 / cw;
    const int cv = blockIdx.x * cw + tid % cw;
    const int n = blockIdx.y;
    const int HW = p.H * p.W;
    const bool active = row < rows && cv < cvecs;
    float acc[V];
#pragma unroll
    for (int k = 0; k < V; ++k) acc[k] = p.type == 0 ? -FLT_MAX : 0.f;
    auto combine = [&](const float (&v)[V]) {
#pragma unroll
        for (int k = 0; k < V; ++k) acc[k] = p.type == 0 ? fmaxf(acc[k], v[k]) : acc[k] + v[k];
    };
    pdl_wait();
    if (active) {
        const T* src = x + (int64_t)n * HW * p.cs + cv * V;
        const int step = rows * splits;
        int i = (int)blockIdx.z * rows + row;
        for (; i < HW; i += kUnroll * step) {
            uint4 raw[kUnroll];
#pragma unroll
            for (int u = 0; u < kUnroll; ++u)
                if (i + u * step < HW) raw[u] = *reinterpret_cast<const uint4*>(src + (int64_t)(i + u * step) * p.cs);
#pragma unroll
            for (int u = 0; u < kUnroll; ++u)
                if (i + u * step < HW) {
                    float v[V];
                    PV<T>::load(reinterpret_cast<const T*>(&raw[u]), v);
                    combine(v);
                }
        }
    }
    for (int left = rows; left > 1;) {
        const int half = (left + 1) / 2;
        if (row >= half && row < left)
#pragma unroll
            for (int k = 0; k < V; ++k) part[tid][k] = acc[k];
        __syncthreads();
        if (row + half < left)
#pragma unroll
            for (int k = 0; k < V; ++k) {
                const float o = part[tid + half * cw][k];
                acc[k] = p.type == 0 ? fmaxf(acc[k], o) : acc[k] + o;
            }
        left = half;
    }
    if (splits > 1) {
        cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
        __syncthreads();        // the rows' exchange is over
        if (row == 0 && blockIdx.z != 0)
#pragma unroll
            for (int k = 0; k < V; ++k) part[tid][k] = acc[k];
        cluster.sync();
        if (row == 0 && blockIdx.z == 0)
            for (int s = 1; s < splits; ++s) {
                const float* other = cluster.map_shared_rank(&part[tid][0], s);
#pragma unroll
                for (int k = 0; k < V; ++k) acc[k] = p.type == 0 ? fmaxf(acc[k], other[k]) : acc[k] + other[k];
            }
        cluster.sync();         // no CTA leaves while its shared memory may be read
        if (blockIdx.z != 0) return;
    }
    if (row == 0 && cv < cvecs) {
        if (p.type == 1) {
            const float div = (float)HW;
#pragma unroll
            for (int k = 0; k < V; ++k) acc[k] = acc[k] / div;
        }
        const int64_t o = (int64_t)n * p.cs + cv * V;
        PV<T>::store(y + o, acc);
        if (kOut2) store_q8<V>(y2 + o, acc, p.out2_scale);
    }
}

__device__ __forceinline__ uint32_t hmax2_u32(uint32_t a, uint32_t b) {
    __half2 r = __hmax2(*reinterpret_cast<__half2*>(&a), *reinterpret_cast<__half2*>(&b));
    return *reinterpret_cast<uint32_t*>(&r);
}

// Small square windows on fp16 maps, on the row stream of row_stream.cuh: 2x2/2, 3x3/1, 3x3/2 and 5x5/1.  An input row is
// reduced along W first (four columns share its vectors), then combined into the output rows it belongs to.  Maxima are
// packed half2; padding is the tensor map's NaN fill, which a maximum ignores.  Averages add in fp32.  The kernel with a
// thread per output vector read each input vector K * K times and divided 64-bit indices for each of them.
// 5x5/1, 24 maps of 256 channels @45x39: 62 -> 12 us; 3x3/2, 256 maps of 64 channels @112: 127 -> 84 us = 94 % of the HBM
// copy rate (a former kernel of its own, 2x2 outputs per thread).
constexpr uint32_t kNegInf2 = 0xFC00FC00u;       // (-inf, -inf) in fp16
struct PoolStreamParams : RowStreamParams {
    int H, W, pt, pb, pl, pr, count_include_pad;
    float out2_scale;
    // Averages: the divisors 1 to 25.  A window outside the map has a sum of 0 and any other: NaN for 0, else 0.
    KnownDivisor count[kMaxKnownDivisor + 2];
};
template <int K, int S> constexpr RowStreamKind kPoolKind = {
    100 + 10 * K + S, S, K, S == 1 ? K : 2, K == 5 ? 2 : 3, K == 3 && S == 2 ? 1 : 0, 15.0 + 8.0 * K / S};

// One output row of a thread to memory.
template <bool kOut2>
__device__ __forceinline__ void pool_store_row(const uint2 (&v)[kRowCols], const uint32_t (&q)[kRowCols], __half* y, int8_t* y2, int64_t off, int cs,
                                               int cols) {
#pragma unroll
    for (int t = 0; t < kRowCols; ++t) {
        if (t >= cols) continue;
        *reinterpret_cast<uint2*>(y + off + t * cs) = v[t];
        if (kOut2) *reinterpret_cast<uint32_t*>(y2 + off + t * cs) = q[t];
    }
}

template <int K, int S, bool kMax, bool kOut2>
__global__ void __launch_bounds__(kRowThreads, 2)
    pool_stream_kernel(const __grid_constant__ CUtensorMap map, __half* __restrict__ y, int8_t* __restrict__ y2, const PoolStreamParams p) {
    constexpr RowStreamKind kind = kPoolKind<K, S>;
    constexpr int IN = (kRowCols - 1) * S + K, A = S == 1 ? K : 1;
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full[kind.NS];
    __shared__ int abort_flag;
    uint8_t* ring = row_stream_init<kind.NS>(map, smem_raw, full, &abort_flag);
    __syncthreads();
    pdl_wait();
    const int c = (int)(blockIdx.x % p.slabs) * p.slab + (int)(threadIdx.x % p.units) * 4;
    const int64_t ypitch = (int64_t)p.OW * p.cs;
    using Acc = typename std::conditional<kMax, uint32_t, f32x2>::type;
    Acc acc[A][kRowCols][2];
    auto combine = [](Acc a, Acc b) -> Acc {
        if constexpr (kMax) return hmax2_u32(a, b);
        else return add2(a, b);
    };
    RowTile t;
    int64_t off = 0;
    int o = 0;                          // output row that the next completed accumulator belongs to
    auto finish = [&](const Acc (&a)[kRowCols][2]) {
        if (o >= 0 && o < t.rows) {
            uint2 v[kRowCols];
            uint32_t q[kRowCols];
            if constexpr (kMax) {
                // a window of nothing but padding or NaN has the maximum of no values
#pragma unroll
                for (int k = 0; k < kRowCols; ++k) {
                    v[k] = make_uint2(hmax2_u32(a[k][0], kNegInf2), hmax2_u32(a[k][1], kNegInf2));
                    if (kOut2) {
                        const float2 lo = __half22float2(*reinterpret_cast<const __half2*>(&v[k].x)), hi = __half22float2(*reinterpret_cast<const __half2*>(&v[k].y));
                        q[k] = quant_pack4(lo.x, lo.y, hi.x, hi.y, p.out2_scale);
                    }
                }
            } else {
                const int hs = (t.oh0 + o) * S - p.pt, he = min(hs + K, p.H + p.pb);
                const int hc = p.count_include_pad ? he - hs : min(he, p.H) - max(hs, 0);
#pragma unroll
                for (int k = 0; k < kRowCols; ++k) {
                    const int ws = (t.ow0 + k) * S - p.pl, we = min(ws + K, p.W + p.pr);
                    const int d = hc * (p.count_include_pad ? we - ws : min(we, p.W) - max(ws, 0));
                    float f[4];
                    unpack2(a[k][0], f[0], f[1]);
                    unpack2(a[k][1], f[2], f[3]);
                    // 16 quotients a thread and row: as divisions they took 2x2/2 at 4 x 60 x 92 x 128 from 9.0 to 14.3 us
                    const KnownDivisor kd = p.count[min((unsigned)d, (unsigned)kMaxKnownDivisor + 1)];
#pragma unroll
                    for (int i = 0; i < 4; ++i) f[i] = divide_by(f[i], kd);
                    const __half2 h0 = __floats2half2_rn(f[0], f[1]), h1 = __floats2half2_rn(f[2], f[3]);
                    v[k] = make_uint2(*reinterpret_cast<const uint32_t*>(&h0), *reinterpret_cast<const uint32_t*>(&h1));
                    if (kOut2) {       // of the fp32 average, by quant_rne as in the other kernel: NaN is the lowest value
                        q[k] = 0;
#pragma unroll
                        for (int i = 0; i < 4; ++i) q[k] |= (uint32_t)(uint8_t)quant_rne(f[i] * p.out2_scale) << (8 * i);
                    }
                }
            }
            pool_store_row<kOut2>(v, q, y, y2, off, p.cs, t.cols);
        }
        ++o;
        off += ypitch;
    };
    row_stream_run<S, K, kind.RS, kind.NS, false>(
        map, p, ring, full, &abort_flag,
        [&](const RowTile& tile) {
            t = tile;
            o = S == 1 ? 1 - K : (K == 3 ? -1 : 0);
            off = (((int64_t)t.n * p.OH + t.oh0 + o) * p.OW + t.ow0) * p.cs + c;
#pragma unroll
            for (int a = 0; a < A; ++a)
#pragma unroll
                for (int k = 0; k < kRowCols; ++k) acc[a][k][0] = acc[a][k][1] = kMax ? (Acc)kNegInf2 : (Acc)0;
        },
        [&](const int rr, const uint2 (&rv)[IN]) {
            Acc h[kRowCols][2];
            if constexpr (kMax) {
#pragma unroll
                for (int k = 0; k < kRowCols; ++k) {
                    h[k][0] = rv[k * S].x;
                    h[k][1] = rv[k * S].y;
#pragma unroll
                    for (int j = 1; j < K; ++j) {
                        h[k][0] = hmax2_u32(h[k][0], rv[k * S + j].x);
                        h[k][1] = hmax2_u32(h[k][1], rv[k * S + j].y);
                    }
                }
            } else {
                f32x2 f[IN][2];
#pragma unroll
                for (int j = 0; j < IN; ++j) f[j][0] = cvt2(rv[j].x), f[j][1] = cvt2(rv[j].y);
#pragma unroll
                for (int k = 0; k < kRowCols; ++k)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        h[k][e] = f[k * S][e];
#pragma unroll
                        for (int j = 1; j < K; ++j) h[k][e] = add2(h[k][e], f[k * S + j][e]);
                    }
            }
            auto into = [&](Acc (&a)[kRowCols][2], bool first) {
#pragma unroll
                for (int k = 0; k < kRowCols; ++k)
#pragma unroll
                    for (int e = 0; e < 2; ++e) a[k][e] = first ? h[k][e] : combine(a[k][e], h[k][e]);
            };
            if constexpr (S == 1) {      // input row i is row a of the window of output row i - a; it completes i - K + 1
#pragma unroll
                for (int a = 0; a < K; ++a) into(acc[(rr + K - a) % K], a == 0);
                finish(acc[(rr + 1) % K]);
            } else if constexpr (K == 2) {
                into(acc[0], rr == 0);
                if (rr == 1) finish(acc[0]);
            } else {                     // rows 2k - 1 and 2k: the second ends output row k - 1 and begins row k
                into(acc[0], false);
                if (rr == 1) {
                    finish(acc[0]);
                    into(acc[0], true);
                }
            }
        });
}

template <int K, int S, bool kMax, bool kOut2>
int launch_pool_stream(exb_ctx* ctx, const PoolParams& d, const __half* x, __half* y, int8_t* y2, cudaStream_t st) {
    static constexpr RowStreamKind kind = kPoolKind<K, S>;
    const RowStreamPlan pl = row_stream_plan(kind, ctx->sm_count, d.N, d.PH, d.PW, d.cs);
    PoolStreamParams p{};
    CUtensorMap map;
    size_t smem;
    const int grid = row_stream_setup(ctx, kind, pl, x, d.N, d.H, d.W, d.pt, d.pl,
                                      kMax ? CU_TENSOR_MAP_FLOAT_OOB_FILL_NAN_REQUEST_ZERO_FMA : CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE, p, map, smem);
    if (grid < 0) return grid;
    p.H = d.H; p.W = d.W; p.pt = d.pt; p.pb = d.pb; p.pl = d.pl; p.pr = d.pr;
    p.count_include_pad = d.count_include_pad; p.out2_scale = d.out2_scale;
    if (!kMax) {
        static const std::array<KnownDivisor, kMaxKnownDivisor + 2> table = [] {
            std::array<KnownDivisor, kMaxKnownDivisor + 2> t;
            t.front() = {NAN, NAN};
            for (int i = 1; i <= kMaxKnownDivisor; ++i) t[i] = known_divisor(i);
            t.back() = {0.f, 0.f};
            return t;
        }();
        memcpy(p.count, table.data(), sizeof(p.count));
    }
    auto kern = pool_stream_kernel<K, S, kMax, kOut2>;
    if (int rc = raise_smem_limit(ctx, kern)) return rc;
    return launch_pdl(ctx, "pool_stream_kernel", kern, dim3((unsigned)grid), dim3((unsigned)pl.threads), smem, st, map, y, y2, p);
}

template <int K, int S>
int launch_pool_stream(exb_ctx* ctx, const PoolParams& d, const void* x, void* y, void* y2, bool out2, cudaStream_t st) {
    const __half* xi = static_cast<const __half*>(x);
    __half* yo = static_cast<__half*>(y);
    int8_t* qo = static_cast<int8_t*>(y2);
    if (d.type == 0) return out2 ? launch_pool_stream<K, S, true, true>(ctx, d, xi, yo, qo, st) : launch_pool_stream<K, S, true, false>(ctx, d, xi, yo, nullptr, st);
    return out2 ? launch_pool_stream<K, S, false, true>(ctx, d, xi, yo, qo, st) : launch_pool_stream<K, S, false, false>(ctx, d, xi, yo, nullptr, st);
}

int pool_dim(int in, int pa, int pb, int k, int s, int pad_mode) {
    // static_cast<int>(ceil|floor(static_cast<float>(in + pa + pb - k) / s)) + 1
    float q = (float)(in + pa + pb - k) / (float)s;
    return (int)(pad_mode == 0 ? ceilf(q) : floorf(q)) + 1;
}

template <typename T>
int launch(exb_ctx* ctx, const exb_pool_desc* d, const PoolParams& p, const void* x, void* y, void* y2,
           cudaStream_t st) {
    constexpr int V = PV<T>::N;
    if (p.cs % V != 0)
        return fail(EXB_ERR_UNSUPPORTED, "pooling needs the physical channel count (%d) to be a multiple of %d for this dtype", p.cs, V);
    const bool out2 = d->out2_dtype == EXB_I8;
    if (d->global_pool) {
        EXB_REQUIRE(p.N <= 65535, "batch %d exceeds the grid limit of global pooling", p.N);
        const int cvecs = p.cs / V, blocks = (cvecs + 31) / 32, cw = (cvecs + blocks - 1) / blocks, rows = 256 / cw;
        int splits = 1;         // until there are two CTAs per SM, as long as a thread keeps a round of loads
        while (splits < 8 && (int64_t)blocks * p.N * splits < 2 * ctx->sm_count && p.H * p.W >= 8 * rows * splits) splits *= 2;
        const dim3 grid(blocks, p.N, splits);
        const T* xi = static_cast<const T*>(x);
        if (out2) return launch_pdl_cluster(ctx, "global_pool_kernel", global_pool_kernel<T, true>, grid, dim3(256), dim3(1, 1, (unsigned)splits), 0, st, xi, static_cast<T*>(y), static_cast<int8_t*>(y2), p, cw, splits);
        return launch_pdl_cluster(ctx, "global_pool_kernel", global_pool_kernel<T, false>, grid, dim3(256), dim3(1, 1, (unsigned)splits), 0, st, xi, static_cast<T*>(y), nullptr, p, cw, splits);
    }
    // The row stream needs rows of 64 bytes for its boxes where a window shares little with its neighbours (stride 2):
    // below 32 channels the kernel with a thread per output vector is 1.2-1.4 times as fast (64 maps @50x51, 16 and 24
    // channels: 4.8-5.4 against 6.2-7.1 us); with stride 1 the stream wins at every width.
    if (std::is_same<T, __half>::value && p.kh == p.kw && p.sh == p.sw) {
        int rc = EXB_ERR_UNSUPPORTED;       // also the answer to more tiles than the stream counts: 2^30 and more tiny maps
        if (p.kh == 5 && p.sh == 1) rc = launch_pool_stream<5, 1>(ctx, p, x, y, y2, out2, st);
        else if (p.kh == 3 && p.sh == 1) rc = launch_pool_stream<3, 1>(ctx, p, x, y, y2, out2, st);
        else if (p.kh == 3 && p.sh == 2 && p.cs >= 32) rc = launch_pool_stream<3, 2>(ctx, p, x, y, y2, out2, st);
        else if (p.kh == 2 && p.sh == 2 && p.cs >= 32) rc = launch_pool_stream<2, 2>(ctx, p, x, y, y2, out2, st);
        if (rc != EXB_ERR_UNSUPPORTED) return rc;
    }
    const int64_t total = (int64_t)p.N * p.PH * p.PW * (p.cs / V);
    const dim3 grid((unsigned)stream_grid(ctx, total, 256));
    const T* xi = static_cast<const T*>(x);
    if (out2) return launch_pdl(ctx, "pool_kernel", pool_kernel<T, true>, grid, dim3(256), 0, st, xi, static_cast<T*>(y), static_cast<int8_t*>(y2), p);
    return launch_pdl(ctx, "pool_kernel", pool_kernel<T, false>, grid, dim3(256), 0, st, xi, static_cast<T*>(y), nullptr, p);
}

int fill_params(const exb_pool_desc* d, PoolParams& p) {
    EXB_REQUIRE(d != nullptr, "null pooling descriptor");
    EXB_REQUIRE(d->N >= 0 && d->H > 0 && d->W > 0 && d->C > 0, "bad pooling input shape");
    EXB_REQUIRE(d->type == 0 || d->type == 1, "unknown pooling method %d", d->type);
    EXB_REQUIRE(d->pad_mode == 0 || d->pad_mode == 1, "pad_mode %d is not implemented", d->pad_mode);
    p.N = d->N; p.H = d->H; p.W = d->W; p.C = d->C;
    p.cs = d->c_stride ? d->c_stride : d->C;
    EXB_REQUIRE(p.cs >= p.C, "c_stride %d < C %d", p.cs, p.C);
    p.type = d->type;
    if (d->global_pool) {
        p.kh = d->H; p.kw = d->W; p.sh = p.sw = 1; p.pt = p.pb = p.pl = p.pr = 0;
    } else {
        p.kh = d->kh; p.kw = d->kw; p.sh = d->stride_h; p.sw = d->stride_w;
        p.pt = d->pad_t; p.pb = d->pad_b; p.pl = d->pad_l; p.pr = d->pad_r;
    }
    EXB_REQUIRE(p.kh > 0 && p.kw > 0 && p.sh > 0 && p.sw > 0, "bad pooling window / stride");
    EXB_REQUIRE(p.pt >= 0 && p.pb >= 0 && p.pl >= 0 && p.pr >= 0, "negative pooling pad");
    p.PH = pool_dim(p.H, p.pt, p.pb, p.kh, p.sh, d->pad_mode);
    p.PW = pool_dim(p.W, p.pl, p.pr, p.kw, p.sw, d->pad_mode);
    EXB_REQUIRE(p.PH > 0 && p.PW > 0, "pooling window larger than the padded input");
    p.count_include_pad = d->count_include_pad;
    p.out2_scale = d->out2_scale;
    return EXB_OK;
}

}  // namespace
}  // namespace exb

using namespace exb;

extern "C" int exb_pool_out_dims(const exb_pool_desc* d, int* PH, int* PW) {
    PoolParams p;
    if (int rc = fill_params(d, p)) return rc;
    EXB_REQUIRE(PH && PW, "null output pointer");
    *PH = p.PH;
    *PW = p.PW;
    return EXB_OK;
}

extern "C" int exb_pool2d_fwd(exb_ctx* ctx, const exb_pool_desc* d, const void* x, void* y, void* y2,
                              void* stream) {
    EXB_REQUIRE(ctx != nullptr, "null context");
    PoolParams p;
    if (int rc = fill_params(d, p)) return rc;
    if (p.N == 0) return EXB_OK;
    EXB_REQUIRE(x && y, "exb_pool2d_fwd: null buffer");
    EXB_REQUIRE(aligned16(x) && aligned16(y), "exb_pool2d_fwd: buffers must be 16-byte aligned");
    if (d->out2_dtype != -1) {
        if (d->out2_dtype != EXB_I8) return fail(EXB_ERR_UNSUPPORTED, "pooling second output must be EXB_I8");
        EXB_REQUIRE(y2 && aligned16(y2), "exb_pool2d_fwd: second output null or misaligned");
    }
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    switch (d->dtype) {
    case EXB_F16: return launch<__half>(ctx, d, p, x, y, y2, st);
    case EXB_F32: return launch<float>(ctx, d, p, x, y, y2, st);
    case EXB_I8:
        if (d->type != 0) return fail(EXB_ERR_UNSUPPORTED, "int8 pooling supports max only");
        if (d->out2_dtype != -1) return fail(EXB_ERR_UNSUPPORTED, "int8 pooling has no second output");
        return launch<int8_t>(ctx, d, p, x, y, y2, st);
    default: return fail(EXB_ERR_UNSUPPORTED, "pooling dtype %d", d->dtype);
    }
}
