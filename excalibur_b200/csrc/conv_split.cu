// Implicit-GEMM convolution for problems of few tiles (small batches, deep layers): every output tile is worked on by a
// cluster of CTAs that share its reduction dimension.
//
// The persistent kernel of conv_tc.cu gives a tile to one CTA (or pair): with one image a 3x3 layer of 512 channels @7x7
// is two tiles, and one warp issues the whole reduction - 144 dependent MMAs and the loads that feed them, 19 us
// (int8), on two of 148 SMs.  Here N tiles are at most 64 channels and the K blocks of a tile are divided over a cluster
// of 1, 2, 4 or 8 CTAs.  Each accumulates its part in TMEM and spills it to its shared memory; after a cluster barrier
// every CTA sums one slice of the tile's pixels over all parts through distributed shared memory and runs the epilogue
// for that slice.  Weights never change on the stream, so their first loads are issued before the programmatic wait for
// the previous kernel; what remains after that wait is one activation load, the MMAs of a few K blocks, the exchange and
// the store.  int8 sums are exact whatever the split; fp16 ones are fp32 sums of at most eight partial sums.
#include "conv_tc_host.cuh"
#include "ptx_sm100.cuh"

#include <math.h>

namespace exb {
namespace {

constexpr int kSplitStages = 16;     // at most
constexpr int kSplitEpiThreads = 256;
constexpr int kSplitThreads = 64 + kSplitEpiThreads;      // warp 0 loads, warp 1 issues MMAs, warps 2-9 drain and store
constexpr int kSplitMaxItems = kTileM * 8 / kSplitEpiThreads;      // of 8 channels, with 64 channels per tile
constexpr uint32_t kSplitMaxSpins = 1u << 21;

struct ConvSplitParams {
    CUtensorMap tmA[4];
    CUtensorMap tmB;
    int N, OH, OW;
    int TW, TH, TN;
    int tiles_w, tiles_h, n_tiles;      // pixel tiles along W and H, channel tiles (image groups are what is left)
    int BN, splits;
    int kw, stride, pad_t, pad_l;
    int cin_pad, cblks, kb_elems, kb_bytes;
    int k_iters;                        // (tap, channel block) pairs; CTA r of a cluster takes [r*k/splits, (r+1)*k/splits)
    int stages, a_bytes, b_bytes, a_tx_bytes;
    int tmem_cols, cout_pad, has_res;
    int res_half;           // the residual is read through a nearest resize by 2
    uint32_t idesc;
    EpiParams e;
    int* error;
};

__device__ __forceinline__ uint4 ld_cluster_16(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared::cluster.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr) : "memory");
    return v;
}

template <bool kInt8>
__device__ __forceinline__ void acc_add(uint4& a, const uint4& b) {
    if (kInt8) {
        a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
    } else {
        a.x = __float_as_uint(__uint_as_float(a.x) + __uint_as_float(b.x));
        a.y = __float_as_uint(__uint_as_float(a.y) + __uint_as_float(b.y));
        a.z = __float_as_uint(__uint_as_float(a.z) + __uint_as_float(b.z));
        a.w = __float_as_uint(__uint_as_float(a.w) + __uint_as_float(b.w));
    }
}

template <bool kInt8, bool kPrelu>
__global__ void __launch_bounds__(kSplitThreads) conv_split_kernel(const __grid_constant__ ConvSplitParams p) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[kSplitStages];
    __shared__ __align__(8) uint64_t empty_bar[kSplitStages];
    __shared__ __align__(8) uint64_t done_bar;
    __shared__ __align__(16) float s_scale[64];
    __shared__ __align__(16) float s_bias[64];
    __shared__ int s_pixel[kTileM], s_res_pixel[kTileM];
    __shared__ uint32_t tmem_base_smem;
    __shared__ int abort_flag;
    // operand ring (1024-byte aligned: the widest swizzle atom); the partial tile takes its place when the MMAs are done
    uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int warp = ptx::uniform_warp(), lane = threadIdx.x & 31;
    const int rank = (int)blockIdx.x % p.splits;
    int t = (int)blockIdx.x / p.splits;
    const int ntile = t % p.n_tiles;
    t /= p.n_tiles;
    const int ow0 = t % p.tiles_w * p.TW;
    t /= p.tiles_w;
    const int oh0 = t % p.tiles_h * p.TH, n0 = t / p.tiles_h * p.TN;
    const int k0 = rank * p.k_iters / p.splits, units = (rank + 1) * p.k_iters / p.splits - k0;
    const int c0 = ntile * p.BN;

    pdl_launch_dependents();
    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (int s = 0; s < p.stages; ++s) {
            ptx::mbar_init(&full_bar[s], 1);
            ptx::mbar_init(&empty_bar[s], 1);
        }
        ptx::mbar_init(&done_bar, 1);
        ptx::fence_mbar_init();
        ptx::tma_prefetch_desc(&p.tmB);
        ptx::tma_prefetch_desc(&p.tmA[0]);
    }
    if (warp == 1) {
        ptx::tmem_alloc(&tmem_base_smem, (uint32_t)p.tmem_cols);
        ptx::tmem_relinquish();
    }
    if (threadIdx.x >= 64 && threadIdx.x < 64 + p.BN) {
        const int c = (int)threadIdx.x - 64, ch = c0 + c;
        s_scale[c] = ch < p.cout_pad ? p.e.scale[ch] : 0.f;
        s_bias[c] = ch < p.cout_pad ? p.e.bias[ch] : 0.f;
    }
    if (warp >= 2 && warp < 6) {       // accumulator row -> pixel of the output, or -1
        const int row = (int)threadIdx.x - 64;
        const int tw = row % p.TW, q = row / p.TW, th = q % p.TH, tn = q / p.TH;
        const int ow = ow0 + tw, oh = oh0 + th, n = n0 + tn;
        s_pixel[row] = tn < p.TN && ow < p.OW && oh < p.OH && n < p.N ? (n * p.OH + oh) * p.OW + ow : -1;
        s_res_pixel[row] = p.res_half ? (n * (p.OH >> 1) + (oh >> 1)) * (p.OW >> 1) + (ow >> 1) : s_pixel[row];
    }
    ptx::tc_fence_before_sync();
    __syncthreads();
    ptx::tc_fence_after_sync();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, tmem_base_smem, 0);
    const uint32_t ring0 = ptx::smem_u32(ring), slot = (uint32_t)(p.a_bytes + p.b_bytes);
    const uint32_t full0 = ptx::smem_u32(&full_bar[0]), empty0 = ptx::smem_u32(&empty_bar[0]);

    // This thread's share of the epilogue: items of 8 channels of a pixel in this CTA's slice of the tile.
    const int et = (int)threadIdx.x - 64;               // 0..255 in warps 2-9
    const int vshift = p.BN == 64 ? 3 : 2, n_items = (kTileM / p.splits) << vshift;
    const int row0 = rank * (kTileM / p.splits);
    bool ok = true;

    if (warp == 0) {
        const uint64_t mapA0 = reinterpret_cast<uint64_t>(&p.tmA[0]), mapB = reinterpret_cast<uint64_t>(&p.tmB);
        // position in the reduction: kernel row, kernel column, channel block
        int r, sx, cb;
        auto seek = [&](int i) {
            const int it = k0 + i, tap = it / p.cblks;
            cb = it - tap * p.cblks;
            r = tap / p.kw;
            sx = tap - r * p.kw;
        };
        auto load_b = [&](int s) {
            ptx::mbar_arrive_expect_tx_u32(full0 + s * 8, (uint32_t)(p.a_tx_bytes + p.b_bytes));
            ptx::tma_load_2d_u32(ring0 + s * slot + p.a_bytes, mapB, full0 + s * 8, (r * p.kw + sx) * p.cin_pad + cb * p.kb_elems, c0);
        };
        auto load_a = [&](int s) {
            int view = 0, dw = sx - p.pad_l, dh = r - p.pad_t;
            if (p.stride == 2) {
                const int pw = dw & 1, ph = dh & 1;
                dw = (dw - pw) >> 1;
                dh = (dh - ph) >> 1;
                view = ph * 2 + pw;
            }
            ptx::tma_load_4d_u32(ring0 + s * slot, mapA0 + view * sizeof(CUtensorMap), full0 + s * 8, cb * p.kb_elems, ow0 + dw, oh0 + dh, n0);
        };
        // the ring's first fill: one lane per stage, weights before the wait for the previous kernel
        const bool first = lane < p.stages && lane < units;
        if (first) {
            seek(lane);
            load_b(lane);
        }
        pdl_wait();
        if (first) load_a(lane);
        if (lane == 0 && units > p.stages) {
            int s = 0;
            uint32_t phase = 0;
            seek(p.stages);
            for (int i = p.stages; i < units; ++i) {      // no division in here: one thread feeds the ring
                if (!ptx::mbar_wait_bounded_u32(empty0 + s * 8, phase, &abort_flag, kSplitMaxSpins)) {
                    ok = false;
                    break;
                }
                load_b(s);
                load_a(s);
                if (++cb == p.cblks) {
                    cb = 0;
                    if (++sx == p.kw) {
                        sx = 0;
                        ++r;
                    }
                }
                if (++s == p.stages) {
                    s = 0;
                    phase ^= 1u;
                }
            }
            if (!ok) ptx::give_up(p.error, 1);
        }
        __syncwarp();
    } else if (warp == 1) {
        pdl_wait();
        {       // the whole warp, uniformly; one elected lane issues (see uniform_warp)
            const uint32_t leader = ptx::elect_one() ? 1u : 0u;
            const uint64_t d0 = ptx::make_smem_desc(ring0, (uint32_t)p.kb_bytes);
            const uint32_t desc_hi = (uint32_t)(d0 >> 32);
            const int ksteps = p.kb_bytes / 32;
            const uint32_t idesc = p.idesc;
            int s = 0;
            uint32_t phase = 0;
            for (int i = 0; i < units; ++i) {
                if (!ptx::mbar_wait_bounded_uniform(full0 + s * 8, phase, &abort_flag, kSplitMaxSpins)) {
                    ok = false;
                    break;
                }
                const uint32_t a_lo = (uint32_t)d0 + ((s * slot) >> 4), b_lo = a_lo + ((uint32_t)p.a_bytes >> 4);
                if (ksteps == 4) {
#pragma unroll
                    for (int ks = 0; ks < 4; ++ks)
                        ptx::tc_mma_lohi<kInt8>(tmem_base, a_lo + 2 * ks, b_lo + 2 * ks, desc_hi, idesc, ks ? 1u : (uint32_t)(i > 0), leader);
                } else {
                    for (int ks = 0; ks < ksteps; ++ks)
                        ptx::tc_mma_lohi<kInt8>(tmem_base, a_lo + 2 * ks, b_lo + 2 * ks, desc_hi, idesc, (i | ks) ? 1u : 0u, leader);
                }
                if (i + p.stages < units) ptx::tc_commit_u32(empty0 + s * 8, leader);
                if (++s == p.stages) {
                    s = 0;
                    phase ^= 1u;
                }
            }
            // without the commit the epilogue sees the abort flag and leaves the ring alone; the producer may be gone already,
            // with its loads still in flight
            if (ok) ptx::tc_commit_u32(ptx::smem_u32(&done_bar), leader);
            else ptx::give_up(p.error, 2);
        }
        __syncwarp();
    }
    // The residual of this thread's items is asked for while the MMAs run.
    uint4 res[kSplitMaxItems];
    if (warp >= 2) {
        pdl_wait();
        if (p.has_res) {
#pragma unroll
            for (int j = 0; j < kSplitMaxItems; ++j) {
                const int item = et + j * kSplitEpiThreads;
                const int row = row0 + (item >> vshift), cl = c0 + (item & ((1 << vshift) - 1)) * 8;
                if (item < n_items && s_pixel[row] >= 0 && cl < p.e.cout_stride)
                    res[j] = *reinterpret_cast<const uint4*>(p.e.residual + (int64_t)s_res_pixel[row] * p.e.cout_stride + cl);
            }
        }
        // accumulator -> shared memory, rows padded by 16 bytes: eight lanes' 16-byte stores cover all banks
        ok = ptx::mbar_wait_bounded_warp(&done_bar, 0, &abort_flag, kSplitMaxSpins);
        if (ok) {
            ptx::tc_fence_after_sync();
            const int q = warp & 3;
            uint8_t* row = ring + (size_t)(q * 32 + lane) * (p.BN * 4 + 16);
            // two warps per lane quarter, half of the columns each
            for (int b = warp < 6 ? 0 : p.BN / 2, e = b + p.BN / 2; b < e; b += 16) {
                uint32_t raw[16];
                ptx::tmem_ld_32x32b_x16(tmem_base + ((uint32_t)(q * 32) << 16) + b, raw);
                ptx::tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    *reinterpret_cast<uint4*>(row + b * 4 + i * 16) = make_uint4(raw[4 * i], raw[4 * i + 1], raw[4 * i + 2], raw[4 * i + 3]);
            }
            ptx::tc_fence_before_sync();
        } else if (lane == 0) {
            atomicExch(p.error, 3);
        }
    }
    __syncwarp();
    if (p.splits > 1) ptx::cluster_sync();
    else __syncthreads();
    if (warp >= 2 && ok) {
#pragma unroll
        for (int j = 0; j < kSplitMaxItems; ++j) {
            const int item = et + j * kSplitEpiThreads;
            const int row = row0 + (item >> vshift), px = item < n_items ? s_pixel[row] : -1;
            const int v = (item & ((1 << vshift) - 1)) * 8, cl = c0 + v;
            if (px < 0 || cl >= p.e.cout_stride) continue;
            const uint32_t at = ring0 + (uint32_t)row * (uint32_t)(p.BN * 4 + 16) + (uint32_t)v * 4;
            uint4 lo, hi;
            if (p.splits == 1) {
                lo = *reinterpret_cast<const uint4*>(ring + (at - ring0));
                hi = *reinterpret_cast<const uint4*>(ring + (at - ring0) + 16);
            } else {
                lo = hi = make_uint4(0, 0, 0, 0);
#pragma unroll 4
                for (int s = 0; s < p.splits; ++s) {
                    const uint32_t a = ptx::map_to_cta(at, (uint32_t)s);
                    acc_add<kInt8>(lo, ld_cluster_16(a));
                    acc_add<kInt8>(hi, ld_cluster_16(a + 16));
                }
            }
            const uint32_t raw[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
            float f[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) f[i] = epi_value<kInt8>(raw[i], s_scale[v + i], s_bias[v + i]);
            if (p.has_res) {
                const __half2* h = reinterpret_cast<const __half2*>(&res[j]);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 r = __half22float2(h[i]);
                    f[2 * i] += r.x;
                    f[2 * i + 1] += r.y;
                }
            }
            if constexpr (kPrelu) {
#pragma unroll
                for (int i = 0; i < 8; ++i) f[i] = f[i] >= 0.f ? f[i] : f[i] * __ldg(p.e.slope + cl + i);
            } else {
                apply_act_vec(f, p.e.act);
            }
            const int64_t off = (int64_t)px * p.e.y_pitch + cl;
            epi_store_vec8(p.e.y, p.e.out_dtype, off, f, p.e.out_scale);
            if (p.e.out2_dtype >= 0) epi_store_vec8(p.e.y2, p.e.out2_dtype, off, f, p.e.out2_scale);
        }
    }
    // no CTA leaves while another one may read its shared memory
    __syncwarp();
    if (p.splits > 1) ptx::cluster_sync();
    else __syncthreads();
    if (warp == 1) {
        ptx::tc_fence_after_sync();
        ptx::tmem_dealloc(tmem_base, (uint32_t)p.tmem_cols);
    }
}

}  // namespace

// Which kernel, and how a tile is divided: modelled time in us of both kernels, fitted to 330 layers (batch 1 to 64,
// 1x1 and 3x3, 32 to 1280 channels, maps of 7 x 7 to 80 x 80; every split of 32 and 64 channels).
// Split kernel: a constant, the cluster's exchange, then K blocks and epilogue of a tile one after the other, stretched by
// the tiles per SM once there are more than SMs.  Persistent kernel: a constant and rounds of tiles.  The constants are
// regression weights, not times of parts: those of 32- and 64-byte K blocks make up for terms the form does not have.  On 330
// other layers (batch 1 to 256, 7 x 7 to 80 x 80, 16 to 960 -> 64 to 1280 channels) the pick is 2 % slower than the fastest
// of both kernels on average, and 5 % or more slower in one of nine, at worst 33 to 39 % where the persistent kernel's N
// tile does not suit either (256 -> 1000 int8 1x1 at 32 x 10 x 10: 10.3 us, divided 7.4).  The line lies near two tiles of 64
// channels per SM.
ConvSplit conv_split_plan(const exb_ctx* ctx, const ConvGeom& g, const exb_conv_weights* w) {
    const ConvSplit none = {0, 0};
    if (g.pool || g.out_dtype == EXB_I32 || (g.cout_stride & 7) || (g.y_pitch & 7) || conv_fold_plan(g).on) return none;
    const int row_bytes = g.cin_stride * (g.in_dtype == EXB_I8 ? 1 : 2);
    const int kb = row_bytes % 128 == 0 ? 128 : (row_bytes % 64 == 0 ? 64 : 32);
    const int k_iters = g.kh * g.kw * (row_bytes / kb);
    const PixelBox box = choose_pixel_box(g.N, g.OH, g.OW);
    const double m_tiles = (double)((g.OW + box.TW - 1) / box.TW) * ((g.OH + box.TH - 1) / box.TH) * ((g.N + box.TN - 1) / box.TN);
    if (m_tiles > 8.0 * ctx->sm_count) return none;
    ConvSplit best = none;
    double best_t = 1e30;
    static const double kSync[4] = {0.0, 0.43, 1.23, 2.02};
    for (int bn = 32; bn <= 64; bn *= 2)
        for (int sp = 1, i = 0; sp <= 8 && sp <= k_iters; sp *= 2, ++i) {
            const double ctas = m_tiles * ((w->cout_pad + bn - 1) / bn) * sp;
            const double stretch = ctas > 1.05 * ctx->sm_count ? ctas / (1.05 * ctx->sm_count) : 1.0;
            const double units = (k_iters + sp - 1) / sp;
            const double step = kb == 32 ? 0.203 : kb == 64 ? 0.239 : 0.246;
            const double t = 1.93 + kSync[i] + stretch * (units * step + (bn == 32 ? 1.09 : 2.23) + 0.36 * kSync[i]);
            if (t < best_t) {
                best_t = t;
                best.BN = bn;
                best.splits = sp;
            }
        }
    const ConvNTile nt = conv_n_tile(ctx, g, w->cout_pad, (int64_t)m_tiles);
    const int bn = nt.BN;
    const bool two = bn <= 128 && !nt.paired;
    const double tiles = m_tiles * nt.n_tiles, slots = (double)ctx->sm_count * (two ? 2 : 1);
    const double rounds = tiles <= slots ? 1.0 : ceil(tiles / slots);
    double share = 1.0;      // two CTAs of an SM share its tensor pipe
    if (two && tiles > ctx->sm_count) share += 0.20 * (tiles < 2 * ctx->sm_count ? tiles / ctx->sm_count - 1 : 1.0);
    double step = 0.305, rest = 5.14;       // one CTA (or pair) per SM, more than 128 channels
    if (two) {
        step = bn <= 64 ? 0.246 : 0.19;
        rest = bn <= 64 ? 0.93 : 2.94;
    } else if (nt.paired) {
        step = 0.208;
        rest = 2.24;
    }
    if (bn > 128 && k_iters * kb < 512) rest = 1.6;      // single CTAs of short reductions
    step *= kb == 128 ? 1.0 : kb == 64 ? 0.21 : 0.39;
    double body = rounds * (k_iters * step + rest + (g.has_res ? 0.45 : 0.0)) * share;
    // int8 tiles of a short K, more of them than fit the SMs as clusters: 96 -> 320 1x1 at 8 x 40 x 40 8.1 us, divided 11.4
    if (two && g.in_dtype == EXB_I8 && k_iters * kb <= 256 && m_tiles * ((w->cout_pad + 63) / 64) > ctx->sm_count) body *= 0.75;
    const double persistent = 4.58 + body;
    return best_t < 0.98 * persistent ? best : none;
}

int conv_split_launch(exb_ctx* ctx, const ConvGeom& g, const ConvSplit& sp, const void* x, const exb_conv_weights* w, const void* residual,
                      void* y, void* y2, cudaStream_t st) {
    auto encode = tensor_map_encoder();
    if (!encode) return fail(EXB_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    const bool int8 = g.in_dtype == EXB_I8;
    const int es = int8 ? 1 : 2, row_bytes = g.cin_stride * es;
    ConvSplitParams p;
    memset(&p, 0, sizeof(p));
    p.N = g.N; p.OH = g.OH; p.OW = g.OW;
    const PixelBox box = choose_pixel_box(g.N, g.OH, g.OW);
    p.TW = box.TW; p.TH = box.TH; p.TN = box.TN;
    p.tiles_w = (g.OW + p.TW - 1) / p.TW;
    p.tiles_h = (g.OH + p.TH - 1) / p.TH;
    const int tiles_nb = (g.N + p.TN - 1) / p.TN;
    p.BN = sp.BN; p.splits = sp.splits;
    p.n_tiles = (w->cout_pad + p.BN - 1) / p.BN;
    p.kw = g.kw; p.stride = g.sh; p.pad_t = g.pt; p.pad_l = g.pl;
    p.cin_pad = g.cin_stride;
    p.kb_bytes = row_bytes % 128 == 0 ? 128 : (row_bytes % 64 == 0 ? 64 : 32);
    p.kb_elems = p.kb_bytes / es;
    p.cblks = row_bytes / p.kb_bytes;
    p.k_iters = g.kh * g.kw * p.cblks;
    p.a_tx_bytes = p.TW * p.TH * p.TN * p.kb_bytes;
    p.a_bytes = round_up(p.a_tx_bytes, 1024);      // the MMA reads 128 rows whatever the box holds: unused ones from what follows
    p.b_bytes = p.BN * p.kb_bytes;
    const int overread = kTileM * p.kb_bytes - p.a_bytes;
    const int units = (p.k_iters + p.splits - 1) / p.splits;
    // two CTAs of neighbouring launches fit an SM side by side (programmatic launch): half of the shared memory each
    p.stages = (96 * 1024 - overread) / (p.a_bytes + p.b_bytes);
    if (p.stages > kSplitStages) p.stages = kSplitStages;
    if (p.stages > units) p.stages = units;
    p.tmem_cols = p.BN <= 32 ? 32 : 64;
    p.cout_pad = w->cout_pad;
    p.has_res = g.has_res;
    p.res_half = g.res_half;
    p.idesc = ptx::make_idesc(int8, kTileM, (uint32_t)p.BN);
    p.e.scale = w->d_scale; p.e.bias = w->d_bias; p.e.slope = w->d_slope; p.e.residual = static_cast<const __half*>(residual);
    p.e.y = y; p.e.y2 = y2; p.e.out_dtype = g.out_dtype; p.e.out2_dtype = g.out2_dtype; p.e.act = g.act;
    p.e.out_scale = g.out_scale; p.e.out2_scale = g.out2_scale; p.e.cout_stride = g.cout_stride; p.e.y_pitch = g.y_pitch;
    p.error = ctx->d_error;
    const FoldPlan no_fold = {false, 0, 0, 0, 0};
    const CUtensorMapSwizzle sw = swizzle_for(p.kb_bytes);
    if (int rc = encode_input_views(g, no_fold, x, p.kb_elems, sw, p.TW, p.TH, p.TN, p.tmA)) return rc;
    {
        const int K = g.kh * w->kw_pack * w->cin_pad;
        cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)w->cout_pad};
        cuuint64_t strides[1] = {(cuuint64_t)K * es};
        cuuint32_t bx[2] = {(cuuint32_t)p.kb_elems, (cuuint32_t)p.BN};
        cuuint32_t estr[2] = {1, 1};
        const CUresult r = encode(&p.tmB, int8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, w->d_w, dims, strides, bx, estr,
                                  CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return fail(EXB_ERR_CUDA, "cuTensorMapEncodeTiled(B) failed with %d", (int)r);
    }
    const int grid = p.tiles_w * p.tiles_h * tiles_nb * p.n_tiles * p.splits;
    size_t smem = (size_t)p.stages * (p.a_bytes + p.b_bytes) + (overread > p.b_bytes ? overread - p.b_bytes : 0);
    const size_t part = (size_t)kTileM * (p.BN * 4 + 16);
    smem = (smem > part ? smem : part) + 1024;
    const bool prelu = g.act == EXB_ACT_PRELU;
    auto kern = int8 ? (prelu ? conv_split_kernel<true, true> : conv_split_kernel<true, false>)
                     : (prelu ? conv_split_kernel<false, true> : conv_split_kernel<false, false>);
    if (int rc = raise_smem_limit(ctx, kern)) return rc;
    return launch_pdl_cluster(ctx, "conv_split_kernel", kern, dim3((unsigned)grid), dim3(kSplitThreads), dim3((unsigned)p.splits), smem, st, p);
}

}  // namespace exb
