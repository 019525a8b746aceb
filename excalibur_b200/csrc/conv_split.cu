// Implicit-GEMM convolution for problems of few tiles (small batches, deep layers): every output tile is worked on by a
// cluster of CTAs that share its reduction dimension.
//
// The persistent kernel of conv_tc.cu gives a tile to one CTA (or pair): with one image a 3x3 layer of 512 channels @7x7
// is two tiles, and one warp issues the whole reduction - 144 dependent MMAs and the loads that feed them, 19 us
// (int8), on two of 148 SMs.  Here N tiles are at most 64 channels and the K blocks of a tile are divided over a cluster
// of 1, 2, 4 or 8 CTAs.  Each accumulates its part in TMEM, moves it to its shared memory and sends every other CTA of the
// cluster that one's slice of the tile's pixels in one bulk copy, which counts its bytes on the receiver's mbarrier; each CTA
// sums the parts of its own slice out of its own shared memory and runs the epilogue for it.  Weights never change on the stream, so their first loads
// are issued before the programmatic wait for the previous kernel; what remains after that wait is one activation load, the
// MMAs of a few K blocks, the exchange and the store.  int8 sums are exact whatever the split; fp16 ones are fp32 sums of at
// most eight partial sums.  An undivided tile goes from TMEM to the result directly, in the column order of the quad epilogue.
//
// Such launches are chains of latencies: per layer of a captured chain 2.6 us undivided (64 -> 384 fp16 1x1 at 9 x 13 x 12), 4.2 and 4.4
// in eight parts (512 -> 512 int8 3x3 at 7 x 7, 256 -> 256 at 14 x 14); with parts summed out of the other CTAs' shared memory
// between cluster barriers 3.6, 5.8 and 5.5.  Copies between CTAs move some 14 bytes per cycle and SM, so only the box's rows are sent.
#include "conv_quad.cuh"
#include "conv_tc_host.cuh"
#include "ptx_sm100.cuh"

#include <math.h>

namespace exb {
namespace {

constexpr int kSplitStages = 16;     // at most
constexpr int kSplitEpiThreads = 256;
constexpr int kSplitThreads = 64 + kSplitEpiThreads;      // warp 0 loads, warp 1 issues MMAs, warps 2-9 drain and store
constexpr int kSplitMaxItems = kTileM * 8 / kSplitEpiThreads;      // of 8 channels of a pixel, with 64 channels per tile
constexpr int kSplitMaxParts = 8;
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
    int rows, slice;        // pixels of a tile's box, and of a CTA's share of it: CTA r finishes [r*slice, (r+1)*slice)
    int recv;               // where the parts of this CTA's slice arrive, in bytes behind the ring's start
    int tmem_cols, cout_pad, has_res;
    int res_half;           // the residual is read through a nearest resize by 2
    uint32_t idesc;
    EpiParams e;
    int* error;
};

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

// Four channels of a pixel: v = act(acc * scale + bias + residual) -> first / second output.
template <bool kInt8, bool kPrelu>
__device__ __forceinline__ void split_store4(const EpiParams& e, const uint4& acc, const float4& sc, const float4& bi, bool has_res,
                                             uint32_t r01, uint32_t r23, int64_t off, int cl) {
    float f[4] = {epi_value<kInt8>(acc.x, sc.x, bi.x), epi_value<kInt8>(acc.y, sc.y, bi.y), epi_value<kInt8>(acc.z, sc.z, bi.z),
                  epi_value<kInt8>(acc.w, sc.w, bi.w)};
    if (has_res) {
        const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&r01)), b = __half22float2(*reinterpret_cast<const __half2*>(&r23));
        f[0] += a.x;
        f[1] += a.y;
        f[2] += b.x;
        f[3] += b.y;
    }
    if constexpr (kPrelu) {
#pragma unroll
        for (int i = 0; i < 4; ++i) f[i] = f[i] >= 0.f ? f[i] : f[i] * __ldg(e.slope + cl + i);
    } else {
        apply_act_vec(f, e.act);
    }
    auto store = [&](void* y, int dtype, float q) {
        if (dtype == EXB_I8) {
            *reinterpret_cast<uint32_t*>(static_cast<int8_t*>(y) + off) = quant_pack4(f[0], f[1], f[2], f[3], q);
        } else if (dtype == EXB_F16) {
            const __half2 a = __floats2half2_rn(f[0], f[1]), b = __floats2half2_rn(f[2], f[3]);
            *reinterpret_cast<uint2*>(static_cast<__half*>(y) + off) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
        } else {
            *reinterpret_cast<float4*>(static_cast<float*>(y) + off) = make_float4(f[0], f[1], f[2], f[3]);
        }
    };
    store(e.y, e.out_dtype, e.out_scale);
    if (e.out2_dtype >= 0) store(e.y2, e.out2_dtype, e.out2_scale);
}

// kDirect: an undivided tile in the quad epilogue's column order.  Otherwise the parts of the cluster's CTAs (two at least) go
// through shared memory.
template <bool kInt8, bool kPrelu, bool kDirect>
__global__ void __launch_bounds__(kSplitThreads) conv_split_kernel(const __grid_constant__ ConvSplitParams p) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[kSplitStages];
    __shared__ __align__(8) uint64_t empty_bar[kSplitStages];
    __shared__ __align__(8) uint64_t done_bar;
    __shared__ __align__(8) uint64_t recv_bar;
    __shared__ __align__(16) float s_scale[64];
    __shared__ __align__(16) float s_bias[64];
    __shared__ int s_pixel[kTileM], s_res_pixel[kTileM];
    __shared__ uint32_t tmem_base_smem;
    __shared__ int abort_flag;
    // operand ring (1024-byte aligned: the widest swizzle atom)
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
        ptx::mbar_init(&recv_bar, 1);
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
        const int at = kDirect ? quad_order(c) : c;
        s_scale[at] = ch < p.cout_pad ? p.e.scale[ch] : 0.f;
        s_bias[at] = ch < p.cout_pad ? p.e.bias[ch] : 0.f;
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
    // first round of the cluster's barrier: every CTA runs, its mbarriers are initialised (waited for before the first part is
    // sent; bytes that arrive ahead of the expectation are counted all the same)
    if (!kDirect) {
        ptx::cluster_arrive();
        if (threadIdx.x == 64) ptx::mbar_arrive_expect_tx(&recv_bar, (uint32_t)(max(min(p.slice, p.rows - rank * p.slice), 0) * (p.splits - 1) * (p.BN * 4 + 16)));
    }
    ptx::tc_fence_after_sync();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, tmem_base_smem, 0);
    const uint32_t ring0 = ptx::smem_u32(ring), slot = (uint32_t)(p.a_bytes + p.b_bytes);
    const uint32_t full0 = ptx::smem_u32(&full_bar[0]), empty0 = ptx::smem_u32(&empty_bar[0]);

    // This thread's share of the epilogue: items of 4 channels of a pixel in this CTA's slice of the tile.
    const int et = (int)threadIdx.x - 64;               // 0..255 in warps 2-9
    const int vshift = p.BN == 64 ? 4 : 3, row0 = rank * p.slice;
    const int n_items = max(min(p.slice, p.rows - row0), 0) << vshift;
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
            const int kc = (r * p.kw + sx) * p.cin_pad + cb * p.kb_elems;
            if (kDirect) ptx::tma_load_5d_u32(ring0 + s * slot + p.a_bytes, mapB, full0 + s * 8, kc, 0, 0, 0, c0 >> 5);
            else ptx::tma_load_2d_u32(ring0 + s * slot + p.a_bytes, mapB, full0 + s * 8, kc, c0);
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
            uint32_t phase = 0, ready = 0;
            const uint32_t stage_mask = (1u << p.stages) - 1u;
            for (int i = 0; i < units; ++i) {
                // Lane l looks at stage l, and one look serves all the units that have landed: a wait for each of them kept the
                // tensor pipe idle for a third of the loop.  All lanes look, without a branch: the code after it takes the
                // warp's uniform registers for its own, which lanes that run apart would overwrite for each other.
                if (!((ready >> s) & 1u)) {
                    const bool landed = ptx::mbar_test_wait_u32(full0 + min(lane, p.stages - 1) * 8, lane < s ? phase ^ 1u : phase);
                    ready = __ballot_sync(0xffffffffu, landed) & stage_mask;
                    __syncwarp();
                }
                if (!((ready >> s) & 1u) && !ptx::mbar_wait_bounded_uniform(full0 + s * 8, phase, &abort_flag, kSplitMaxSpins)) {
                    ok = false;
                    break;
                }
                ready &= ~(1u << s);
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
    if constexpr (kDirect) {
        if (warp >= 2) {
            pdl_wait();
            // two warps per lane quarter, 16 accumulator rows each; lane quads as in the persistent kernel's quad epilogue
            const int q = warp & 3, cq = lane & 3, h = warp < 6 ? 0 : 1, row = q * 32 + h * 16 + (lane >> 2);
            const int pa = s_pixel[row], pb = s_pixel[row + 8], nblk = p.BN >> 5, c = c0 + cq * 8;
            if (p.has_res) {
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    const bool in = b < nblk && c + b * 32 < p.e.cout_stride;
                    res[2 * b] = in && pa >= 0 ? __ldg(reinterpret_cast<const uint4*>(p.e.residual + (int64_t)s_res_pixel[row] * p.e.cout_stride + c + b * 32)) : make_uint4(0, 0, 0, 0);
                    res[2 * b + 1] = in && pb >= 0 ? __ldg(reinterpret_cast<const uint4*>(p.e.residual + (int64_t)s_res_pixel[row + 8] * p.e.cout_stride + c + b * 32)) : make_uint4(0, 0, 0, 0);
                }
            }
            ok = ptx::mbar_wait_bounded_warp(&done_bar, 0, &abort_flag, kSplitMaxSpins);
            if (ok) {
                ptx::tc_fence_after_sync();
                uint32_t raw[2][16];
                const uint32_t taddr = tmem_base + ((uint32_t)(q * 32 + h * 16) << 16);
                ptx::tmem_ld_16x256b_x4(taddr, raw[0]);
                if (nblk == 2) ptx::tmem_ld_16x256b_x4(taddr + 32, raw[1]);
                ptx::tmem_ld_wait(raw[0]);
                ptx::tmem_ld_wait(raw[1]);
                ptx::tc_fence_before_sync();
                auto drain = [&](auto act, auto with_res, auto outputs) __attribute__((always_inline)) {
                    constexpr int kAct = decltype(act)::value;
                    constexpr bool kRes = decltype(with_res)::value;
                    constexpr int kOut = decltype(outputs)::value;
                    const float qs = kOut == kQuadI8 ? p.e.out_scale : p.e.out2_scale;
                    const f32x2 out2_scale = pack2(qs, qs);
                    __half* const y = static_cast<__half*>(p.e.y);
                    int8_t* const y2 = static_cast<int8_t*>(kOut == kQuadI8 ? p.e.y : p.e.y2);
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        if (b >= nblk) break;
                        f32x2 sc[4], bi[4];
                        quad_scales(s_scale, s_bias, b * 32, cq, sc, bi);
                        const bool in = c + b * 32 < p.e.cout_stride;
                        const int64_t oa = (int64_t)pa * p.e.y_pitch + c + b * 32, ob = (int64_t)pb * p.e.y_pitch + c + b * 32;
                        quad_pixel<kInt8, kAct, kRes, kOut, 0>(raw[b], sc, bi, res[2 * b], in && pa >= 0, y + oa, y2 + oa, out2_scale);
                        quad_pixel<kInt8, kAct, kRes, kOut, 2>(raw[b], sc, bi, res[2 * b + 1], in && pb >= 0, y + ob, y2 + ob, out2_scale);
                    }
                };
                if (!quad_dispatch<true>(kPrelu ? -1 : quad_variant(p.e, p.has_res != 0), drain)) {
#pragma unroll
                    for (int b = 0; b < 2; ++b)      // (scales are kept from this tile's first channel on)
                        if (b < nblk && c + b * 32 < p.e.cout_stride)
                            epi_quad_rows<kInt8, kPrelu>(p.e, s_scale - c0, s_bias - c0, c + b * 32, cq, pa, pb, p.has_res != 0, res[2 * b], res[2 * b + 1],
                                                         raw[b]);
                }
            } else if (lane == 0) {
                atomicExch(p.error, 3);
            }
        }
    } else {
        const int pitch = p.BN * 4 + 16;      // a part's row: eight lanes' 16-byte accesses cover all banks
        uint8_t* recv = ring + p.recv;
        if (warp >= 2) {
            pdl_wait();
            if (p.has_res) {
#pragma unroll
                for (int j = 0; j < 2 * kSplitMaxItems; ++j) {
                    const int item = et + j * kSplitEpiThreads;
                    const int row = row0 + (item >> vshift), cl = c0 + (item & ((1 << vshift) - 1)) * 4;
                    if (item < n_items && s_pixel[row] >= 0 && cl < p.e.cout_stride) {
                        const uint2 v = *reinterpret_cast<const uint2*>(p.e.residual + (int64_t)s_res_pixel[row] * p.e.cout_stride + cl);
                        if (j & 1) {
                            res[j >> 1].z = v.x;
                            res[j >> 1].w = v.y;
                        } else {
                            res[j >> 1].x = v.x;
                            res[j >> 1].y = v.y;
                        }
                    }
                }
            }
            ok = ptx::mbar_wait_bounded_warp(&done_bar, 0, &abort_flag, kSplitMaxSpins);
        }
        __syncwarp();
        ptx::cluster_wait();
        if (warp >= 2) {
            const int q = warp & 3, row = q * 32 + lane;
            if (ok && q * 32 < p.rows) {
                ptx::tc_fence_after_sync();
                // the box's rows take the ring's place; two warps per lane quarter, half of the columns each
                const int b0 = warp < 6 ? 0 : p.BN / 2;
                const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + b0;
                uint32_t raw[2][16];
                ptx::tmem_ld_32x32b_x16(taddr, raw[0]);
                if (p.BN == 64) ptx::tmem_ld_32x32b_x16(taddr + 16, raw[1]);
                ptx::tmem_ld_wait(raw[0]);
                ptx::tmem_ld_wait(raw[1]);
                if (row < p.rows) {      // there is room for no more
                    uint4* dst = reinterpret_cast<uint4*>(ring + row * pitch + b0 * 4);
#pragma unroll
                    for (int i = 0; i < 4; ++i) dst[i] = make_uint4(raw[0][4 * i], raw[0][4 * i + 1], raw[0][4 * i + 2], raw[0][4 * i + 3]);
                    if (p.BN == 64)
#pragma unroll
                        for (int i = 0; i < 4; ++i) dst[4 + i] = make_uint4(raw[1][4 * i], raw[1][4 * i + 1], raw[1][4 * i + 2], raw[1][4 * i + 3]);
                }
                __syncwarp();
                ptx::tc_fence_before_sync();
                ptx::fence_proxy_async();
            }
            __syncwarp();
            asm volatile("bar.sync 1, 256;" ::: "memory");      // warps 2-9 (all of them, whatever their waits gave)
            ok = ok && *static_cast<volatile int*>(&abort_flag) == 0;
            // lane r of the first of them sends CTA r the rows of its slice, part `rank` of what that one sums
            const int theirs = min(p.slice, p.rows - lane * p.slice);
            if (ok && warp == 2 && lane < p.splits && lane != rank && theirs > 0)
                ptx::copy_to_cta(ptx::map_to_cta(ptx::smem_u32(recv) + (uint32_t)(rank * p.slice * pitch), (uint32_t)lane), ring0 + (uint32_t)(lane * p.slice * pitch),
                                 (uint32_t)(theirs * pitch), ptx::map_to_cta(ptx::smem_u32(&recv_bar), (uint32_t)lane));
            __syncwarp();
            if (ok) ok = ptx::mbar_wait_bounded_warp(&recv_bar, 0, &abort_flag, kSplitMaxSpins);
            if (!ok && lane == 0) atomicExch(p.error, 3);
        }
        // second round: no CTA leaves while parts may still be on their way to it (waited for at the end)
        __syncwarp();
        ptx::cluster_arrive();
        if (warp >= 2 && ok) {
            auto finish = [&](auto parts) __attribute__((always_inline)) {
                constexpr int S = decltype(parts)::value, kItems = kSplitMaxParts / S;
                uint4 part[kItems][S];
#pragma unroll
                for (int j = 0; j < kItems; ++j) {
                    const int item = et + j * kSplitEpiThreads;
                    const int at = (item >> vshift) * pitch + (item & ((1 << vshift) - 1)) * 16;
                    if (item < n_items)
#pragma unroll
                        for (int s = 0; s < S; ++s)
                            part[j][s] = *reinterpret_cast<const uint4*>((s == rank ? ring + row0 * pitch : recv + s * p.slice * pitch) + at);
                }
#pragma unroll
                for (int j = 0; j < kItems; ++j) {
                    const int item = et + j * kSplitEpiThreads;
                    const int v = (item & ((1 << vshift) - 1)) * 4, cl = c0 + v;
                    const int px = item < n_items ? s_pixel[row0 + (item >> vshift)] : -1;
                    if (px < 0 || cl >= p.e.cout_stride) continue;
                    uint4 a = part[j][0];
#pragma unroll
                    for (int s = 1; s < S; ++s) acc_add<kInt8>(a, part[j][s]);
                    const float4 sc = *reinterpret_cast<const float4*>(s_scale + v), bi = *reinterpret_cast<const float4*>(s_bias + v);
                    split_store4<kInt8, kPrelu>(p.e, a, sc, bi, p.has_res != 0, j & 1 ? res[j >> 1].z : res[j >> 1].x, j & 1 ? res[j >> 1].w : res[j >> 1].y,
                                                (int64_t)px * p.e.y_pitch + cl, cl);
                }
            };
            if (p.splits == 8) finish(std::integral_constant<int, 8>());
            else if (p.splits == 4) finish(std::integral_constant<int, 4>());
            else finish(std::integral_constant<int, 2>());
        }
        __syncwarp();
        ptx::cluster_wait();
    }
    __syncwarp();
    __syncthreads();
    if (warp == 1) {
        ptx::tc_fence_after_sync();
        ptx::tmem_dealloc(tmem_base, (uint32_t)p.tmem_cols);
    }
}

}  // namespace

// Shared memory of a launch.
struct SplitRing {
    int stages, a_bytes, b_bytes;
    int part;      // of all CTAs of a cluster for one's slice
};
static SplitRing split_ring(const exb_ctx* ctx, int rows, int kb_bytes, int bn, int splits, int k_iters, int grid) {
    SplitRing r;
    r.a_bytes = round_up(rows * kb_bytes, 1024);      // the MMA reads 128 rows whatever the box holds: unused ones from what follows
    r.b_bytes = bn * kb_bytes;
    r.part = splits == 1 ? 0 : (rows + splits - 1) / splits * splits * (bn * 4 + 16);
    // two CTAs of neighbouring launches fit an SM side by side (programmatic launch): half of the shared memory each, and all
    // of it where the neighbours find SMs of their own, or where one CTA per SM walks through more than two such rings (not
    // larger clusters: at one CTA per SM those of eight reach some 130 SMs, and 144 CTAs took two waves, 8.5 -> 12.2 us on
    // 512 -> 136 fp16 3x3 at 2 x 26 x 13)
    const int units = (k_iters + splits - 1) / splits;
    const auto stages = [&](int room) { return (room - (kTileM * kb_bytes - r.a_bytes) - r.part) / (r.a_bytes + r.b_bytes); };
    r.stages = stages(109 * 1024);
    if (2 * grid <= ctx->sm_count || (grid <= ctx->sm_count && splits <= 2 && units > 2 * r.stages)) r.stages = stages(ctx->smem_optin - 6 * 1024);
    if (r.stages > kSplitStages) r.stages = kSplitStages;
    if (r.stages > units) r.stages = units;
    return r;
}

// What both models of the launch of a layer read.
struct SplitProblem {
    PixelBox box;
    double m_tiles;
    int kb, k_iters;      // bytes of a K block, K blocks of a tile
};

// The pick of the first model: both kernels' times in a captured chain, fitted to 590 layers before the layouts of their launches
// were modelled.  splits = 0: the persistent kernel.
static ConvSplit first_pick(const exb_ctx* ctx, const ConvGeom& g, const exb_conv_weights* w, const SplitProblem& q) {
    ConvSplit best = {0, 0, q.box.TW, q.box.TH, q.box.TN};
    double best_t = 1e30;
    static const double kParts[4] = {0.0, 1.0, 0.53, 0.46};      // an exchange of 1, 2, 4, 8 parts beside its volume
    const double unit = q.kb == 128 ? 0.218 : q.kb == 64 ? 0.209 : 0.192;
    for (int bn = 32; bn <= 64; bn *= 2)
        for (int sp = 1, i = 0; sp <= kSplitMaxParts && (sp == 1 || 2 * sp <= q.k_iters); sp *= 2, ++i) {      // two K blocks a part
            const double ctas = q.m_tiles * ((w->cout_pad + bn - 1) / bn) * sp;
            const double stretch = ctas > 1.02 * ctx->sm_count ? ctas / (1.02 * ctx->sm_count) : 1.0;
            const double units = (q.k_iters + sp - 1) / sp;
            const double volume = q.box.TW * q.box.TH * q.box.TN * bn * (sp - 1) / (sp * 8192.0);
            const double t = 0.8 + kParts[i] + 1.29 * volume +
                             stretch * (units * unit * (bn == 32 ? 0.962 : 1.0) + (bn == 32 ? 1.40 : 1.52) + 1.31 * volume - (sp > 1 ? 0.36 : 0.0));
            if (t < best_t) {
                best_t = t;
                best.BN = bn;
                best.splits = sp;
            }
        }
    const ConvNTile nt = conv_n_tile(ctx, g, w->cout_pad, (int64_t)q.m_tiles);
    const bool two = nt.BN <= 128 && !nt.paired;
    const double tiles = q.m_tiles * nt.n_tiles, slots = (double)ctx->sm_count * (two ? 2 : 1);
    const double rounds = tiles <= slots ? 1.0 : ceil(tiles / slots);
    double share = 1.0, step = 0.292, rest = 1.45;      // one CTA per SM
    if (two) {
        if (tiles > ctx->sm_count) share += 0.35 * (tiles < 2 * ctx->sm_count ? tiles / ctx->sm_count - 1 : 1.0);
        step = nt.BN <= 64 ? 0.216 : 0.304;
        rest = nt.BN <= 64 ? 0.0 : 1.09;
    } else if (nt.paired) {
        step = 0.207;
        rest = 1.71;
    }
    step *= q.kb == 128 ? 1.0 : q.kb == 64 ? 0.65 : 0.56;
    double body = rounds * (q.k_iters * step + rest + (g.has_res ? 1.5 : 0.0)) * share;
    // int8 tiles of a short K, more of them than fit the SMs as clusters
    if (two && g.in_dtype == EXB_I8 && q.k_iters * q.kb <= 256 && q.m_tiles * ((w->cout_pad + 63) / 64) > ctx->sm_count)
        body *= g.out_dtype == EXB_I8 && g.out2_dtype < 0 ? 0.8 : 1.28;
    if (best_t >= 3.92 + body) best.splits = 0;
    return best;
}

// Modelled time of a launch of the split kernel in us, fitted like conv_tc_time to 1200 layers (batch 1 to 256, 1x1 and 3x3, 16 to
// 1280 -> 16 to 1280 channels, maps of 4 x 4 to 160 x 160; every split of 32 and 64 channels).  A layer's time is the mean of
// two measurements, a captured chain of its own launches and one in which they alternate with another layer's: the persistent
// kernel loses 1.2 to 1.6 us between launches of other kernels, the split kernel 0 to 0.5.  The constants are regression
// weights, not times of parts: a constant, what the exchange costs by the number of parts, the chain of a CTA (K blocks, of
// which those that the ring does not hold wait for their loads, the epilogue, the volume of the exchange) and, beyond one CTA
// per SM, what they take from each other.  Two run side by side on an SM, fewer where clusters of four and eight do not fill
// the SMs that are wired together (at 1.9 and 1.8 per SM times jump by half); beyond that the chain is walked once more.
static double split_time(const exb_ctx* ctx, const exb_conv_weights* w, const SplitProblem& q, int bn, int sp) {
    static const double kParts[4] = {0.0, 1.347, 0.899, 1.002}, kPlaces[4] = {2.0, 2.0, 1.9, 1.8};      // CTAs per SM of one wave
    const int i = sp == 1 ? 0 : sp == 2 ? 1 : sp == 4 ? 2 : 3;
    const double unit = q.kb == 128 ? 0.1487 : q.kb == 64 ? 0.1923 : 0.1965, shared = q.kb == 128 ? 0.0679 : q.kb == 64 ? 0.0343 : 0.0341;
    const double ctas = q.m_tiles * ((w->cout_pad + bn - 1) / bn) * sp, per_sm = ctas / ctx->sm_count, full = per_sm / kPlaces[i];
    const int grid = per_sm > 0.5 && per_sm <= 1 ? (int)ctas : ctx->sm_count + 1;      // (small grids were fitted with half a ring)
    const int units = (q.k_iters + sp - 1) / sp, stages = split_ring(ctx, kTileM, q.kb, bn, sp, q.k_iters, grid).stages;
    const double epi = (bn == 32 ? 0.696 : 0.915) + 0.670 * bn * (sp - 1) / (sp * 64.0);
    const double chain = units * unit + 0.445 * (units - stages) / stages + epi;
    return 1.663 + kParts[i] + chain * (full <= 1 ? 1.0 : 0.116 * full + 0.884 * ceil(full)) +
           (per_sm > 1 ? per_sm - 1 : 0.0) * (units * shared * (bn == 32 ? 1.105 : 1.0) + 1.548 * epi);
}

// Which kernel, and how a tile is divided.  Two models have to agree: the first one's pick stays unless the second, which knows
// the layouts, promises 7 % more: of 118 drawn layers it promised less in five, four of which it made 10 to 32 % slower, and
// more in nine, of which seven were 7 to 33 % faster and two 2 % slower; of 110 others 0.985 of the first pick's time.
// fp16 layers keep the order of their sums, whose last bits, rounded through the layers of a network, show in its results
// (1e-4): the number of parts stays the first model's, undivided tiles and a persistent kernel that goes through the taps in
// the same order are exchanged for each other.  int8 sums are exact whatever the order.  A part has two K blocks at least:
// parts of one were the fastest choice of 12 of 304 drawn layers, by 2 to 10 %, and without them small batches of the same
// image more often keep one order.
// 288 -> 192 int8 3x3 stride 2 at 8 x 56 x 56, whose undivided tiles just fit the SMs, 23.4 -> 15.7 us in two parts; 48 -> 264 fp16 3x3
// at 2 x 64 x 50 11.8 -> 10.2.
static ConvSplit search_split_plan(const exb_ctx* ctx, const ConvGeom& g, const exb_conv_weights* w) {
    const ConvSplit none = {0, 0, 0, 0, 0};
    if (g.pool || g.out_dtype == EXB_I32 || (g.cout_stride & 7) || (g.y_pitch & 7) || conv_fold_plan(g).on) return none;
    const int row_bytes = g.cin_stride * (g.in_dtype == EXB_I8 ? 1 : 2);
    SplitProblem q;
    q.kb = row_bytes % 128 == 0 ? 128 : (row_bytes % 64 == 0 ? 64 : 32);
    q.k_iters = g.kh * g.kw * (row_bytes / q.kb);
    q.box = choose_pixel_box(g.N, g.OH, g.OW);
    q.m_tiles = (double)((g.OW + q.box.TW - 1) / q.box.TW) * ((g.OH + q.box.TH - 1) / q.box.TH) * ((g.N + q.box.TN - 1) / q.box.TN);
    if (q.m_tiles > 8.0 * ctx->sm_count) return none;
    const ConvSplit first = first_pick(ctx, g, w, q);
    bool tap_order;      // as undivided tiles sum
    const double persistent = conv_tc_time(ctx, g, w, &tap_order);
    const double limit = 0.93 * (first.splits ? split_time(ctx, w, q, first.BN, first.splits) : persistent);
    const bool exact = g.in_dtype == EXB_I8;
    ConvSplit best = first;
    double best_t = limit;
    // between launches of other kernels the persistent one loses twice what its modelled time holds (32 -> 160 fp16 1x1 at
    // 9 x 50 x 45 in a network: 9 us, undivided tiles 7)
    if (first.splits && persistent + 0.7 < best_t && (exact || (first.splits == 1 && tap_order))) {
        best_t = persistent;
        best.splits = 0;
    }
    if (first.splits || exact || tap_order)      // (a persistent launch that has no layout is refused)
        for (int bn = 32; bn <= 64 && (first.splits || persistent < 1e30); bn *= 2)
            for (int sp = 1; sp <= kSplitMaxParts && (sp == 1 || 2 * sp <= q.k_iters); sp *= 2) {
                if (!exact && sp != (first.splits ? first.splits : 1)) continue;
                const double t = split_time(ctx, w, q, bn, sp);
                if (t < best_t) {
                    best_t = t;
                    best.BN = bn;
                    best.splits = sp;
                }
            }
    return best.splits ? best : none;
}

// The same, searched once per layer and thread (0.2 us of every eager call): a pure function of the values that are compared,
// and the last layer that fell into each of 64 slots is kept.
ConvSplit conv_split_plan(const exb_ctx* ctx, const ConvGeom& g, const exb_conv_weights* w) {
    struct Layer {
        ConvGeom g;
        int cout_pad, cin_pad, kw_pack, sm_count, smem_optin;
    };
    struct Kept {
        Layer layer;
        ConvSplit plan;
        bool used;
    };
    static thread_local Kept kept[64];
    static_assert(sizeof(Layer) == sizeof(ConvGeom) + 5 * sizeof(int) && sizeof(ConvGeom) % sizeof(int) == 0, "compared by its bytes");
    const Layer layer = {g, w->cout_pad, w->cin_pad, w->kw_pack, ctx->sm_count, ctx->smem_optin};
    uint32_t h = 2166136261u;
    for (int v : {g.N, g.OH, g.OW, g.cin_stride, w->cout_pad, g.kh, g.has_res}) h = (h ^ (uint32_t)v) * 16777619u;
    Kept& k = kept[(h ^ (h >> 16)) & 63u];
    if (!k.used || memcmp(&k.layer, &layer, sizeof(Layer)) != 0) {
        k.plan = search_split_plan(ctx, g, w);
        memcpy(&k.layer, &layer, sizeof(Layer));
        k.used = true;
    }
    return k.plan;
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
    p.TW = sp.TW; p.TH = sp.TH; p.TN = sp.TN;
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
    p.rows = p.TW * p.TH * p.TN;
    p.slice = (p.rows + p.splits - 1) / p.splits;
    p.a_tx_bytes = p.TW * p.TH * p.TN * p.kb_bytes;
    const bool direct = p.splits == 1;
    const int grid = p.tiles_w * p.tiles_h * tiles_nb * p.n_tiles * p.splits;
    const SplitRing ring = split_ring(ctx, p.rows, p.kb_bytes, p.BN, p.splits, p.k_iters, grid);
    p.stages = ring.stages;
    p.a_bytes = ring.a_bytes;
    p.b_bytes = ring.b_bytes;
    const int overread = kTileM * p.kb_bytes - p.a_bytes;
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
    if (int rc = encode_weights(g, w, p.kb_elems, sw, p.BN, direct, &p.tmB)) return rc;
    size_t smem = (size_t)p.stages * (p.a_bytes + p.b_bytes) + (overread > p.b_bytes ? overread - p.b_bytes : 0);
    if (!direct) {
        if (smem < (size_t)ring.part) smem = ring.part;      // the box's rows take the ring's place
        p.recv = (int)((smem + 15) / 16 * 16);
        smem = (size_t)p.recv + ring.part;
    }
    smem += 1024;
    const bool prelu = g.act == EXB_ACT_PRELU;
    auto kern = int8 ? (prelu ? conv_split_kernel<true, true, false> : conv_split_kernel<true, false, false>)
                     : (prelu ? conv_split_kernel<false, true, false> : conv_split_kernel<false, false, false>);
    if (direct)
        kern = int8 ? (prelu ? conv_split_kernel<true, true, true> : conv_split_kernel<true, false, true>)
                    : (prelu ? conv_split_kernel<false, true, true> : conv_split_kernel<false, false, true>);
    if (int rc = raise_smem_limit(ctx, kern)) return rc;
    return launch_pdl_cluster(ctx, "conv_split_kernel", kern, dim3((unsigned)grid), dim3(kSplitThreads), dim3((unsigned)p.splits), smem, st, p);
}

}  // namespace exb
