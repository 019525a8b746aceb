// Sliding windows over channel-last fp16 maps, input rows streamed through shared memory: what the 3x3 depthwise
// convolution and the pooling kernels share.
//
// A CTA owns a tile of 4 * groups output columns x R output rows x `slab` channels of one image.  One thread brings
// the input rows in with TMA, RS rows per stage, NS - 1 stages ahead of the arithmetic (the fill value outside the map
// is the padding); the ring runs on across the tiles of the persistent CTA.  A thread owns 4 channels x 4 output
// columns and consumes an input row the moment it has read it: the row adds to every output row it belongs to, so
// nothing but accumulators is carried from row to row.
//
// Such kernels are bound by HBM on large maps.  Loads that wait in registers (a thread keeping its own window of rows)
// left DRAM half idle: bytes in flight were limited by registers and stood still during the arithmetic.  Here 50-100 KB
// per SM are in flight whatever the threads do.
#pragma once
#include <math.h>

#include "common.cuh"
#include "ptx_sm100.cuh"
#include "tensor_map.cuh"

namespace exb {

constexpr int kRowCols = 4;          // output columns per thread
constexpr int kRowThreads = 256;     // at most, per CTA
constexpr uint32_t kRowMaxSpins = 1u << 21;

struct RowStreamParams {
    int OH, OW, cs;
    int slab, units, groups;        // channels of a CTA, slab / 4, groups of kRowCols output columns
    int slabs, tiles_w, bands, tiles;
    int R, stages;                  // output rows per tile, stages per tile
    int row_bytes, slot_bytes;      // one input row of a tile, one stage of the ring
    int x0, y0;                     // input column / row of the first tile's box
    int* error;
};

// Start of a kernel on the stream: barriers initialised (a __syncthreads and pdl_wait() must follow), ring address.
template <int NS>
__device__ __forceinline__ uint8_t* row_stream_init(const CUtensorMap& map, uint8_t* smem_raw, uint64_t* full, int* abort_flag) {
    pdl_launch_dependents();
    if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int i = 0; i < NS; ++i) ptx::mbar_init(&full[i], 1);
        ptx::fence_mbar_init();
        ptx::tma_prefetch_desc(&map);
    }
    return reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
}

// What a thread works on in the current tile.
struct RowTile {
    int oh0, ow0, rows, cols;       // cols = 0: no column of this thread lies in the map
    int n;
};

// Runs the CTA's tiles.  tile(t) is called at the start of each tile, row(index within the stage as a constant, the
// thread's input of that row: IN vectors of 4 channels) for every input row, in order.  Returns after the last tile or when a bounded wait ran out (error word set).
template <int S, int K, int RS, int NS, bool kSharedPlace, class Tile, class Row>
__device__ __forceinline__ void row_stream_run(const CUtensorMap& map, const RowStreamParams& p, uint8_t* ring, uint64_t* full, int* abort_flag,
                                               Tile tile_fn, Row row_fn) {
    constexpr int IN = (kRowCols - 1) * S + K;
    const int tid = threadIdx.x;
    // the grid is a multiple of the slab count: a CTA keeps its channels from tile to tile
    const int slab0 = (int)(blockIdx.x % p.slabs) * p.slab;
    const int u = tid % p.units, g = tid / p.units;
    // Thread 0: next stage to request.  The tile's place is worked out once per tile: six divisions in front of every stage held
    // its warp, and at the barrier behind the stage all others, up (fp16 144 channels @56 x 56, 256 images 82.8 -> 81.0 us, 16 channels
    // @103 x 10 stride 2, 98 images 11.2 -> 9.5).  Every thread carries what one of them needs through the arithmetic, unless it
    // stands in shared memory: taken where that arithmetic has no register left for it (depthwise int8 results at stride 1, all
    // 128: 192 channels @28 x 28, 256 images 44.7 us with divisions per stage, 47.2 with the place in registers, 46.0 in shared
    // memory; 160 @56 x 56, 64 images 42.6, 44.1, 43.0; 144 @56 x 56, 256 images 92.0, 91.3, 89.0; 576 @14 x 14 34.8, 32.8, 32.2).
    __shared__ __align__(16) int4 shared_place;
    __shared__ int shared_tile;
    int4 own_place;
    int own_tile;
    int4& place = kSharedPlace ? shared_place : own_place;      // x, y, image, stage of the tile
    int& next_tile = kSharedPlace ? shared_tile : own_tile;
    if (!kSharedPlace || tid == 0) {
        next_tile = (int)blockIdx.x;
        place = make_int4(0, 0, 0, 0);
    }
    auto request = [&](int slot) {
        const int tile = next_tile;
        if (tile >= p.tiles) return;
        int4 at = place;
        if (at.w == 0) {
            int t = tile / p.slabs;
            at.x = t % p.tiles_w * (p.groups * kRowCols * S) + p.x0;
            t /= p.tiles_w;
            at.y = t % p.bands * (p.R * S) + p.y0;
            at.z = t / p.bands;
        }
        const uint32_t bar = ptx::smem_u32(&full[slot]);
        ptx::mbar_arrive_expect_tx_u32(bar, (uint32_t)(RS * p.row_bytes));
        ptx::tma_load_4d_u32(ptx::smem_u32(ring + (size_t)slot * p.slot_bytes), reinterpret_cast<uint64_t>(&map), bar, slab0, at.x, at.y, at.z);
        at.y += RS;
        if (++at.w == p.stages) {
            at.w = 0;
            next_tile = tile + gridDim.x;
        }
        place = at;
    };
    if (tid == 0)
        for (int i = 0; i < NS - 1; ++i) request(i);
    const uint8_t* src0 = ring + ((size_t)g * kRowCols * S * p.slab + u * 4) * 2;
    const uint32_t px_bytes = (uint32_t)p.slab * 2;
    int slot = 0;
    uint32_t phase = 0;
    for (int tile = (int)blockIdx.x; tile < p.tiles; tile += gridDim.x) {
        int t = tile / p.slabs;
        const int tw = t % p.tiles_w;
        t /= p.tiles_w;
        RowTile rt;
        rt.n = t / p.bands;
        rt.oh0 = (t % p.bands) * p.R;
        rt.ow0 = (tw * p.groups + g) * kRowCols;
        rt.rows = min(p.R, p.OH - rt.oh0);
        rt.cols = g < p.groups ? min(kRowCols, p.OW - rt.ow0) : 0;
        tile_fn(rt);
        for (int st = 0; st < p.stages; ++st) {
            if (tid == 0) request(slot == 0 ? NS - 1 : slot - 1);      // the slot read in the previous stage
            const bool got = ptx::mbar_wait_bounded(&full[slot], phase, abort_flag, kRowMaxSpins);
            if (got && rt.cols > 0) {
                const uint8_t* src = src0 + (size_t)slot * p.slot_bytes;
#pragma unroll
                for (int rr = 0; rr < RS; ++rr) {
                    uint2 rv[IN];
#pragma unroll
                    for (int j = 0; j < IN; ++j) rv[j] = *reinterpret_cast<const uint2*>(src + j * px_bytes);
                    src += p.row_bytes;
                    row_fn(rr, rv);
                }
            }
            // everybody has read the slot (it is requested again at the top of the next stage); a wait that ran out
            // takes all threads out together
            if (!__syncthreads_and(got)) {
                if (tid == 0) ptx::give_up(p.error, 4);
                return;
            }
            if (++slot == NS) {
                slot = 0;
                phase ^= 1u;
            }
        }
    }
}

// How a launch is cut: slab x column groups fill the threads of a CTA, R output rows are a tile.
struct RowStreamPlan {
    int N, OH, OW, cs, kind, sms;       // what it was made for
    int slab, groups, threads, tiles_w, R, stages, ctas_per_sm;
};

// What the cut depends on besides the shape.
struct RowStreamKind {
    int id;                  // distinguishes kernels in a kept plan, from 1
    int S, K, RS, NS;        // stride, window, rows and stages of the ring
    int lead;                // rows loaded ahead of the tile's first window row
    double issue;            // issue cycles of a warp per input row, on one SM
};

// The cut with the least modelled time, in SM cycles: what the whole SM has to issue and to move, plus twice the chain of
// the busiest CTA - rows one after the other, each a load, dependent arithmetic and a store, slower the more warps share
// the SM.  Constants fitted to 21 depthwise layers (batch 1 to 256, 7 x 7 to 112 x 112, 16 to 960 channels), about 80
// cuts of each: the pick is within 3 % of the best cut on average, 19 % at worst.  Large maps get whole pixels (slab =
// all channels), small ones many small CTAs.  Rows of less than 128 bytes cost TMA and L2 about double.
inline RowStreamPlan row_stream_search(const RowStreamKind& k, int sms, int N, int OH, int OW, int cs) {
    static const int kRows[] = {1, 2, 3, 4, 6, 7, 10, 11, 13, 14, 16, 19, 21, 28};
    RowStreamPlan best = {N, OH, OW, cs, k.id, sms, 0, 0, 0, 0, 0, 0, 0};
    double best_t = 1e30;
    const int cols = (OW + kRowCols - 1) / kRowCols;
    for (int slab = cs <= 256 ? cs : 256; slab >= 8; slab -= 8) {
        if (cs % slab) continue;
        const int units = slab / 4;
        const int gmax = kRowThreads / units < cols ? kRowThreads / units : cols;
        int prev_groups = 0;
        for (int tiles_w = (cols + gmax - 1) / gmax; tiles_w <= cols; ++tiles_w) {
            const int groups = (cols + tiles_w - 1) / tiles_w;
            const int in_w = (groups * kRowCols - 1) * k.S + k.K;
            if (groups == prev_groups || in_w > 256) continue;
            prev_groups = groups;
            const int threads = (groups * units + 31) / 32 * 32;
            const int slot = (k.RS * in_w * slab * 2 + 127) / 128 * 128;
            const int smem = k.NS * slot + 1024 + 256;
            int per_sm = 512 / threads;          // up to 128 registers per thread
            if (per_sm > 227 * 1024 / smem) per_sm = 227 * 1024 / smem;
            if (per_sm > 8) per_sm = 8;
            if (per_sm < 1) continue;
            for (int R : kRows) {
                const int rows_in = k.lead + (R - 1) * k.S + k.K;
                if (R * k.S > 28) break;         // longer tiles measured slower: the last round of tiles is coarser
                if (rows_in % k.RS && (k.S == 1 || k.lead)) continue;      // stages only partly used
                if (R > 1 && R >= OH + k.RS) break;
                const int stages = (rows_in + k.RS - 1) / k.RS;
                const double bands = (OH + R - 1) / R;
                const double rows = stages * k.RS;
                const double per = (double)N * (cs / slab) * tiles_w * bands / sms;
                const double waves = ceil(per / per_sm);
                const double issue = per * rows * k.issue * (threads / 32);
                const double mem = per * rows * slab * 2 * (in_w * (slab < 64 ? 2 : 1) + groups * kRowCols / (double)k.S) / 40.0;
                const double resident = per < 1 ? 1 : (per < per_sm ? per : per_sm);
                const double chain = waves * (rows * (300.0 + 7.0 * resident * (threads / 32)) + 800.0);
                const double t = (issue > mem ? issue : mem) + 2.0 * chain;
                if (t < best_t) {
                    best_t = t;
                    best.slab = slab; best.groups = groups; best.threads = threads; best.tiles_w = tiles_w; best.R = R;
                    best.stages = stages; best.ctas_per_sm = per_sm;
                }
            }
        }
    }
    return best;
}

// The cut of a shape, searched once (some microseconds): the last one that fell into each of 256 slots is kept.
inline RowStreamPlan row_stream_plan(const RowStreamKind& k, int sms, int N, int OH, int OW, int cs) {
    static std::mutex mutex;
    static RowStreamPlan kept[256];
    uint32_t h = 2166136261u;
    for (int v : {k.id, sms, N, OH, OW, cs}) h = (h ^ (uint32_t)v) * 16777619u;
    std::lock_guard<std::mutex> lock(mutex);
    RowStreamPlan& e = kept[(h ^ (h >> 16)) & 255u];
    if (e.kind != k.id || e.N != N || e.OH != OH || e.OW != OW || e.cs != cs || e.sms != sms) e = row_stream_search(k, sms, N, OH, OW, cs);
    return e;
}

// Fills the parameters and the tensor map of a launch; returns the grid size, or a negative status.
inline int row_stream_setup(const exb_ctx* ctx, const RowStreamKind& k, const RowStreamPlan& pl, const __half* x, int N, int H, int W, int pt, int plft,
                            CUtensorMapFloatOOBfill fill, RowStreamParams& p, CUtensorMap& map, size_t& smem) {
    auto encode = tensor_map_encoder();
    if (!encode) return fail(EXB_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    if (!pl.slab) return fail(EXB_ERR_UNSUPPORTED, "sliding-window tile does not fit shared memory");
    p.OH = pl.OH; p.OW = pl.OW; p.cs = pl.cs;
    p.slab = pl.slab; p.units = pl.slab / 4; p.groups = pl.groups; p.slabs = pl.cs / pl.slab; p.tiles_w = pl.tiles_w;
    p.R = pl.R; p.bands = (pl.OH + pl.R - 1) / pl.R; p.stages = pl.stages;
    const int64_t tiles = (int64_t)N * p.bands * p.tiles_w * p.slabs;
    if (tiles > INT32_MAX / 2) return fail(EXB_ERR_UNSUPPORTED, "sliding-window tensor too large");
    p.tiles = (int)tiles;
    const int in_w = (pl.groups * kRowCols - 1) * k.S + k.K;
    p.row_bytes = in_w * p.slab * 2;
    p.slot_bytes = (k.RS * p.row_bytes + 127) / 128 * 128;
    p.x0 = -plft; p.y0 = -pt - k.lead;
    p.error = ctx->d_error;
    smem = (size_t)k.NS * p.slot_bytes + 128;
    cuuint64_t dims[4] = {(cuuint64_t)pl.cs, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)N};
    cuuint64_t strides[3] = {(cuuint64_t)pl.cs * 2, (cuuint64_t)W * pl.cs * 2, (cuuint64_t)H * W * pl.cs * 2};
    cuuint32_t box[4] = {(cuuint32_t)p.slab, (cuuint32_t)in_w, (cuuint32_t)k.RS, 1};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    const CUresult r = encode(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, const_cast<__half*>(x), dims, strides, box, estr,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, fill);
    if (r != CUDA_SUCCESS) return fail(EXB_ERR_CUDA, "cuTensorMapEncodeTiled(rows) failed with %d", (int)r);
    int grid = ctx->sm_count * pl.ctas_per_sm / p.slabs * p.slabs;
    if (grid < p.slabs) grid = p.slabs;
    return grid > p.tiles ? p.tiles : grid;
}

}  // namespace exb
