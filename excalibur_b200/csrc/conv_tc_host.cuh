// Host-side pieces that the tensor-core convolution kernels share: pixel boxes and tensor maps of the input.
#pragma once
#include "conv_common.cuh"
#include "tensor_map.cuh"

namespace exb {

constexpr int kTileM = 128;      // output pixels (accumulator rows) of a tile

inline int round_up(int a, int b) { return (a + b - 1) / b * b; }

inline CUtensorMapSwizzle swizzle_for(int kb_bytes) {
    return kb_bytes == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : (kb_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
}

struct PixelBox {
    int N, OH, OW;       // what it was chosen for
    int TW, TH, TN;
};

// The pixel box (TW x TH x TN <= 128 rows) that wastes the fewest MMA rows; ties go to the widest box (longest contiguous
// runs for the TMA unit), then the tallest.
inline PixelBox search_pixel_box(int N, int OH, int OW) {
    PixelBox b = {N, OH, OW, 1, 1, 1};
    double best = -1.0;
    for (int tw = 1; tw <= OW && tw <= kTileM; ++tw)
        for (int th = 1; th <= OH && tw * th <= kTileM; ++th) {
            int tn = kTileM / (tw * th);
            if (tn > N) tn = N;
            if (tn < 1) continue;
            const int64_t tiles = (int64_t)((OW + tw - 1) / tw) * ((OH + th - 1) / th) * ((N + tn - 1) / tn);
            const double eff = (double)OW * OH * N / ((double)tiles * kTileM);
            const bool better = eff > best + 1e-9 || (eff > best - 1e-9 && (tw > b.TW || (tw == b.TW && th > b.TH)));
            if (better) {
                best = eff;
                b.TW = tw; b.TH = th; b.TN = tn;
            }
        }
    return b;
}

// The same, searched once per shape and thread (the search is some 500 candidates, 4 us of every eager call): the last shape
// that fell into each of 256 slots is kept.
inline PixelBox choose_pixel_box(int N, int OH, int OW) {
    static thread_local PixelBox kept[256];
    uint32_t h = 2166136261u;
    for (int v : {N, OH, OW}) h = (h ^ (uint32_t)v) * 16777619u;
    PixelBox& e = kept[(h ^ (h >> 16)) & 255u];
    if (e.N != N || e.OH != OH || e.OW != OW) e = search_pixel_box(N, OH, OW);
    return e;
}

// Tensor maps of the input: one view per input parity (only view 0 for stride 1).  Rows may be physically padded.
inline int encode_input_views(const ConvGeom& g, const FoldPlan& fold, const void* x, int kb_elems, CUtensorMapSwizzle sw, int box_w, int box_h,
                              int box_n, CUtensorMap (&maps)[4]) {
    auto encode = tensor_map_encoder();
    const bool int8 = g.in_dtype == EXB_I8;
    const int es = int8 ? 1 : 2;
    const CUtensorMapDataType dt = int8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    const size_t px_bytes = (size_t)g.cin_stride * es, row_pitch = (size_t)g.w_pitch * px_bytes;
    const int st = g.sh, nviews = st == 1 ? 1 : 4;
    for (int v = 0; v < nviews; ++v) {
        const int ph = v >> 1, pw = v & 1;
        if (fold.on && pw) continue;   // the folded layout walks W inside the K row
        // rows / columns of this view: indices ph, ph + st, ... < H
        const int vh = (g.H - ph + st - 1) / st, vw = (g.W - pw + st - 1) / st;
        if (vh <= 0 || vw <= 0) return fail(EXB_ERR_UNSUPPORTED, "stride-2 convolution needs H and W of at least 2");
        cuuint32_t box[4] = {(cuuint32_t)kb_elems, (cuuint32_t)box_w, (cuuint32_t)box_h, (cuuint32_t)box_n};
        cuuint32_t estr[4] = {1, 1, 1, 1};
        char* base = const_cast<char*>(static_cast<const char*>(x)) + (size_t)ph * row_pitch;
        CUresult r;
        if (fold.on) {
            // dim0: F pixels x cin_stride channels (one K row), dim1: output columns, stepping
            // stride_w pixels (windows of neighbouring columns overlap), dim2: rows of this parity.
            cuuint64_t dims[4] = {(cuuint64_t)kb_elems, (cuuint64_t)g.OW, (cuuint64_t)vh, (cuuint64_t)g.N};
            cuuint64_t strides[3] = {(cuuint64_t)g.sw * px_bytes, (cuuint64_t)st * row_pitch, (cuuint64_t)g.H * row_pitch};
            r = encode(&maps[v], dt, 4, base + (size_t)(g.w_pad - fold.pl_eff) * px_bytes, dims, strides, box, estr,
                       CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        } else {
            cuuint64_t dims[4] = {(cuuint64_t)g.cin_stride, (cuuint64_t)vw, (cuuint64_t)vh, (cuuint64_t)g.N};
            cuuint64_t strides[3] = {(cuuint64_t)st * px_bytes, (cuuint64_t)st * row_pitch, (cuuint64_t)g.H * row_pitch};
            r = encode(&maps[v], dt, 4, base + (size_t)(pw + g.w_pad) * px_bytes, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
                       CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        }
        if (r != CUDA_SUCCESS) return fail(EXB_ERR_CUDA, "cuTensorMapEncodeTiled(A view %d) failed with %d", v, (int)r);
    }
    return EXB_OK;
}

// Tensor map of the packed weights [cout][K], boxes of `rows` rows and a K block.  `quad`: in the column order of the quad
// epilogue (rows in whole 32-channel blocks).  Row 32*block + 8*j + 2*g + e is seen as (e: 2, j: 4, g: 4, block) and traversed
// e, j, g, block: shared-memory row (= accumulator column) 8*g + 2*j + e of a block holds output channel 8*j + 2*g + e.
inline int encode_weights(const ConvGeom& g, const exb_conv_weights* w, int kb_elems, CUtensorMapSwizzle sw, int rows, bool quad, CUtensorMap* map) {
    auto encode = tensor_map_encoder();
    const bool int8 = g.in_dtype == EXB_I8;
    const int K = g.kh * w->kw_pack * w->cin_pad;
    const cuuint64_t kb = (cuuint64_t)K * (int8 ? 1 : 2);
    const cuuint64_t dims2[2] = {(cuuint64_t)K, (cuuint64_t)w->cout_pad}, strides2[1] = {kb};
    const cuuint32_t box2[2] = {(cuuint32_t)kb_elems, (cuuint32_t)rows};
    const cuuint64_t dims5[5] = {(cuuint64_t)K, 2, 4, 4, (cuuint64_t)(weight_rows(w->cout_pad) / 32)}, strides5[4] = {kb, 8 * kb, 2 * kb, 32 * kb};
    const cuuint32_t box5[5] = {(cuuint32_t)kb_elems, 2, 4, 4, (cuuint32_t)(rows / 32)};
    const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    const CUresult r = encode(map, int8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, quad ? 5 : 2, w->d_w, quad ? dims5 : dims2,
                              quad ? strides5 : strides2, quad ? box5 : box2, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? EXB_OK : fail(EXB_ERR_CUDA, "cuTensorMapEncodeTiled(B) failed with %d", (int)r);
}

}  // namespace exb
