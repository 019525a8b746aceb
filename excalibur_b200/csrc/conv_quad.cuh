// The quad epilogue of the tensor-core convolution kernels: four neighbouring lanes hold one pixel, 8 consecutive channels each
// (see the epilogue of conv_tc.cu).
#pragma once
#include <type_traits>

#include "conv_common.cuh"

namespace exb {

// Two pixels' 8 consecutive channels from one 16x256b.x4 fragment (raw[4g + e] first pixel, raw[4g + 2 + e] second
// pixel, channels cl + 2g + e).  Scale and bias are read once for both pixels, from the quad-ordered copy: the four
// floats of channels 8*j + 4*i .. + 3 of a 32-channel block sit at 32*block + 16*i + 4*j, so that the four lanes of a
// pixel read one contiguous 64-byte piece per load (channel order would put neighbouring lanes on the same banks).
template <bool kInt8, bool kPrelu>
__device__ __forceinline__ void epi_quad_rows(const EpiParams& e, const float* q_scale, const float* q_bias, int cl, int cq,
                                              int pa, int pb, bool add_res, const uint4& ra, const uint4& rb,
                                              const uint32_t (&raw)[16]) {
    float va[8], vb[8];
    const float4* sc = reinterpret_cast<const float4*>(q_scale + (cl & ~31) + 4 * cq);
    const float4* bi = reinterpret_cast<const float4*>(q_bias + (cl & ~31) + 4 * cq);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const float4 s4 = sc[4 * i], b4 = bi[4 * i];
        va[4 * i + 0] = epi_value<kInt8>(raw[8 * i + 0], s4.x, b4.x);
        va[4 * i + 1] = epi_value<kInt8>(raw[8 * i + 1], s4.y, b4.y);
        va[4 * i + 2] = epi_value<kInt8>(raw[8 * i + 4], s4.z, b4.z);
        va[4 * i + 3] = epi_value<kInt8>(raw[8 * i + 5], s4.w, b4.w);
        vb[4 * i + 0] = epi_value<kInt8>(raw[8 * i + 2], s4.x, b4.x);
        vb[4 * i + 1] = epi_value<kInt8>(raw[8 * i + 3], s4.y, b4.y);
        vb[4 * i + 2] = epi_value<kInt8>(raw[8 * i + 6], s4.z, b4.z);
        vb[4 * i + 3] = epi_value<kInt8>(raw[8 * i + 7], s4.w, b4.w);
    }
    if (add_res) {
        const __half2* ha = reinterpret_cast<const __half2*>(&ra);
        const __half2* hb = reinterpret_cast<const __half2*>(&rb);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 fa = __half22float2(ha[i]), fb = __half22float2(hb[i]);
            va[2 * i] += fa.x;
            va[2 * i + 1] += fa.y;
            vb[2 * i] += fb.x;
            vb[2 * i + 1] += fb.y;
        }
    }
    if constexpr (kPrelu) {
        const float4 l0 = __ldg(reinterpret_cast<const float4*>(e.slope + cl)), l1 = __ldg(reinterpret_cast<const float4*>(e.slope + cl) + 1);
        const float sl[8] = {l0.x, l0.y, l0.z, l0.w, l1.x, l1.y, l1.z, l1.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            va[i] = va[i] >= 0.f ? va[i] : va[i] * sl[i];
            vb[i] = vb[i] >= 0.f ? vb[i] : vb[i] * sl[i];
        }
    } else {
        apply_act_vec(va, e.act);
        apply_act_vec(vb, e.act);
    }
    if (pa >= 0) {
        const int64_t off = (int64_t)pa * e.y_pitch + cl;
        epi_store_vec8(e.y, e.out_dtype, off, va, e.out_scale);
        if (e.out2_dtype >= 0) epi_store_vec8(e.y2, e.out2_dtype, off, va, e.out2_scale);
    }
    if (pb >= 0) {
        const int64_t off = (int64_t)pb * e.y_pitch + cl;
        epi_store_vec8(e.y, e.out_dtype, off, vb, e.out_scale);
        if (e.out2_dtype >= 0) epi_store_vec8(e.y2, e.out2_dtype, off, vb, e.out2_scale);
    }
}

// The lean form of the same for the outputs that layers have in earnest: fp16, alone or with an int8 copy, behind no
// activation, ReLU, ReLU6 or SiLU.  What bounds short reductions is the instruction stream of the epilogue warps (16
// instructions per value in the general form), so everything that can be is known at compile time, sums are formed two at a
// time, clamps act on packed halves (rounding is monotone and 0 and 6 are halves: the same results), and the accumulator is
// handed back after the last load.  32 -> 160 int8 1x1 + ReLU6 at 64 x 56 x 56 29.5 -> 19.8 us, 64 -> 64 fp16 1x1 + SiLU at
// 16 x 160 x 160 37.5 -> 30.4.
enum QuadAct { kQuadNone = 0, kQuadRelu = 1, kQuadRelu6 = 2, kQuadSilu = 3 };
template <int kAct>
using QuadActC = std::integral_constant<int, kAct>;

// What is stored: fp16, fp16 with an int8 copy, int8 alone (y2 and out2_scale are then the only output's).
enum QuadOut { kQuadF16 = 0, kQuadBoth = 1, kQuadI8 = 2 };
template <int kOut>
using QuadOutC = std::integral_constant<int, kOut>;

// activation | residual << 2 | outputs << 3, or -1 where the general form is needed
__device__ __forceinline__ int quad_variant(const EpiParams& e, bool has_res) {
    const bool i8 = e.out_dtype == EXB_I8 && e.out2_dtype < 0;
    if (!i8 && (e.out_dtype != EXB_F16 || (e.out2_dtype >= 0 && e.out2_dtype != EXB_I8))) return -1;
    const int more = (has_res ? 4 : 0) | (i8 ? kQuadI8 << 3 : e.out2_dtype >= 0 ? kQuadBoth << 3 : 0);
    if (e.act == EXB_ACT_NONE) return kQuadNone | more;
    if (e.act == EXB_ACT_RELU) return kQuadRelu | more;
    if (more) return -1;
    return e.act == EXB_ACT_RELU6 ? kQuadRelu6 : e.act == EXB_ACT_SILU ? kQuadSilu : -1;
}

// f(activation, residual, outputs) with the variant's compile-time values; false where there is none.  kI8: the kernel also has
// layers whose only output is int8.
template <bool kI8, typename F>
__device__ __forceinline__ bool quad_dispatch(int variant, F&& f) {
    using std::false_type;
    using std::true_type;
    typedef QuadOutC<kQuadF16> f16;
    typedef QuadOutC<kQuadBoth> both;
    typedef QuadOutC<kQuadI8> i8;
    if (variant == kQuadRelu6) f(QuadActC<kQuadRelu6>(), false_type(), f16());
    else if (variant == kQuadSilu) f(QuadActC<kQuadSilu>(), false_type(), f16());
    else if (variant == kQuadRelu) f(QuadActC<kQuadRelu>(), false_type(), f16());
    else if (variant == kQuadNone) f(QuadActC<kQuadNone>(), false_type(), f16());
    else if (variant == (kQuadRelu | 4)) f(QuadActC<kQuadRelu>(), true_type(), f16());
    else if (variant == (kQuadNone | 4)) f(QuadActC<kQuadNone>(), true_type(), f16());
    else if (variant == (kQuadRelu | 8)) f(QuadActC<kQuadRelu>(), false_type(), both());
    else if (variant == (kQuadNone | 8)) f(QuadActC<kQuadNone>(), false_type(), both());
    else if (variant == (kQuadRelu | 12)) f(QuadActC<kQuadRelu>(), true_type(), both());
    else if (variant == (kQuadNone | 12)) f(QuadActC<kQuadNone>(), true_type(), both());
    else if (kI8 && variant == (kQuadRelu | 16)) f(QuadActC<kQuadRelu>(), false_type(), i8());
    else if (kI8 && variant == (kQuadNone | 16)) f(QuadActC<kQuadNone>(), false_type(), i8());
    else if (kI8 && variant == (kQuadRelu | 20)) f(QuadActC<kQuadRelu>(), true_type(), i8());
    else return false;
    return true;
}

// Scale and bias of this thread's 8 channels from the quad-ordered copies.
__device__ __forceinline__ void quad_scales(const float* q_scale, const float* q_bias, int cl, int cq, f32x2 (&sc)[4], f32x2 (&bi)[4]) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int at = (cl & ~31) + 4 * cq + 16 * i;
        const ulonglong2 s = *reinterpret_cast<const ulonglong2*>(q_scale + at), c = *reinterpret_cast<const ulonglong2*>(q_bias + at);
        sc[2 * i] = s.x;
        sc[2 * i + 1] = s.y;
        bi[2 * i] = c.x;
        bi[2 * i + 1] = c.y;
    }
}

// Where the quad-ordered copies keep channel c.
__device__ __forceinline__ int quad_order(int c) { return (c & ~31) | ((c & 4) << 2) | ((c & 24) >> 1) | (c & 3); }

template <bool kInt8>
__device__ __forceinline__ f32x2 quad_value(uint32_t r0, uint32_t r1, f32x2 scale, f32x2 bias) {
    return fma2(kInt8 ? pack2((float)(int)r0, (float)(int)r1) : pack2(__uint_as_float(r0), __uint_as_float(r1)), scale, bias);
}

// One pixel's 8 consecutive channels; raw[4 * i + kFirst] and the next are the accumulators of pair i.
template <bool kInt8, int kAct, bool kRes, int kOut, int kFirst>
__device__ __forceinline__ void quad_pixel(const uint32_t (&raw)[16], const f32x2 (&sc)[4], const f32x2 (&bi)[4], const uint4& res, bool store,
                                           __half* y, int8_t* y2, f32x2 out2_scale) {
    constexpr bool kHalf = kOut != kQuadI8, kByte = kOut != kQuadF16;
    uint32_t o[4];
    int qv[8];
    const uint32_t rr[4] = {res.x, res.y, res.z, res.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        f32x2 v = quad_value<kInt8>(raw[4 * i + kFirst], raw[4 * i + kFirst + 1], sc[i], bi[i]);
        if (kRes) v = add2(v, cvt2(rr[i]));
        float a, b;
        unpack2(v, a, b);
        if (kAct == kQuadSilu) {
            a *= sigmoid_fast(a);
            b *= sigmoid_fast(b);
        }
        if (kByte && kAct == kQuadRelu) {      // int8 is quantised from the fp32 value
            a = fmaxf(a, 0.f);
            b = fmaxf(b, 0.f);
        }
        __half2 h = __floats2half2_rn(a, b);
        if ((kAct == kQuadRelu && !kByte) || kAct == kQuadRelu6) h = __hmax2(h, __half2half2(__ushort_as_half(0)));
        if (kAct == kQuadRelu6) h = __hmin2(h, __half2half2(__ushort_as_half(0x4600)));      // 6
        o[i] = *reinterpret_cast<const uint32_t*>(&h);
        if (kByte) {
            float qa, qb;
            unpack2(mul2(pack2(a, b), out2_scale), qa, qb);
            qv[2 * i] = __float2int_rn(qa);
            qv[2 * i + 1] = __float2int_rn(qb);
        }
    }
    if (!store) return;
    if (kHalf) *reinterpret_cast<uint4*>(y) = make_uint4(o[0], o[1], o[2], o[3]);
    if (kByte) *reinterpret_cast<uint2*>(y2) = make_uint2(sat_pack4(qv[0], qv[1], qv[2], qv[3]), sat_pack4(qv[4], qv[5], qv[6], qv[7]));
}

}  // namespace exb
