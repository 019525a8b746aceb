// Shared declarations of the C-ABI implementation: context, error reporting, launch helpers
// and the scalar conversion rules every kernel uses.
#pragma once
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdarg.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include <mutex>
#include <set>
#include <utility>

#include "../../include/excalibur_b200.h"

struct exb_ctx {
    int device;
    int sm_count;
    int smem_optin;          // max dynamic shared memory per block (opt-in)
    int* d_error;            // error word written by kernels whose bounded waits ran out: the device's view
    int* h_error;            // and the host's of the same mapped word
    int pdl;                 // launch the conv kernel with programmatic stream serialization (default 1; EXB_PDL=0 turns it off)
};

namespace exb {

// Record a message for exb_last_error_string() and return `code`.
int fail(int code, const char* fmt, ...);

// A failing runtime call is reported once and cleared (cudaGetLastError), so that it cannot be blamed on the next
// launch's check.
#define EXB_CUDA_TRY(expr)                                                                  \
    do {                                                                                    \
        cudaError_t e__ = (expr);                                                           \
        if (e__ != cudaSuccess) {                                                           \
            (void)cudaGetLastError();                                                       \
            return ::exb::fail(EXB_ERR_CUDA, "%s failed: %s (%s:%d)", #expr,                \
                               cudaGetErrorString(e__), __FILE__, __LINE__);                \
        }                                                                                   \
    } while (0)

#define EXB_REQUIRE(cond, ...)                                                              \
    do {                                                                                    \
        if (!(cond)) return ::exb::fail(EXB_ERR_BAD_ARG, __VA_ARGS__);                      \
    } while (0)

// Launch check.  cudaGetLastError returns AND clears the calling thread's error: a launch that was refused (or an
// error some other code of the process left behind) is reported by this call only and does not make every later
// launch of the library fail.  Sticky errors (a faulted context) keep coming back from the runtime by themselves.
inline int after_launch(const char* what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        return fail(EXB_ERR_CUDA, "launch of %s failed: %s", what, cudaGetErrorString(e));
    return EXB_OK;
}

// The dynamic shared-memory limit is an attribute of the kernel function on a device, shared by every thread that
// launches it: it is raised to the device's maximum once, never lowered, so that concurrent launches from several
// host threads (one pipeline replica per thread) cannot undercut each other.  Occupancy follows the bytes a launch
// actually asks for, not this limit.
template <typename K>
inline int raise_smem_limit(const exb_ctx* ctx, K kern) {
    static std::mutex attr_mutex;
    static std::set<std::pair<const void*, int>> raised;
    static thread_local std::pair<const void*, int> last;      // what this thread launched before, without the lock
    const auto key = std::make_pair(reinterpret_cast<const void*>(kern), ctx->device);
    if (last == key) return EXB_OK;
    std::lock_guard<std::mutex> lock(attr_mutex);
    if (!raised.count(key)) {
        cudaFuncAttributes fa;
        EXB_CUDA_TRY(cudaFuncGetAttributes(&fa, kern));      // static + dynamic shared memory share the device limit
        EXB_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, ctx->smem_optin - (int)fa.sharedSizeBytes));
        raised.insert(key);
    }
    last = key;
    return EXB_OK;
}

// Launch with programmatic stream serialization: the grid may be scheduled while the previous kernel of the stream
// drains.  Every kernel launched this way calls pdl_wait() before it touches global memory that another kernel
// writes or reads.
template <typename... KArgs, typename... Args>
inline int launch_pdl_cluster(const exb_ctx* ctx, const char* what, void (*kern)(KArgs...), dim3 grid, dim3 block, dim3 cluster, size_t smem,
                              cudaStream_t st, Args&&... args) {
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (ctx->pdl) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster.x * cluster.y * cluster.z > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = cluster.x;
        attr[n].val.clusterDim.y = cluster.y;
        attr[n++].val.clusterDim.z = cluster.z;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, KArgs(args)...);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return fail(EXB_ERR_CUDA, "launch of %s failed: %s", what, cudaGetErrorString(e));
    }
    return after_launch(what);
}
template <typename... KArgs, typename... Args>
inline int launch_pdl(const exb_ctx* ctx, const char* what, void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                      Args&&... args) {
    return launch_pdl_cluster(ctx, what, kern, grid, block, dim3(1), smem, st, static_cast<Args&&>(args)...);
}
// The same where the caller checks with after_launch() itself.
template <typename... KArgs, typename... Args>
inline void launch_overlapped(const exb_ctx* ctx, void (*kern)(KArgs...), dim3 grid, dim3 block, cudaStream_t st, Args&&... args) {
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ctx->pdl ? 1 : 0;
    (void)cudaLaunchKernelEx(&cfg, kern, KArgs(args)...);
}
// Let the next kernel of the stream be scheduled as soon as SMs free up / wait for the previous one's memory.
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Both, for kernels with nothing to do before the previous one is complete: they still gain the launch itself, 2 us of a
// small kernel's 4-8.
__device__ __forceinline__ void pdl_enter() {
    pdl_launch_dependents();
    pdl_wait();
}

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

inline size_t dtype_size(int dt) {
    switch (dt) {
    case EXB_F16: return 2;
    case EXB_I8: return 1;
    case EXB_F32: return 4;
    case EXB_I32: return 4;
    default: return 0;
    }
}

// ---- device-side scalar rules -------------------------------------------------------------
// Quantise, half away from zero then truncate and saturate: the reference's float32_to_int8.
__device__ __forceinline__ int quant_half_away(float v) {
    float t = v >= 0.f ? v + 0.5f : v - 0.5f;
    t = fminf(fmaxf(t, -128.f), 127.f);
    return (int)t;  // truncation toward zero
}
// Quantise, round half to even, saturate.
__device__ __forceinline__ int quant_rne(float v) {
    float t = rintf(v);
    t = fminf(fmaxf(t, -128.f), 127.f);
    return (int)t;
}

// Two floats in a 64-bit register pair: one instruction for two IEEE operations.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, const f32x2& c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 cvt2(uint32_t h) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h));
    return pack2(f.x, f.y);
}

// Four integers -> four int8 (saturated), packed little-endian in 32 bits.
__device__ __forceinline__ uint32_t sat_pack4(int q0, int q1, int q2, int q3) {
    uint32_t r;
    // cvt.pack.sat.s8.s32.b32 d, a, b, c:  d = (c << 16) | (sat8(a) << 8) | sat8(b)
    asm("{\n\t.reg .b32 t;\n\t"
        "cvt.pack.sat.s8.s32.b32 t, %4, %3, 0;\n\t"
        "cvt.pack.sat.s8.s32.b32 %0, %2, %1, t;\n\t}"
        : "=r"(r)
        : "r"(q0), "r"(q1), "r"(q2), "r"(q3));
    return r;
}
// Four floats -> four int8 (round half to even, saturate).
__device__ __forceinline__ uint32_t quant_pack4(float a, float b, float c, float d, float qscale) {
    return sat_pack4(__float2int_rn(a * qscale), __float2int_rn(b * qscale), __float2int_rn(c * qscale), __float2int_rn(d * qscale));
}

// 1 / (1 + e^-v) for the sigmoid-type activations: hardware reciprocal plus one Newton step (within 1 ulp of the
// IEEE division at a third of its instructions).  The exponent is clamped so that the denominator stays finite
// (the Newton step of an infinite one would be NaN); e^80 already gives a sigmoid of 2e-35.
__device__ __forceinline__ float sigmoid_fast(float v) {
    const float d = 1.f + __expf(fminf(-v, 80.f));
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    return fmaf(r, fmaf(-d, r, 1.f), r);
}

__device__ __forceinline__ float apply_act(float v, int act) {
    switch (act) {
    case EXB_ACT_NONE: return v;
    case EXB_ACT_RELU: return v >= 0.f ? v : 0.f;
    case EXB_ACT_RELU6_QUIRK: return (v >= 0.f && v <= 6.f) ? v : 0.f;
    case EXB_ACT_SIGMOID: return sigmoid_fast(v);
    case EXB_ACT_MISH: return v * tanhf(v > 20.f ? v : log1pf(expf(v)));   // ln(1 + e^v) = v to fp32 accuracy above 20
    case EXB_ACT_RELU6: return fminf(fmaxf(v, 0.f), 6.f);
    case EXB_ACT_SILU: return v * sigmoid_fast(v);
    case EXB_ACT_HARDSWISH: return v * fminf(fmaxf(fmaf(v, 1.f / 6.f, 0.5f), 0.f), 1.f);
    default: return v;
    }
}

// The same over a small register vector, with the selector outside the element loop: one uniform
// branch per vector instead of a switch per element.
template <int N>
__device__ __forceinline__ void apply_act_vec(float (&v)[N], int act) {
    if (act == EXB_ACT_NONE) return;
    if (act == EXB_ACT_RELU) {
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = fmaxf(v[i], 0.f);
    } else if (act == EXB_ACT_RELU6) {
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = fminf(fmaxf(v[i], 0.f), 6.f);
    } else if (act == EXB_ACT_SILU) {
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = v[i] * sigmoid_fast(v[i]);
    } else if (act == EXB_ACT_HARDSWISH) {
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = v[i] * fminf(fmaxf(fmaf(v[i], 1.f / 6.f, 0.5f), 0.f), 1.f);
    } else if (act == EXB_ACT_SIGMOID) {
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = sigmoid_fast(v[i]);
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) v[i] = apply_act(v[i], act);
    }
}

inline bool act_supported(int act) {
    return act == EXB_ACT_NONE || act == EXB_ACT_RELU || act == EXB_ACT_RELU6_QUIRK ||
           act == EXB_ACT_SIGMOID || act == EXB_ACT_MISH || act == EXB_ACT_RELU6 || act == EXB_ACT_SILU || act == EXB_ACT_HARDSWISH;
}

// Grid for a bandwidth-bound grid-stride kernel: enough CTAs to fill every SM a few times
// over, a multiple of the SM count, never more than the work needs.
inline int stream_grid(const exb_ctx* ctx, int64_t work_items, int threads, int ctas_per_sm = 8) {
    int64_t need = (work_items + threads - 1) / threads;
    int64_t cap = (int64_t)ctx->sm_count * ctas_per_sm;
    if (need < 1) need = 1;
    return (int)(need < cap ? need : cap);
}

}  // namespace exb
