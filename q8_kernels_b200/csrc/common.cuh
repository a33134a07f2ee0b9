// Shared helpers for the sm_100a kernels: error reporting for the C ABI,
// element-type tags, 8-bit casts with the two rounding flavours the reference
// uses, and small vector load/store utilities.
#pragma once

#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <stdint.h>
#include <stdio.h>

#include <atomic>

#include "../../include/q8_kernels_b200.h"

namespace q8k {

// ---------------------------------------------------------------- host-side errors
void set_error_detail(const char* fmt, ...);

#define Q8K_REQUIRE(cond, code, ...)                      \
    do {                                                  \
        if (!(cond)) {                                    \
            q8k::set_error_detail(__VA_ARGS__);           \
            return (code);                                \
        }                                                 \
    } while (0)

#define Q8K_CUDA_OK(expr)                                                          \
    do {                                                                           \
        cudaError_t _e = (expr);                                                   \
        if (_e != cudaSuccess) {                                                   \
            q8k::set_error_detail("%s failed: %s", #expr, cudaGetErrorString(_e)); \
            return Q8K_ERR_CUDA;                                                   \
        }                                                                          \
    } while (0)

int gemm_num_sms();                          // SMs of the current device (148 if it cannot be asked)

// Raise a kernel's dynamic shared memory limit, once per device (the call costs about 1 us, a launch 2.5).  The setting
// lives as long as the device's context; `done` belongs to the one kernel.
inline int allow_dynamic_smem(const void* kern, int bytes, std::atomic<uint64_t>& done) {
    int dev = 0;
    Q8K_CUDA_OK(cudaGetDevice(&dev));
    const uint64_t bit = dev < 64 ? 1ull << dev : 0ull;
    if ((done.load(std::memory_order_relaxed) & bit) != 0) return Q8K_OK;
    Q8K_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    done.fetch_or(bit, std::memory_order_relaxed);
    return Q8K_OK;
}

// Launch as a programmatic dependent of whatever runs before it on the stream: the kernel may become resident while its
// predecessor drains, so the launch latency and everything it does before pdl_wait() are hidden.  The kernel must call
// pdl_wait() in every thread before it touches global memory.  cluster > 1: CTAs per cluster along x.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_dependent(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, int cluster,
                                    Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kern, KArgs(args)...);
}

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// ---------------------------------------------------------------- programmatic dependent launch
// Wait until the kernels this one depends on have completed and their writes are visible (at once when it was launched
// without the attribute), then let the next kernel on the stream become resident as soon as every CTA has got here.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ---------------------------------------------------------------- element types
struct e4m3_t { uint8_t bits; };

template <int DT> struct DType;
template <> struct DType<Q8K_DT_F32>  { using type = float; };
template <> struct DType<Q8K_DT_F16>  { using type = __half; };
template <> struct DType<Q8K_DT_BF16> { using type = __nv_bfloat16; };
template <> struct DType<Q8K_DT_E4M3> { using type = e4m3_t; };
template <> struct DType<Q8K_DT_I8>   { using type = int8_t; };

inline int dtype_size(int dt) {
    switch (dt) {
        case Q8K_DT_F32: return 4;
        case Q8K_DT_F16: case Q8K_DT_BF16: return 2;
        case Q8K_DT_E4M3: case Q8K_DT_I8: return 1;
        default: return 0;
    }
}

// ---------------------------------------------------------------- scalar conversions
__device__ __forceinline__ float e4m3_to_float(uint8_t v) {
    __half_raw h = __nv_cvt_fp8_to_halfraw(v, __NV_E4M3);
    return __half2float(__half(h));
}

// fp32 -> e4m3, round to nearest even, saturating to +-448 (cvt.rn.satfinite).
// Used by the GEMM epilogue and inside attention.
__device__ __forceinline__ uint8_t float_to_e4m3_sat(float x) {
    return (uint8_t)__nv_cvt_float_to_fp8(x, __NV_SATFINITE, __NV_E4M3);
}
__device__ __forceinline__ uint16_t float2_to_e4m3x2_sat(float lo, float hi) {
    return (uint16_t)__nv_cvt_float2_to_fp8x2(make_float2(lo, hi), __NV_SATFINITE, __NV_E4M3);
}

// fp32 -> e4m3 the way the c10 software cast does it: round to nearest even,
// and anything that rounds beyond 448 (|x| > 464, inf, NaN) becomes NaN with
// the sign kept.  For |x| <= 464 this equals the saturating hardware cast.
__device__ __forceinline__ uint8_t float_to_e4m3_c10(float x) {
    uint8_t r = float_to_e4m3_sat(x);
    const bool overflow = !(fabsf(x) <= 464.0f);          // true for NaN as well
    if (overflow) r = (uint8_t)(0x7F | ((__float_as_uint(x) >> 24) & 0x80));
    return r;
}

// Eight values at once, same bytes as float_to_e4m3_c10 on each: four packed saturating conversions, and
// only if some |x| exceeds 464 or a NaN went in (the conversion returns 0x7F for it, whatever its sign)
// the element-wise form.
__device__ __forceinline__ uint2 pack8_e4m3_c10(const float (&x)[8]) {
    uint2 w;
    w.x = (uint32_t)float2_to_e4m3x2_sat(x[0], x[1]) | ((uint32_t)float2_to_e4m3x2_sat(x[2], x[3]) << 16);
    w.y = (uint32_t)float2_to_e4m3x2_sat(x[4], x[5]) | ((uint32_t)float2_to_e4m3x2_sat(x[6], x[7]) << 16);
    const float m = fmaxf(fmaxf(fmaxf(fabsf(x[0]), fabsf(x[1])), fmaxf(fabsf(x[2]), fabsf(x[3]))),
                          fmaxf(fmaxf(fabsf(x[4]), fabsf(x[5])), fmaxf(fabsf(x[6]), fabsf(x[7]))));
    const uint32_t nan_bytes = (((w.x & 0x7f7f7f7fu) + 0x01010101u) | ((w.y & 0x7f7f7f7fu) + 0x01010101u)) & 0x80808080u;
    if (m > 464.0f || nan_bytes != 0u) {
        union { uint2 v; uint8_t b[8]; } o;
#pragma unroll
        for (int j = 0; j < 8; ++j) o.b[j] = float_to_e4m3_c10(x[j]);
        w = o.v;
    }
    return w;
}

// Both values rounded to bf16 (nearest even) and widened again: one packed conversion and two bit moves.
__device__ __forceinline__ void round_through_bf16x2(float& a, float& b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    const uint32_t w = *reinterpret_cast<const uint32_t*>(&h);
    a = __uint_as_float(w << 16);
    b = __uint_as_float(w & 0xffff0000u);
}

template <typename T> __device__ __forceinline__ float to_float(T v);
template <> __device__ __forceinline__ float to_float<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_float<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float to_float<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <> __device__ __forceinline__ float to_float<e4m3_t>(e4m3_t v) { return e4m3_to_float(v.bits); }
template <> __device__ __forceinline__ float to_float<int8_t>(int8_t v) { return (float)v; }

// "plain C++ conversion" of the SIMT ops: bf16/fp16 RNE, e4m3 c10-style.
template <typename T> __device__ __forceinline__ T from_float(float v);
template <> __device__ __forceinline__ float from_float<float>(float v) { return v; }
template <> __device__ __forceinline__ __half from_float<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 from_float<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <> __device__ __forceinline__ e4m3_t from_float<e4m3_t>(float v) { return e4m3_t{float_to_e4m3_c10(v)}; }

// Four e4m3 bytes widened through two packed e4m3x2 -> f16x2 conversions (exact).
__device__ __forceinline__ void e4m3x4_to_float(uint32_t w, float (&o)[4]) {
    const __half2_raw lo = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(w & 0xffffu), __NV_E4M3);
    const __half2_raw hi = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(w >> 16), __NV_E4M3);
    const float2 a = __half22float2(__half2(lo)), c = __half22float2(__half2(hi));
    o[0] = a.x; o[1] = a.y; o[2] = c.x; o[3] = c.y;
}

// ---------------------------------------------------------------- vector access
// N consecutive elements of T <-> fp32 registers.  N * sizeof(T) must be 4, 8,
// 16 or 32 bytes and the address aligned to min(16, N*sizeof(T)).
template <int BYTES> struct Vec;
template <> struct Vec<2>  { using type = uint16_t; };
template <> struct Vec<4>  { using type = uint32_t; };
template <> struct Vec<8>  { using type = uint2; };
template <> struct Vec<16> { using type = uint4; };

template <typename T, int N>
__device__ __forceinline__ void load_vec(const T* __restrict__ p, float (&out)[N]) {
    constexpr int BYTES = N * sizeof(T);
    if constexpr (BYTES <= 16) {
        using V = typename Vec<BYTES>::type;
        union { V v; T e[N]; } u;
        u.v = *reinterpret_cast<const V*>(p);
#pragma unroll
        for (int i = 0; i < N; ++i) out[i] = to_float<T>(u.e[i]);
    } else {
        static_assert(BYTES % 16 == 0, "vector width");
        constexpr int PER = 16 / sizeof(T);
#pragma unroll
        for (int c = 0; c < BYTES / 16; ++c) {
            union { uint4 v; T e[PER]; } u;
            u.v = reinterpret_cast<const uint4*>(p)[c];
#pragma unroll
            for (int i = 0; i < PER; ++i) out[c * PER + i] = to_float<T>(u.e[i]);
        }
    }
}

template <typename T, int N>
__device__ __forceinline__ void store_vec(T* __restrict__ p, const float (&in)[N]) {
    constexpr int BYTES = N * sizeof(T);
    if constexpr (BYTES <= 16) {
        using V = typename Vec<BYTES>::type;
        if constexpr (__is_same(T, __nv_bfloat16) && N % 2 == 0) {
            union { V v; __nv_bfloat162 e2[N / 2]; } u;
#pragma unroll
            for (int i = 0; i < N; i += 2) u.e2[i / 2] = __floats2bfloat162_rn(in[i], in[i + 1]);
            *reinterpret_cast<V*>(p) = u.v;
        } else {
            union { V v; T e[N]; } u;
#pragma unroll
            for (int i = 0; i < N; ++i) u.e[i] = from_float<T>(in[i]);
            *reinterpret_cast<V*>(p) = u.v;
        }
    } else {
        static_assert(BYTES % 16 == 0, "vector width");
        constexpr int PER = 16 / sizeof(T);
#pragma unroll
        for (int c = 0; c < BYTES / 16; ++c) {
            if constexpr (sizeof(T) == 2 && __is_same(T, __nv_bfloat16)) {
                union { uint4 v; __nv_bfloat162 e2[4]; } u;    // packed conversions, same rounding
#pragma unroll
                for (int i = 0; i < 8; i += 2) u.e2[i / 2] = __floats2bfloat162_rn(in[c * 8 + i], in[c * 8 + i + 1]);
                reinterpret_cast<uint4*>(p)[c] = u.v;
            } else {
                union { uint4 v; T e[PER]; } u;
#pragma unroll
                for (int i = 0; i < PER; ++i) u.e[i] = from_float<T>(in[c * PER + i]);
                reinterpret_cast<uint4*>(p)[c] = u.v;
            }
        }
    }
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
// sm_100 packed fp32 pairs: one issue slot does two lanes of FMA-pipe work, each lane rounded as
// the scalar instruction would be.
__device__ __forceinline__ float2 ffma2(float2 a, float2 b, float2 c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(d)
        : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)),
          "l"(*reinterpret_cast<unsigned long long*>(&c)));
    return *reinterpret_cast<float2*>(&d);
}
__device__ __forceinline__ float2 fmul2(float2 a, float2 b) {
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;"
        : "=l"(d)
        : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)));
    return *reinterpret_cast<float2*>(&d);
}
__device__ __forceinline__ float2 fadd2(float2 a, float2 b) {
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;"
        : "=l"(d)
        : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)));
    return *reinterpret_cast<float2*>(&d);
}
__device__ __forceinline__ float2 fsub2(float2 a, float2 b) {
    unsigned long long d;
    asm("sub.rn.f32x2 %0, %1, %2;"
        : "=l"(d)
        : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)));
    return *reinterpret_cast<float2*>(&d);
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// The stride-1 stage of a pair of bf16 values: both as fp32, their sum and difference.  The mixed-precision add takes one
// operand as bf16, so only the other one has to be widened.  The fused Hadamard kernels are bound by instruction issue: this and the
// absmax taken before the 16-bit rounding (see hadamard.cu) bring int8 rows, 24576 x 2048, from 41.3 to 40.3 us,
// e4m3 rows from 35.1 to 34.1, with norm + modulation from 52.4 to 51.2 and 45.5 to 44.6; 6144 x 8192 48.5 -> 47.8 and
// 42.6 -> 42.2 (CUDA graphs).
__device__ __forceinline__ void butterfly_bf16x2(uint32_t w, float& sum, float& diff) {
    const float hi = __uint_as_float(w & 0xffff0000u);
    asm("{\n\t"
        ".reg .b16 lo, up;\n\t"
        "mov.b32 {lo, up}, %2;\n\t"
        "add.rn.f32.bf16 %0, lo, %3;\n\t"
        "sub.rn.f32.bf16 %1, lo, %3;\n\t"
        "}"
        : "=f"(sum), "=f"(diff)
        : "r"(w), "f"(hi));
}

// Walsh-Hadamard stages of stride FIRST (1 or 2) .. V/2 over V consecutive elements: stride 1 scalar, the rest packed
template <int V, int FIRST = 1>
__device__ __forceinline__ void butterfly_consecutive(float (&v)[V]) {
    if constexpr (FIRST == 1) {
#pragma unroll
        for (int i = 0; i < V; i += 2) {
            const float a = v[i], b = v[i + 1];
            v[i] = __fadd_rn(a, b);
            v[i + 1] = __fsub_rn(a, b);
        }
    }
#pragma unroll
    for (int st = 2; st < V; st <<= 1) {
#pragma unroll
        for (int h = 0; h < V / 2; h += 2) {                   // h, h+1 index two adjacent butterflies
            const int lo = h & (st - 1);
            const int i = ((h - lo) << 1) + lo;
            const float2 a = make_float2(v[i], v[i + 1]);
            const float2 b = make_float2(v[i + st], v[i + st + 1]);
            const float2 su = fadd2(a, b), di = fsub2(a, b);
            v[i] = su.x; v[i + 1] = su.y;
            v[i + st] = di.x; v[i + st + 1] = di.y;
        }
    }
}

// tanh-GELU of the reference (csrc/gemm/q8_matmul_bias.cu:29-33).
__device__ __forceinline__ float gelu_tanh_precise(float x) {
    const float u = 0.7978845608028654f * (x + 0.044715f * x * x * x);
    return 0.5f * x * (1.0f + tanhf(u));
}

}  // namespace q8k
