// Fast Walsh-Hadamard transform along the last dim, with an optional fused
// per-row absmax quantizer epilogue (the producer of the 8-bit GEMM operand).
//
// Arithmetic contract (csrc/fast_hadamard/fast_hadamard_transform_common.h:86-161
// of the reference): fp32 butterflies (a+b, a-b) applied for stride 1, 2, 4, ...
// in ascending order, then one multiply by `scale` and the output cast.  Every
// butterfly is one fp32 add, so any schedule that keeps the stage order gives the
// same bits.
//
// Two schedules, both one pass over HBM:
//  * rows of <= 256 elements: a group of G = n/8 lanes owns a row (8 elements
//    per lane, one 16-byte load), 32/G rows per warp; stages 0-2 in registers,
//    the rest by xor-shuffles inside the group.
//  * rows of 512 .. 16384 elements: 64 values per thread; stages 0-5 run in registers on consecutive
//    elements, the rest after one padded shared-memory exchange (two above 2048), all on packed fp32
//    pairs; no shuffles.

#include <type_traits>
#include "common.cuh"

namespace q8k {

enum class Epilogue { Cast, Quant };

template <int N>
__device__ __forceinline__ void fwht_regs(float (&v)[N]) {
#pragma unroll
    for (int s = 1; s < N; s <<= 1) {
#pragma unroll
        for (int j = 0; j < N / 2; ++j) {
            const int lo = j & (s - 1);
            const int i = ((j - lo) << 1) + lo;
            const float a = v[i], b = v[i + s];
            v[i] = __fadd_rn(a, b);
            v[i + s] = __fsub_rn(a, b);
        }
    }
}

// One butterfly stage between lanes that differ in bit `mask`.
template <int N>
__device__ __forceinline__ void fwht_lanes(float (&v)[N], int lane, int mask) {
    const bool upper = (lane & mask) != 0;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const float other = __shfl_xor_sync(0xffffffffu, v[i], mask);
        v[i] = upper ? __fsub_rn(other, v[i]) : __fadd_rn(v[i], other);
    }
}

// Round the scaled transform to the dtype the unfused chain would have stored.
template <typename T> __device__ __forceinline__ float round_through(float v) {
    return to_float<T>(from_float<T>(v));
}

template <typename Tq> __device__ __forceinline__ uint8_t quantize_one(float y) {
    if constexpr (std::is_same_v<Tq, int8_t>) return (uint8_t)(int8_t)(int)roundf(y);
    else return float_to_e4m3_c10(y);
}

template <int N> struct ByteVec;
template <> struct ByteVec<1>  { using type = uint8_t; };
template <> struct ByteVec<2>  { using type = uint16_t; };
template <> struct ByteVec<4>  { using type = uint32_t; };
template <> struct ByteVec<8>  { using type = uint2; };
template <> struct ByteVec<16> { using type = uint4; };

template <typename T, int N>
__device__ __forceinline__ void store_elems(T* p, const float (&v)[N]) {
    using V = typename ByteVec<N * sizeof(T)>::type;
    if constexpr (std::is_same_v<T, __nv_bfloat16> && N % 2 == 0) {
        union { V vec; __nv_bfloat162 e2[N / 2]; } u;          // packed conversions, same rounding
#pragma unroll
        for (int i = 0; i < N; i += 2) u.e2[i / 2] = __floats2bfloat162_rn(v[i], v[i + 1]);
        *reinterpret_cast<V*>(p) = u.vec;
    } else {
        union { V vec; T e[N]; } u;
#pragma unroll
        for (int i = 0; i < N; ++i) u.e[i] = from_float<T>(v[i]);
        *reinterpret_cast<V*>(p) = u.vec;
    }
}

template <typename Tq, int N>
__device__ __forceinline__ void store_quant(Tq* p, const float (&v)[N], float qscale, bool zero_row) {
    using V = typename ByteVec<N>::type;
    union { V vec; uint8_t b[N]; } u;
#pragma unroll
    for (int i = 0; i < N; ++i) u.b[i] = quantize_one<Tq>(zero_row ? 0.f : __fmul_rn(v[i], qscale));
    *reinterpret_cast<V*>(p) = u.vec;
}

// ------------------------------------------------------------------ small rows
// LOG_G = log2(lanes per row).  Tout is the cast output type (Cast) or the
// quantised type (Quant: int8_t or e4m3_t).
template <typename Tin, typename Tout, int LOG_G, Epilogue EPI>
__global__ void __launch_bounds__(128)
hadamard_small_kernel(const Tin* __restrict__ x, Tout* __restrict__ out, float* __restrict__ scales,
                      int64_t rows, int dim, int64_t x_row_stride, float scale) {
    constexpr int G = 1 << LOG_G;
    constexpr int ROWS_PER_CTA = 128 / G;
    const int lane = threadIdx.x & 31;
    const int sub = threadIdx.x & (G - 1);
    const int64_t row = (int64_t)blockIdx.x * ROWS_PER_CTA + (threadIdx.x >> LOG_G);
    const bool row_ok = row < rows;
    const int e = sub * 8;

    float v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = 0.f;
    if (row_ok && e < dim) load_vec<Tin, 8>(x + row * x_row_stride + e, v);

    fwht_regs<8>(v);
#pragma unroll
    for (int m = 1; m < G; m <<= 1) fwht_lanes<8>(v, lane, m);

    if constexpr (EPI == Epilogue::Cast) {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = __fmul_rn(v[j], scale);
        if (row_ok && e < dim) store_elems<Tout, 8>(out + row * (int64_t)dim + e, v);
    } else {
        float amax = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            v[j] = round_through<Tin>(__fmul_rn(v[j], scale));
            if (e + j < dim) amax = fmaxf(amax, fabsf(v[j]));
        }
#pragma unroll
        for (int m = 1; m < G; m <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, m));
        const float qmax = std::is_same_v<Tout, int8_t> ? 127.0f : 448.0f;
        const float qscale = __fdiv_rn(qmax, amax);
        if (row_ok && e < dim) store_quant<Tout, 8>(out + row * (int64_t)dim + e, v, qscale, amax == 0.f);
        if (row_ok && sub == 0) scales[row] = __fdiv_rn(1.0f, qscale);
    }
}

// ------------------------------------------------------------------ large rows
// Butterflies work on packed fp32 pairs (add/sub.f32x2), so a stage costs half an instruction per element; only the
// stride-1 stage is scalar.

// Layout of a phase that butterflies bits [LO, LO+B): thread t owns groups j = 0 .. 2^B-1 of
// C = V >> B consecutive elements each.  The thread index supplies the other bits of the
// element index: its low LO-log2(C) bits sit below the group bits, the rest above them.
template <int LOG_V, int B, int LO>
struct PhaseLayout {
    static constexpr int LOG_C = LOG_V - B;
    static constexpr int C = 1 << LOG_C;
    static constexpr int G = 1 << B;
    static constexpr int BITS = B;
    static constexpr int LOW = LO;
    static_assert(LO >= LOG_C, "group bits must lie above the run bits");
    __device__ static __forceinline__ int elem(int t, int j) {
        constexpr int LOWT = LO - LOG_C;
        return ((t & ((1 << LOWT) - 1)) << LOG_C) + (j << LO) + ((t >> LOWT) << (LO + B));
    }
};

// butterflies between groups (stride = whole groups of C >= 4 elements): all packed
template <typename L, int V>
__device__ __forceinline__ void butterfly_groups(float (&v)[V]) {
#pragma unroll
    for (int s = 0; s < L::BITS; ++s) {
        const int gs = 1 << s;
#pragma unroll
        for (int h = 0; h < L::G / 2; ++h) {
            const int lo = h & (gs - 1);
            const int j = ((h - lo) << 1) + lo;
#pragma unroll
            for (int c = 0; c < L::C; c += 2) {
                const float2 a = make_float2(v[j * L::C + c], v[j * L::C + c + 1]);
                const float2 b = make_float2(v[(j + gs) * L::C + c], v[(j + gs) * L::C + c + 1]);
                const float2 su = fadd2(a, b), di = fsub2(a, b);
                v[j * L::C + c] = su.x; v[j * L::C + c + 1] = su.y;
                v[(j + gs) * L::C + c] = di.x; v[(j + gs) * L::C + c + 1] = di.y;
            }
        }
    }
}

// Units of whole warps walk over the rows (a grid of as many CTAs as fit the device): a row of up to 2048 elements
// belongs to one warp or a part of one, a longer row to one CTA.  A thread has 64 values.  Per row: the raw elements
// were copied into the unit's staging buffer by cp.async while the row before was being transformed; a thread reads
// its 64 consecutive elements, does stages 0-5 in registers, and the remaining stages after one exchange through
// shared memory (two above 2048).  The first exchange never leaves a warp and the staged elements are read by the
// warp that copied them, so rows of up to 2048 elements need no block barrier at all and longer ones two (three with
// norm + modulation: the mean square is summed over the CTA).
//
// Bound by instruction issue and the FMA pipe (add/sub.f32x2 issue every second clock: 11 stages are 11 clocks per
// element and scheduler), no longer by barriers and shared memory: 8 bytes per element of exchange (16 above 2048)
// and 2 x the input size of staging, all accesses conflict-free with immediate offsets.  128 registers, 16 warps per SM.
// Measured, 24576 x 2048, bf16 in, CUDA graph over inputs larger than L2 (one CTA per row pair, block-wide barriers,
// two exchanges before): bf16 out 43.6 -> 33.7 us (0.92 of the copy rate), e4m3 rows 45.3 -> 34.1 us, int8 rows
// 47.1 -> 40.3 us (one F2I per element on the 8-clock conversion unit), with norm + modulation 72.3 -> 51.2 us (int8).
// 6144 x 8192: 49.5 -> 41.2, 50.1 -> 42.2, 53.2 -> 47.8, 109 -> 73.7 us.  Tried: 128 values per thread for 4096 and
// 8192 (one exchange, half the warps; 59 us for int8 rows of 8192), XOR swizzles instead of pads (39.4 us, e4m3 rows).

__device__ __forceinline__ void cp_async_zfill(uint32_t dst, const void* src, int cp_bytes, bool valid) {
    if (cp_bytes == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(dst), "l"(src), "r"(valid ? 8 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// NORM_MOD adds the block's pre-linear prologue in front of the transform, with the bf16 roundings
// of the separate ops it replaces: n = bf16(x * rsqrt(mean x^2)); u = bf16(bf16(n * bf16(1 + s)) + h)
// where s, h are the per-batch modulation rows (bf16 [rows / rows_per_mod, dim]).  A CTA stays inside one batch entry
// and keeps its two modulation rows in shared memory.
// int8 rows (Cast only) are dequantised on the way in: v = bf16(q * scales[row]), the weight of a backward pass.
// FULL: dim is the power of two itself, so no element of a row needs a bounds test.

// Raw staging: position of the 16-byte chunk c (row order) of a row whose threads own CPT chunks each, such
// that eight consecutive threads reading their k-th chunk touch eight different bank groups.
template <int CPT>
__device__ __forceinline__ constexpr int raw_pos(int c) {
    if constexpr (CPT >= 8) return c ^ ((c / CPT) & 7);
    else return c ^ ((c / CPT / (8 / CPT)) & (CPT - 1));
}

// fp32 exchange, V = 64: natural element order in 16-byte chunks, one pad chunk after the 16 chunks that a
// thread writes (eight consecutive threads hit eight bank groups) and, where a layout with runs of 8 elements
// reads it, one more after every 8.  Pads instead of an XOR: the position is thread term + constant, so every
// access has an immediate offset and costs no address arithmetic.
template <bool PAD8>
__device__ __forceinline__ constexpr int xpos(int q) { return q + (q >> 4) + (PAD8 ? q >> 3 : 0); }

template <typename L, bool PAD8, bool WRITE>
__device__ __forceinline__ void xch_access(char* xb, float (&v)[64], int t) {
    const int e0 = L::elem(t, 0);
    char* base = xb + (xpos<PAD8>(e0 >> 2) << 4) + (L::C < 4 ? ((e0 >> 1) & 1) << 3 : 0);
#pragma unroll
    for (int j = 0; j < L::G; ++j) {
        if constexpr (L::C >= 4) {
#pragma unroll
            for (int k = 0; k < L::C / 4; ++k) {
                float4* a = reinterpret_cast<float4*>(base + (xpos<PAD8>(((j << L::LOW) >> 2) + k) << 4));
                float* r = v + j * L::C + 4 * k;
                if constexpr (WRITE) *a = make_float4(r[0], r[1], r[2], r[3]);
                else { const float4 f = *a; r[0] = f.x; r[1] = f.y; r[2] = f.z; r[3] = f.w; }
            }
        } else {
            float2* a = reinterpret_cast<float2*>(base + (xpos<PAD8>((j << L::LOW) >> 2) << 4));
            if constexpr (WRITE) *a = make_float2(v[2 * j], v[2 * j + 1]);
            else { const float2 f = *a; v[2 * j] = f.x; v[2 * j + 1] = f.y; }
        }
    }
}

template <typename Tin, int LOG_N, bool NORM_MOD>
struct StreamGeo {
    static constexpr int LOG_V = 6, V = 64;                    // values per thread
    static constexpr int N = 1 << LOG_N, T = N / V;
    static constexpr int R = LOG_N - LOG_V;                    // stages left after the register phase
    static constexpr int B1 = R <= LOG_V - 1 ? R : (R + 1) / 2;   // one exchange while runs of two elements remain, else two
    static constexpr int B2 = R - B1;
    static_assert(B1 <= 5, "the first exchange stays inside a warp");
    static constexpr bool PAD8 = LOG_V - B1 == 3 || (B2 > 0 && LOG_V - B2 == 3);
    static constexpr int UNIT = T < 32 ? 32 : T;               // threads that work on the same rows
    static constexpr int RPU = UNIT / T;                       // rows per unit and turn
    static constexpr int THREADS = T > 32 ? T : 128;
    static constexpr int UNITS = THREADS / UNIT;
    static constexpr int RAW = RPU * N * (int)sizeof(Tin);     // bytes per unit
    static constexpr int XROW = (N / 4 + N / 64 + (PAD8 ? N / 32 : 0)) * 16;
    static constexpr int XCH = RPU * XROW;
    static constexpr int MOD = NORM_MOD ? 2 * N * 2 : 0;       // bytes per CTA: 1 + scale and shift rows (bf16)
    static constexpr int smem(int units) { return units * (RAW + XCH) + MOD; }
    static constexpr int SMEM = smem(UNITS);
    static constexpr int BY_SMEM = (228 * 1024) / (SMEM + 1024);
    static constexpr int BY_REGS = 65536 / (THREADS * 128);
    static constexpr int CTAS = BY_SMEM < BY_REGS ? BY_SMEM : BY_REGS;
};

template <typename Tin, typename Tout, int LOG_N, Epilogue EPI, bool NORM_MOD, bool FULL>
__global__ void __launch_bounds__(StreamGeo<Tin, LOG_N, NORM_MOD>::THREADS, StreamGeo<Tin, LOG_N, NORM_MOD>::CTAS)
hadamard_stream_kernel(const Tin* __restrict__ x, Tout* __restrict__ out, float* __restrict__ scales, unsigned rows, int dim,
                       int64_t x_row_stride, float scale, const __nv_bfloat16* __restrict__ mod_scale,
                       const __nv_bfloat16* __restrict__ mod_shift, unsigned rows_per_mod, unsigned blocks_per_mod) {
    constexpr bool DEQ = std::is_same_v<Tin, int8_t>;
    static_assert(!DEQ || EPI == Epilogue::Cast, "int8 rows are only transformed, not quantised again");
    using Geo = StreamGeo<Tin, LOG_N, NORM_MOD>;
    constexpr int N = Geo::N, V = Geo::V, T = Geo::T, UNIT = Geo::UNIT, RPU = Geo::RPU, LOG_V = Geo::LOG_V;
    constexpr int B1 = Geo::B1, B2 = Geo::B2;
    constexpr bool PAD8 = Geo::PAD8;
    using L0 = PhaseLayout<LOG_V, 0, LOG_V>;
    using L1 = PhaseLayout<LOG_V, B1, LOG_V>;
    using L2 = PhaseLayout<LOG_V, B2, LOG_V + B1>;
    using LF = std::conditional_t<(B2 > 0), L2, L1>;
    constexpr int C = LF::C;
    static_assert(C >= 2 && C <= 8, "runs of 2, 4 or 8 elements");
    constexpr bool IN8 = sizeof(Tin) == 1;
    constexpr int CPB = IN8 ? 8 : 16;                          // bytes per copy: 8 elements, so a copy never straddles dim
    constexpr int ITEMS = V / 8;                               // copies per thread and row
    constexpr int CPT = V * (int)sizeof(Tin) / 16;             // 16-byte chunks per thread and row
    constexpr int W = T < 32 ? T : 32;                         // threads of a row within one warp: they copy what they read

    extern __shared__ __align__(16) char stream_smem[];
    // two reductions of a row over the CTA's warps, an array each: a warp may be a row ahead when a slower one reads
    __shared__ float red_ss[8], red_max[8];
    static_assert(T <= 32 || B2 > 0, "the second exchange's barrier separates each array's reads from its next writes");
    const int tu = threadIdx.x % UNIT;
    const int unit = threadIdx.x / UNIT;
    const int t = tu % T;
    const int r_in = tu / T;
    char* raw = stream_smem + unit * Geo::RAW + r_in * (N * (int)sizeof(Tin));
    const int units = NORM_MOD && Geo::UNITS > 1 ? (int)blockDim.x / UNIT : Geo::UNITS;
    char* xch = stream_smem + units * Geo::RAW + unit * Geo::XCH + r_in * Geo::XROW;
    const uint32_t raw_addr = (uint32_t)__cvta_generic_to_shared(raw);
    const unsigned mod = NORM_MOD ? blockIdx.x / blocks_per_mod : 0u;
    const unsigned blk = NORM_MOD ? blockIdx.x - mod * blocks_per_mod : blockIdx.x;
    const unsigned first = mod * rows_per_mod;
    const unsigned count = NORM_MOD ? (rows - first < rows_per_mod ? rows - first : rows_per_mod) : rows;   // rows of this group
    const unsigned step = (NORM_MOD ? blocks_per_mod : gridDim.x) * (unsigned)(units * RPU);
    unsigned rel = (blk * (unsigned)units + (unsigned)unit) * (unsigned)RPU;   // first row of this unit, relative to the group

    auto load_rows = [&](unsigned rel0) {
        const bool ok = rel0 + r_in < count;
        const Tin* xr = x + (int64_t)(ok ? first + rel0 + r_in : first) * x_row_stride;
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            const int item = (t / W) * (W * ITEMS) + k * W + t % W;
            const bool valid = ok && (FULL || item * 8 < dim);
            const int c = IN8 ? item >> 1 : item;
            cp_async_zfill(raw_addr + ((uint32_t)raw_pos<CPT>(c) << 4) + (IN8 ? (uint32_t)(item & 1) << 3 : 0u),
                           xr + (valid ? item * 8 : 0), CPB, valid);
        }
        cp_async_commit();
    };
    pdl_wait();
    pdl_release();
    load_rows(rel);

    __nv_bfloat16* mod_smem = reinterpret_cast<__nv_bfloat16*>(stream_smem + units * (Geo::RAW + Geo::XCH));
    if constexpr (NORM_MOD) {
        // 1 + scale and shift rows of this CTA's batch entry, staged like the raw rows (bf16: CPT = V / 8)
        const __nv_bfloat16* sc = mod_scale + (int64_t)mod * dim;
        const __nv_bfloat16* sh = mod_shift + (int64_t)mod * dim;
        const __nv_bfloat162 one2 = __floats2bfloat162_rn(1.0f, 1.0f);
        auto load_mod = [&](int stride) {
            for (int c = threadIdx.x; c < N / 8; c += stride) {
                uint4 s8 = make_uint4(0, 0, 0, 0), h8 = make_uint4(0, 0, 0, 0);
                if (FULL || c * 8 < dim) {
                    s8 = *reinterpret_cast<const uint4*>(sc + c * 8);
                    h8 = *reinterpret_cast<const uint4*>(sh + c * 8);
                }
                uint32_t* w = &s8.x;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const __nv_bfloat162 m1 = __hadd2_rn(one2, *reinterpret_cast<const __nv_bfloat162*>(w + j));
                    w[j] = *reinterpret_cast<const uint32_t*>(&m1);
                }
                reinterpret_cast<uint4*>(mod_smem)[raw_pos<CPT>(c)] = s8;
                reinterpret_cast<uint4*>(mod_smem + N)[raw_pos<CPT>(c)] = h8;
            }
        };
        if (units == Geo::UNITS) load_mod(Geo::THREADS);       // a constant stride: all loads at once
        else load_mod(units * UNIT);
        __syncthreads();
    }

    for (; rel < count; rel += step) {
        const unsigned row = first + rel + r_in;
        const bool row_ok = rel + r_in < count;
        cp_async_wait_all();
        __syncwarp();                                          // the row has landed; the exchange of the row before has been read
        float v[V];
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            if constexpr (IN8) {
                if (k % 2 == 0) {
                    const uint4 u = *reinterpret_cast<const uint4*>(raw + (raw_pos<CPT>(t * CPT + k / 2) << 4));
                    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        float f[4];
                        if constexpr (DEQ) {
                            const float rs = row_ok ? scales[row] : 0.f;
#pragma unroll
                            for (int j = 0; j < 4; ++j) f[j] = __fmul_rn((float)(int8_t)(w[i] >> (8 * j)), rs);
                            round_through_bf16x2(f[0], f[1]);
                            round_through_bf16x2(f[2], f[3]);
                        } else {
                            e4m3x4_to_float(w[i], f);
                        }
#pragma unroll
                        for (int j = 0; j < 4; ++j) v[k * 8 + i * 4 + j] = f[j];
                    }
                }
            } else {
                const uint4 u = *reinterpret_cast<const uint4*>(raw + (raw_pos<CPT>(t * CPT + k) << 4));
                const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if constexpr (NORM_MOD) {
                        v[k * 8 + 2 * i] = __uint_as_float(w[i] << 16);
                        v[k * 8 + 2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
                    } else {
                        butterfly_bf16x2(w[i], v[k * 8 + 2 * i], v[k * 8 + 2 * i + 1]);
                    }
                }
            }
        }
        if constexpr (NORM_MOD) {
            // rows of up to 2048 elements: partial sums of 32 elements; longer rows: of 64.  Then a tree over the
            // partial sums of 1024 (2048) elements each, and those in sequence.
            constexpr int PS = T <= 32 ? 32 : 64;
            float ss = 0.f;
#pragma unroll
            for (int i = 0; i < PS; ++i) ss = fmaf(v[i], v[i], ss);
            if constexpr (PS == 32) {
                float ss1 = 0.f;
#pragma unroll
                for (int i = 32; i < 64; ++i) ss1 = fmaf(v[i], v[i], ss1);
                ss += ss1;
            }
#pragma unroll
            for (int m = 1; m < W; m <<= 1) ss += __shfl_xor_sync(0xffffffffu, ss, m);
            if constexpr (T > 32) {
                if ((threadIdx.x & 31) == 0) red_ss[threadIdx.x >> 5] = ss;
                __syncthreads();
                ss = red_ss[0];
#pragma unroll
                for (int k = 1; k < T / 32; ++k) ss += red_ss[k];
            }
            const float rr = rsqrtf(ss * (1.0f / (float)dim));
#pragma unroll
            for (int k = 0; k < ITEMS; ++k) {
                // packed bf16 arithmetic gives exactly the roundings of the separate ops: a product of two bf16
                // values is exact in fp32, and a sum of two is either exact in fp32 or so lopsided that both
                // roundings return the larger operand; _rn keeps multiply and add from fusing.  (Elements beyond
                // dim are zero in x and in both rows, and stay zero.)
                const int pos = raw_pos<CPT>(t * CPT + k);
                const uint4 s8 = reinterpret_cast<const uint4*>(mod_smem)[pos];
                const uint4 h8 = reinterpret_cast<const uint4*>(mod_smem + N)[pos];
                const uint32_t sw[4] = {s8.x, s8.y, s8.z, s8.w}, hw[4] = {h8.x, h8.y, h8.z, h8.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 xr2 = fmul2(make_float2(v[k * 8 + 2 * i], v[k * 8 + 2 * i + 1]), make_float2(rr, rr));
                    const __nv_bfloat162 n = __floats2bfloat162_rn(xr2.x, xr2.y);
                    const __nv_bfloat162 u = __hadd2_rn(__hmul2_rn(n, *reinterpret_cast<const __nv_bfloat162*>(sw + i)),
                                                        *reinterpret_cast<const __nv_bfloat162*>(hw + i));
                    const uint32_t uw = *reinterpret_cast<const uint32_t*>(&u);
                    butterfly_bf16x2(uw, v[k * 8 + 2 * i], v[k * 8 + 2 * i + 1]);
                }
            }
        }
        butterfly_consecutive<V, IN8 ? 1 : 2>(v);
        xch_access<L0, PAD8, true>(xch, v, t);
        __syncwarp();
        load_rows(rel + step);                                 // this warp has read its part of the staging buffer
        xch_access<L1, PAD8, false>(xch, v, t);
        butterfly_groups<L1, V>(v);
        if constexpr (B2 > 0) {
            xch_access<L1, PAD8, true>(xch, v, t);             // a thread overwrites what it alone has read
            __syncthreads();
            xch_access<L2, PAD8, false>(xch, v, t);
            butterfly_groups<L2, V>(v);
        }

        const float2 sc2 = make_float2(scale, scale);
#pragma unroll
        for (int i = 0; i < V; i += 2) {
            const float2 m = fmul2(make_float2(v[i], v[i + 1]), sc2);
            v[i] = m.x; v[i + 1] = m.y;
        }
        Tout* outr = out + (int64_t)row * dim;
        // Group j of this thread starts at element e0 + (j << LOW), inside the row if (j << LOW) < lim.  The asm keeps the
        // compiler from holding up to 32 such comparisons in registers across the rows (168 of them, or spills).
        const int e0 = LF::elem(t, 0);
        int lim = dim - e0;
        if constexpr (!FULL) asm volatile("" : "+r"(lim));
        auto in_row = [&](int j) { return FULL || (j << LF::LOW) < lim; };
        // Of 32 groups, eight at a time whose elements all lie beyond dim are neither rounded, reduced nor quantised.
        // Measured, 6144 x 1536 (neither of the two before -> now): int8 rows 16.7 -> 14.0 us, e4m3 rows 12.9 -> 12.6 us;
        // 6144 x 1544, where nothing can be skipped: 16.9 -> 15.3 us.
        constexpr int SKIP = !FULL && LF::G == 32 ? 8 : LF::G;
        auto any_in_row = [&](int j) { return SKIP == LF::G || (j << LF::LOW) < dim; };
        if constexpr (EPI == Epilogue::Cast) {
            if constexpr (std::is_same_v<Tout, __nv_bfloat16>) {
#pragma unroll
                for (int j = 0; j < LF::G; ++j) {
                    float o[C];
#pragma unroll
                    for (int i = 0; i < C; ++i) o[i] = v[j * C + i];
                    if (row_ok && in_row(j)) store_elems<Tout, C>(outr + e0 + (j << LF::LOW), o);
                }
            } else {
                static_assert(std::is_same_v<Tout, e4m3_t>, "cast to bf16 or e4m3");
#pragma unroll
                for (int f = 0; f < V; f += 8) {
                    float o[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) o[i] = v[f + i];
                    union { uint2 w; typename ByteVec<C>::type b[8 / C]; } u;
                    u.w = pack8_e4m3_c10(o);
#pragma unroll
                    for (int g = 0; g < 8 / C; ++g) {
                        const int j = f / C + g;
                        if (row_ok && in_row(j))
                            *reinterpret_cast<typename ByteVec<C>::type*>(reinterpret_cast<uint8_t*>(outr) + e0 + (j << LF::LOW)) = u.b[g];
                    }
                }
            }
        } else {
            // Round to the input dtype (what the unfused chain stores) and take the row's absmax: of the fp32 values, rounded
            // afterwards (bf16), or of the e4m3 bytes widened to fp16 pairs (exact).  NaNs do not count, as with fmaxf.
            uint32_t pk[V / (IN8 ? 4 : 2)];
            float amax;
            if constexpr (IN8) {
                __half2 m2 = __floats2half2_rn(0.f, 0.f);
#pragma unroll
                for (int jc = 0; jc < LF::G; jc += SKIP) {
                    if (any_in_row(jc)) {
#pragma unroll
                        for (int f = jc * C; f < (jc + SKIP) * C; f += 8) {
                            float o[8];
#pragma unroll
                            for (int i = 0; i < 8; ++i) o[i] = v[f + i];
                            const uint2 w = pack8_e4m3_c10(o);
                            pk[f / 4] = w.x;
                            pk[f / 4 + 1] = w.y;
#pragma unroll
                            for (int g = 0; g < 4; ++g) {
                                const uint32_t ww = g < 2 ? w.x : w.y;
                                const __half2_raw h = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(g & 1 ? ww >> 16 : ww & 0xffffu), __NV_E4M3);
                                if (in_row((f + 2 * g) / C)) m2 = __hmax2(m2, __habs2(__half2(h)));
                            }
                        }
                    }
                }
                amax = fmaxf(__low2float(m2), __high2float(m2));
            } else {
                float mx[2] = {0.f, 0.f};
#pragma unroll
                for (int jc = 0; jc < LF::G; jc += SKIP) {
                    if (any_in_row(jc)) {
#pragma unroll
                        for (int f = jc * C; f < (jc + SKIP) * C; f += 2) {
                            const __nv_bfloat162 w = __floats2bfloat162_rn(v[f], v[f + 1]);
                            pk[f / 2] = *reinterpret_cast<const uint32_t*>(&w);
                            float& m = mx[(f / 2) & 1];
                            if (in_row(f / C)) asm("max.f32 %0, %0, %1, %2;" : "+f"(m) : "f"(fabsf(v[f])), "f"(fabsf(v[f + 1])));
                        }
                    }
                }
                amax = __bfloat162float(__float2bfloat16_rn(fmaxf(mx[0], mx[1])));   // rounding keeps the order
            }
#pragma unroll
            for (int m = 1; m < (T < 32 ? T : 32); m <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, m));
            if constexpr (T > 32) {
                if ((threadIdx.x & 31) == 0) red_max[threadIdx.x >> 5] = amax;
                __syncthreads();
                amax = red_max[0];
#pragma unroll
                for (int k = 1; k < T / 32; ++k) amax = fmaxf(amax, red_max[k]);
            }
            const float qmax = std::is_same_v<Tout, int8_t> ? 127.0f : 448.0f;
            const float qscale = __fdiv_rn(qmax, amax);
            if (row_ok && t == 0) scales[row] = __fdiv_rn(1.0f, qscale);
            const float qmul = amax == 0.f ? 0.f : qscale;     // an all-zero row quantises to zeros (0 * 0, not 0 * inf)
            const float2 q2 = make_float2(qmul, qmul);
            constexpr int P = C < 4 ? C : 4;                   // values per packing step
#pragma unroll
            for (int jc = 0; jc < LF::G; jc += SKIP) {
                if (any_in_row(jc)) {
#pragma unroll
                    for (int j = jc; j < jc + SKIP; ++j) {
                        union { typename ByteVec<C>::type b; uint32_t w[C >= 4 ? C / 4 : 1]; } u;
#pragma unroll
                        for (int i = 0; i < C; i += P) {
                            float y[4];
#pragma unroll
                            for (int h = 0; h < P; h += 2) {
                                const int f = j * C + i + h;
                                float2 a;
                                if constexpr (IN8) {
                                    const uint32_t ww = pk[f / 4];
                                    const __half2_raw hr = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(f & 2 ? ww >> 16 : ww & 0xffffu), __NV_E4M3);
                                    a = __half22float2(__half2(hr));
                                } else {
                                    a = make_float2(__uint_as_float(pk[f / 2] << 16), __uint_as_float(pk[f / 2] & 0xffff0000u));
                                }
                                a = fmul2(a, q2);
                                // round half away from zero (C round()) of |y| < 2^22: adding the largest float below 0.5 with
                                // y's sign and truncating gives floor(|y| + 0.5) for every fp32 y, ties included
                                if constexpr (std::is_same_v<Tout, int8_t>)
                                    a = fadd2(a, make_float2(copysignf(0.49999997f, a.x), copysignf(0.49999997f, a.y)));
                                y[h] = a.x;
                                y[h + 1] = a.y;
                            }
                            uint32_t w;
                            if constexpr (std::is_same_v<Tout, int8_t>) {
                                w = __byte_perm((uint32_t)__float2int_rz(y[0]), (uint32_t)__float2int_rz(y[1]), 0x0040);
                                if constexpr (P == 4)
                                    w = __byte_perm(w, __byte_perm((uint32_t)__float2int_rz(y[2]), (uint32_t)__float2int_rz(y[3]), 0x0040), 0x5410);
                            } else {
                                // |y| <= 448 (1 + 2^-23) for finite rows, where the saturating cast and the c10 cast (overflow ->
                                // NaN beyond 464) agree; a NaN stays a NaN in both
                                w = (uint32_t)float2_to_e4m3x2_sat(y[0], y[1]);
                                if constexpr (P == 4) w |= (uint32_t)float2_to_e4m3x2_sat(y[2], y[3]) << 16;
                            }
                            u.w[i / 4] = w;
                        }
                        if (row_ok && in_row(j))
                            *reinterpret_cast<typename ByteVec<C>::type*>(reinterpret_cast<uint8_t*>(outr) + e0 + (j << LF::LOW)) = u.b;
                    }
                }
            }
        }
        // the other warps have read the exchange before it is overwritten (with a quantizer: the absmax barrier)
        if constexpr (T > 32 && EPI == Epilogue::Cast) __syncthreads();
    }
    cp_async_wait_all();                                       // (the copies behind the last row were empty)
}

template <typename Tin, typename Tout, int LOG_N, Epilogue EPI, bool NORM_MOD>
static int launch_stream(const Tin* x, Tout* out, float* scales, int64_t rows, int dim, int64_t stride, float scale,
                         const __nv_bfloat16* ms, const __nv_bfloat16* mh, int64_t rows_per_mod, cudaStream_t st) {
    using Geo = StreamGeo<Tin, LOG_N, NORM_MOD>;
    const bool full = dim == Geo::N;
    auto kern = full ? hadamard_stream_kernel<Tin, Tout, LOG_N, EPI, NORM_MOD, true>
                     : hadamard_stream_kernel<Tin, Tout, LOG_N, EPI, NORM_MOD, false>;
    if (Geo::SMEM > 47 * 1024) {                               // (with the static reduction words, above the 48 KB default)
        static std::atomic<uint64_t> smem_done[2];
        if (int rc = allow_dynamic_smem((const void*)kern, Geo::SMEM, smem_done[full])) return rc;
    }
    const int64_t slots = (int64_t)gemm_num_sms() * Geo::CTAS;
    constexpr int per_cta = Geo::UNITS * Geo::RPU;
    int64_t groups = 1, group_rows = rows;
    if (NORM_MOD) {
        group_rows = rows_per_mod < rows ? rows_per_mod : rows;
        groups = (rows + group_rows - 1) / group_rows;
    }
    const int64_t need = (group_rows + per_cta - 1) / per_cta;
    int64_t blocks = slots / groups < 1 ? 1 : slots / groups;
    if (blocks > need) blocks = need;
    // A CTA stays inside one batch entry: where one turn takes all rows of an entry and there are more entries than CTAs fit
    // the device, it gets only as many units, so that more fit.  4096 x 1 x 2048 30.1 -> 15.0 us, 512 x 2 x 2048 6.8 ->
    // 5.9 us (before the streamed kernel: 16.3 and 6.1).  With fewer entries the other units help to load the modulation
    // rows (1 x 1 x 2048: 3.2 us, 3.4 with one unit).
    const int units = NORM_MOD && need == 1 && groups > slots ? (int)((group_rows + Geo::RPU - 1) / Geo::RPU) : Geo::UNITS;
    Q8K_CUDA_OK(launch_dependent(kern, (unsigned)(blocks * groups), units * Geo::UNIT, Geo::smem(units), st, 1, x, out, scales, (unsigned)rows,
                                 dim, stride, scale, ms, mh, (unsigned)group_rows, (unsigned)blocks));
    return Q8K_OK;
}

// ------------------------------------------------------------------ dispatch
template <typename Tin, typename Tout, Epilogue EPI>
static int launch_hadamard(const void* x, void* out, float* scales, int64_t rows, int dim,
                           int64_t stride, float scale, cudaStream_t st, const char* op) {
    int log_n = 3;
    while ((1 << log_n) < dim) ++log_n;
    const Tin* xi = (const Tin*)x;
    Tout* o = (Tout*)out;
    if (log_n <= 8) {
        const int log_g = log_n - 3;
        const int rows_per_cta = 128 >> log_g;
        const unsigned grid = (unsigned)((rows + rows_per_cta - 1) / rows_per_cta);
#define Q8K_HS(LG) case LG: hadamard_small_kernel<Tin, Tout, LG, EPI><<<grid, 128, 0, st>>>(xi, o, scales, rows, dim, stride, scale); break
        switch (log_g) { Q8K_HS(0); Q8K_HS(1); Q8K_HS(2); Q8K_HS(3); Q8K_HS(4); Q8K_HS(5); }
#undef Q8K_HS
    } else {
#define Q8K_HS(LN) case LN: return launch_stream<Tin, Tout, LN, EPI, false>(xi, o, scales, rows, dim, stride, scale, nullptr, nullptr, 1, st)
        switch (log_n) {
            Q8K_HS(9); Q8K_HS(10); Q8K_HS(11); Q8K_HS(12); Q8K_HS(13); Q8K_HS(14);
            default: set_error_detail("%s: dim %d exceeds 16384", op, dim); return Q8K_ERR_UNSUPPORTED;
        }
#undef Q8K_HS
    }
    Q8K_CUDA_OK(cudaGetLastError());
    return Q8K_OK;
}

// fused RMSNorm + modulation + Hadamard + quantizer (bf16 rows of 512 .. 8192 elements)
template <typename Tout>
static int launch_norm_mod_quant(const void* x, const void* mod_scale, const void* mod_shift, void* q, float* scales,
                                 int64_t rows, int dim, int64_t rows_per_mod, float scale, cudaStream_t st) {
    int log_n = 9;
    while ((1 << log_n) < dim) ++log_n;
    const __nv_bfloat16* xi = (const __nv_bfloat16*)x;
    const __nv_bfloat16* ms = (const __nv_bfloat16*)mod_scale;
    const __nv_bfloat16* mh = (const __nv_bfloat16*)mod_shift;
    Tout* o = (Tout*)q;
#define Q8K_NM(LN) case LN: return launch_stream<__nv_bfloat16, Tout, LN, Epilogue::Quant, true>(xi, o, scales, rows, dim, dim, scale, ms, mh, rows_per_mod, st)
    switch (log_n) {
        Q8K_NM(9); Q8K_NM(10); Q8K_NM(11); Q8K_NM(12); Q8K_NM(13);
        default: set_error_detail("norm_modulate_quant: dim %d not in [512, 8192]", dim); return Q8K_ERR_UNSUPPORTED;
    }
#undef Q8K_NM
}

static int check_hadamard_args(const char* op, const void* x, int x_dtype, const void* out, int64_t rows,
                               int dim, int64_t stride) {
    Q8K_REQUIRE(rows >= 0 && rows <= 0x7fffffffLL, Q8K_ERR_INVALID_ARG, "%s: rows %lld out of range", op, (long long)rows);
    Q8K_REQUIRE(dim > 0 && dim % 8 == 0, Q8K_ERR_INVALID_ARG, "%s: dim %d must be a positive multiple of 8", op, dim);
    Q8K_REQUIRE(dim <= 16384, Q8K_ERR_UNSUPPORTED, "%s: dim %d exceeds 16384", op, dim);
    if (rows == 0) return Q8K_OK;
    Q8K_REQUIRE(x && out, Q8K_ERR_INVALID_ARG, "%s: null pointer", op);
    Q8K_REQUIRE(x_dtype == Q8K_DT_BF16 || x_dtype == Q8K_DT_E4M3, Q8K_ERR_UNSUPPORTED,
                "%s: input dtype %d is not bf16 or e4m3", op, x_dtype);
    const int in_align = x_dtype == Q8K_DT_BF16 ? 16 : 8;
    Q8K_REQUIRE((reinterpret_cast<uintptr_t>(x) % in_align) == 0 && (stride * dtype_size(x_dtype)) % in_align == 0 && stride >= dim,
                Q8K_ERR_INVALID_ARG, "%s: x must be %d-byte aligned with a row stride >= dim that keeps rows aligned", op, in_align);
    Q8K_REQUIRE(aligned16(out), Q8K_ERR_INVALID_ARG, "%s: out must be 16-byte aligned", op);
    return Q8K_OK;
}

}  // namespace q8k

using namespace q8k;

extern "C" int q8k_fast_hadamard_transform(const void* x, int x_dtype, void* out, int out_dtype,
                                           int64_t rows, int dim, int64_t x_row_stride, float scale,
                                           void* stream) {
    const char* op = "fast_hadamard_transform";
    if (int rc = check_hadamard_args(op, x, x_dtype, out, rows, dim, x_row_stride)) return rc;
    if (rows == 0) return Q8K_OK;
    cudaStream_t st = (cudaStream_t)stream;
    constexpr Epilogue C = Epilogue::Cast;
    if (x_dtype == Q8K_DT_BF16 && out_dtype == Q8K_DT_BF16) return launch_hadamard<__nv_bfloat16, __nv_bfloat16, C>(x, out, nullptr, rows, dim, x_row_stride, scale, st, op);
    if (x_dtype == Q8K_DT_BF16 && out_dtype == Q8K_DT_E4M3) return launch_hadamard<__nv_bfloat16, e4m3_t, C>(x, out, nullptr, rows, dim, x_row_stride, scale, st, op);
    if (x_dtype == Q8K_DT_E4M3 && out_dtype == Q8K_DT_BF16) return launch_hadamard<e4m3_t, __nv_bfloat16, C>(x, out, nullptr, rows, dim, x_row_stride, scale, st, op);
    if (x_dtype == Q8K_DT_E4M3 && out_dtype == Q8K_DT_E4M3) return launch_hadamard<e4m3_t, e4m3_t, C>(x, out, nullptr, rows, dim, x_row_stride, scale, st, op);
    set_error_detail("%s: output dtype %d is not bf16 or e4m3", op, out_dtype);
    return Q8K_ERR_UNSUPPORTED;
}

extern "C" int q8k_dequant_hadamard(const void* x, const float* row_scales, void* out, int64_t rows, int dim, float scale,
                                    void* stream) {
    const char* op = "dequant_hadamard";
    Q8K_REQUIRE(rows >= 0 && rows <= 0x7fffffffLL, Q8K_ERR_INVALID_ARG, "%s: rows %lld out of range", op, (long long)rows);
    Q8K_REQUIRE(dim > 256 && dim <= 16384 && dim % 8 == 0, Q8K_ERR_UNSUPPORTED, "%s: dim %d not a multiple of 8 in (256, 16384]", op, dim);
    if (rows == 0) return Q8K_OK;
    Q8K_REQUIRE(x && row_scales && out && aligned16(x) && aligned16(out), Q8K_ERR_INVALID_ARG, "%s: null or misaligned pointer", op);
    float* rs = const_cast<float*>(row_scales);                // read only: the kernel's scales argument is an output otherwise
    const int8_t* xi = (const int8_t*)x;
    __nv_bfloat16* o = (__nv_bfloat16*)out;
    cudaStream_t st = (cudaStream_t)stream;
    int log_n = 9;
    while ((1 << log_n) < dim) ++log_n;
#define Q8K_DH(LN) case LN: return launch_stream<int8_t, __nv_bfloat16, LN, Epilogue::Cast, false>(xi, o, rs, rows, dim, dim, scale, nullptr, nullptr, 1, st)
    switch (log_n) { Q8K_DH(9); Q8K_DH(10); Q8K_DH(11); Q8K_DH(12); Q8K_DH(13); Q8K_DH(14); }
#undef Q8K_DH
    return Q8K_ERR_UNSUPPORTED;
}

extern "C" int q8k_hadamard_quant(const void* x, int x_dtype, void* q, int q_dtype, float* scales,
                                  int64_t rows, int dim, int64_t x_row_stride, float scale, void* stream) {
    const char* op = "hadamard_quant";
    if (int rc = check_hadamard_args(op, x, x_dtype, q, rows, dim, x_row_stride)) return rc;
    if (rows == 0) return Q8K_OK;
    Q8K_REQUIRE(scales != nullptr, Q8K_ERR_INVALID_ARG, "%s: null scales pointer", op);
    cudaStream_t st = (cudaStream_t)stream;
    constexpr Epilogue Q = Epilogue::Quant;
    if (x_dtype == Q8K_DT_BF16 && q_dtype == Q8K_DT_I8)   return launch_hadamard<__nv_bfloat16, int8_t, Q>(x, q, scales, rows, dim, x_row_stride, scale, st, op);
    if (x_dtype == Q8K_DT_BF16 && q_dtype == Q8K_DT_E4M3) return launch_hadamard<__nv_bfloat16, e4m3_t, Q>(x, q, scales, rows, dim, x_row_stride, scale, st, op);
    if (x_dtype == Q8K_DT_E4M3 && q_dtype == Q8K_DT_I8)   return launch_hadamard<e4m3_t, int8_t, Q>(x, q, scales, rows, dim, x_row_stride, scale, st, op);
    if (x_dtype == Q8K_DT_E4M3 && q_dtype == Q8K_DT_E4M3) return launch_hadamard<e4m3_t, e4m3_t, Q>(x, q, scales, rows, dim, x_row_stride, scale, st, op);
    set_error_detail("%s: quantised dtype %d is not int8 or e4m3", op, q_dtype);
    return Q8K_ERR_UNSUPPORTED;
}

extern "C" int q8k_norm_modulate_quant(const void* x, const void* mod_scale, const void* mod_shift, void* q, int q_dtype,
                                       float* scales, int64_t rows, int dim, int64_t rows_per_mod, float scale,
                                       void* stream) {
    const char* op = "norm_modulate_quant";
    if (int rc = check_hadamard_args(op, x, Q8K_DT_BF16, q, rows, dim, dim)) return rc;
    if (rows == 0) return Q8K_OK;
    Q8K_REQUIRE(dim >= 257 && dim % 16 == 0, Q8K_ERR_UNSUPPORTED, "%s: dim %d must be a multiple of 16 above 256", op, dim);
    Q8K_REQUIRE(mod_scale && mod_shift && scales, Q8K_ERR_INVALID_ARG, "%s: null pointer", op);
    Q8K_REQUIRE(aligned16(mod_scale) && aligned16(mod_shift), Q8K_ERR_INVALID_ARG, "%s: modulation rows must be 16-byte aligned", op);
    Q8K_REQUIRE(rows_per_mod >= 1, Q8K_ERR_INVALID_ARG, "%s: rows_per_mod must be >= 1", op);
    cudaStream_t st = (cudaStream_t)stream;
    if (q_dtype == Q8K_DT_I8) return launch_norm_mod_quant<int8_t>(x, mod_scale, mod_shift, q, scales, rows, dim, rows_per_mod, scale, st);
    if (q_dtype == Q8K_DT_E4M3) return launch_norm_mod_quant<e4m3_t>(x, mod_scale, mod_shift, q, scales, rows, dim, rows_per_mod, scale, st);
    set_error_detail("%s: quantised dtype %d is not int8 or e4m3", op, q_dtype);
    return Q8K_ERR_UNSUPPORTED;
}
