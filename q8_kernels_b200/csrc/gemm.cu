// 8-bit GEMM with fused dequant + bias + tanh-GELU epilogue:  C[b] = act((A[b] . B[b]^T) * (sa[m] * sb[n]) + bias[n]).
//
//   A [bs_a, M, K], B [bs_b, N, K]  int8 (kind::i8, int32 accumulate) or
//   e4m3 (kind::f8f6f4, fp32 accumulate), both K-contiguous.
//
// Epilogue arithmetic follows csrc/gemm/q8_matmul_bias.cu:29-33,315-371 of the
// reference: float(acc) * (sa*sb) + bias, optional tanh-GELU, then bf16 (RNE)
// or e4m3 (saturating).
//
// This file checks the arguments and chooses between the two kernels: 256 x 256 tiles on CTA pairs (gemm_pair.cu) and
// 128 x bn tiles, for int8 with K split over clusters (gemm_split.cu).

#include "gemm_common.cuh"

namespace q8k {

// ------------------------------------------------------------------ host side
static int g_num_sms = 0;

int gemm_num_sms() {
    if (g_num_sms == 0) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess) return 148;
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) return 148;
        g_num_sms = n;
    }
    return g_num_sms;
}

// Tile width and K split of the split kernel, and whether the pair kernel is the better one.  The times (us) come from
// CUDA-graph timings with weights streamed from HBM, M = 1 .. 6144, N = 1024 .. 10240, K = 1024 .. 8192, and reproduce
// those to about 10 %.  (Fitted without dependent launch, which hides about 2 us of either kernel's set-up.)
//   split: 4.0 for launch, set-up and drain; per 128-byte K slab the larger of 0.165 (one slab through the issuing
//          threads) and its bytes at 140 GB/s (one SM's L2 port; 1.7 x the bytes where K is not a multiple of 128 and
//          rows straddle cache lines), times the CTAs of the busiest SM, and 1.5 for every CTA beyond the first there;
//          3.85e-5 bn^2 for the epilogue; the exchange of a K split; 0.06 per MB of weights
//   pair:  6.5 + 0.31 per slab and wave of 74 tiles.  This is whole waves: where narrow_plan cuts the last one, the pair kernel
//          takes up to a sixth less.
// Examples, int8 (pair or 128 x 128 tiles before -> now): M = 128, N = K = 2048 9.5 -> 5.2 (bn 32);  M = 77, N = 10240,
// K = 4096 15.4 -> 11.6 (bn 80);  M = 128, N = 2048, K = 8192 23.1 -> 9.0 (bn 64, sk 4);  M = 1024, N = 2048, K = 8192
// 26.2 -> 18.0 (bn 128).  At N = K = 2048 the line to the pair kernel lies between M = 1024 (12.2 -> 8.4) and M = 2048
// (12.6 against 14.9).
// Just above a full wave the whole-wave model still sends to the split kernel what narrow pair tiles do faster (7 % of the sizes
// that have such tiles, M = 129 .. 12289; split against pair): fp8 M = 2433, N = 2048, K = 4096 31.5 against 24.2;  M = 5000,
// N = 1024, K = 4096 26.9 against 20.1;  M = 10000, N = 512, K = 8192 51.3 against 38.5;  M = 1200, N = K = 4096 21.9 against
// 20.2;  but M = 4640, N = 1024, K = 8192 33.5 against 36.4 and M = 300, N = 10240, K = 4096 21.1 against 22.7.
// Half of a pair tile is padding where M or N is at most 128, so there the split kernel is the rule; but one tile per CTA
// pays its set-up for every tile, and from three rounds of pair tiles on the persistent pair kernel is faster all the same
// (int8, pair against split): N = 128, K = 1024 M = 24576 11.5 against 11.4, M = 49152 15.7 against 20.9, M = 196608 45.3
// against 60.9;  N = 64, K = 512, M = 98304 17.4 against 18.9;  N = 16 28.2 against 23.8 (K = 1024, M = 98304: split).
// With weights of their own per batch entry: 32 x (M = 100, N = 4096, K = 1024) 33.5 against 37.5, 32 x (M = 128, N = 2048,
// K = 128) 14.4 against 10.8 (split).  M <= 128 rows on shared weights: split (N = 65536, K = 1024, M = 77 22.0 against 18.5).
// Only int8 splits K: its partial sums are exact.  fp32 partials would round in another order than one accumulator,
// and an fp8 row would then have other bits in a call with other M or N (it has the same in every call, and stacked
// weights give the bits of the separate ones).
struct SplitChoice { bool use; int bn, sk; };
static SplitChoice choose_split(bool int8, int M, int N, int K, int batch, int sms) {
    const int iters = (K + kGemmBK - 1) / kGemmBK;
    const double m_tiles = (double)((M + kGemmBM - 1) / kGemmBM) * batch;
    const int a_rows = split_a_rows(M);
    SplitChoice c = {true, 128, 1};
    double best = 1e30;
    for (int sk = 1; sk <= (int8 ? 4 : 1); sk *= 2) {
        if (iters < 2 * sk && sk > 1) break;
        for (int bn = 32; bn <= 256; bn += sk == 4 ? 32 : 16) {
            if (bn > 32 && bn - 16 >= N) break;
            const double ctas = m_tiles * ((N + bn - 1) / bn) * sk;
            const double per_sm = ctas <= sms ? 1.0 : (double)(int64_t)((ctas + sms - 1) / sms);
            const double bytes = (a_rows + bn) * 128.0 / 140e3 * (K % 128 != 0 ? 1.7 : 1.0);
            double t = 4.0 + 1.5 * (per_sm - 1.0)
                     + per_sm * ((iters + sk - 1) / sk * (bytes > 0.165 ? bytes : 0.165) + 3.85e-5 * bn * bn);
            if (sk > 1) t += 1.2 + (sk == 2 ? 0.0145 : 0.028) * bn;
            if (t < best) { best = t; c.bn = bn; c.sk = sk; }
        }
    }
    best += 0.06e-6 * N * K;
    const double tiles = (double)((M + 255) / 256) * ((N + 255) / 256) * batch;
    const double waves = (double)(int64_t)((tiles + sms / 2 - 1) / (sms / 2));
    if (M > kGemmBM && N > 128) c.use = best < 0.95 * (6.5 + 0.31 * iters * waves);
    else c.use = waves < 3 || !((N >= 64 && N <= 128) || (batch > 1 && M >= 64 && iters >= 8));
    return c;
}

// On shared weights a batch is more rows of one product.  Returns the batch that is left.
static int fold_batch(int& bs_a, int bs_b, int& M) {
    if (bs_b == 1) {
        M *= bs_a;
        bs_a = 1;
    }
    return bs_a > bs_b ? bs_a : bs_b;
}

static int gemm_8bit(bool int8, const void* a, const void* b, const float* bias, const float* a_scales,
                     const float* b_scales, void* out, int out_dtype, int bs_a, int bs_b, int M, int N, int K,
                     int fuse_gelu, int* dev_status, void* stream, const void* resid = nullptr,
                     const void* gate = nullptr, int64_t rows_per_gate = 1) {
    const char* op = int8 ? "q8_mm" : "fp8_mm";
    Q8K_REQUIRE(a && b && a_scales && b_scales && out, Q8K_ERR_INVALID_ARG, "%s: null pointer", op);
    Q8K_REQUIRE(bs_a >= 1 && bs_b >= 1 && (bs_a == bs_b || bs_a == 1 || bs_b == 1), Q8K_ERR_INVALID_ARG,
                "%s: batch mismatch (%d vs %d)", op, bs_a, bs_b);
    Q8K_REQUIRE(M >= 0 && N > 0 && K > 0, Q8K_ERR_INVALID_ARG, "%s: bad shape M=%d N=%d K=%d", op, M, N, K);
    Q8K_REQUIRE(N % 16 == 0 && K % 16 == 0, Q8K_ERR_INVALID_ARG, "%s: N=%d and K=%d must be multiples of 16", op, N, K);
    Q8K_REQUIRE(aligned16(a) && aligned16(b) && aligned16(out), Q8K_ERR_INVALID_ARG,
                "%s: a, b and out must be 16-byte aligned", op);
    Q8K_REQUIRE(out_dtype == Q8K_DT_BF16 || out_dtype == Q8K_DT_E4M3, Q8K_ERR_UNSUPPORTED,
                "%s: output dtype %d is not bf16 or e4m3", op, out_dtype);
    Q8K_REQUIRE((int64_t)bs_a * M <= 0x7fffffffLL && (int64_t)bs_b * N <= 0x7fffffffLL, Q8K_ERR_TOO_LARGE,
                "%s: batch * rows exceeds 2^31", op);
    if (M == 0) return Q8K_OK;
    const int batch = fold_batch(bs_a, bs_b, M);

    GemmParams p;
    p.a_scales = a_scales;
    p.b_scales = b_scales;
    p.bias = bias;
    p.out = out;
    p.status = dev_status;
    p.resid = reinterpret_cast<const __nv_bfloat16*>(resid);
    p.gate = reinterpret_cast<const __nv_bfloat16*>(gate);
    p.rows_per_gate = rows_per_gate > 0 ? rows_per_gate : 1;
    p.M = M; p.N = N; p.K = K;
    p.batch_a = bs_a > 1; p.batch_b = bs_b > 1;
    cudaStream_t st = (cudaStream_t)stream;
    const bool gelu = fuse_gelu != 0;
    const bool e4m3 = out_dtype == Q8K_DT_E4M3;

    const bool fuse_resid = resid != nullptr;
    if (fuse_resid) {
        Q8K_REQUIRE(!gelu && !e4m3, Q8K_ERR_UNSUPPORTED, "%s: the gate/residual tail needs a bf16 output without GELU", op);
        Q8K_REQUIRE(aligned16(resid) && aligned16(gate), Q8K_ERR_INVALID_ARG, "%s: gate and residual must be 16-byte aligned", op);
    }
    const SplitChoice choice = choose_split(int8, M, N, K, batch, gemm_num_sms());
    if (!choice.use) {
        const int rc = launch_gemm_pair(int8, gelu, e4m3, fuse_resid, a, b, p, bs_a, bs_b, st);
        if (rc != Q8K_ERR_UNSUPPORTED) return rc;              // (the device cannot co-schedule the pairs)
    }
    return launch_gemm_split(int8, gelu, e4m3, fuse_resid, a, b, p, bs_a, bs_b, choice.bn, choice.sk, st);
}

}  // namespace q8k

extern "C" int q8k_mm_plan(int int8, int bs_a, int bs_b, int M, int N, int K, int plan[3]) {
    using q8k::set_error_detail;
    Q8K_REQUIRE(plan != nullptr && bs_a >= 1 && bs_b >= 1 && M > 0 && N > 0 && K > 0 && (int64_t)bs_a * M <= 0x7fffffffLL,
                Q8K_ERR_INVALID_ARG, "mm_plan: null plan or bad shape");
    const int batch = q8k::fold_batch(bs_a, bs_b, M);
    const q8k::SplitChoice c = q8k::choose_split(int8 != 0, M, N, K, batch, q8k::gemm_num_sms());
    plan[0] = c.use ? 0 : 1;
    plan[1] = c.use ? c.bn : 256;
    plan[2] = c.use ? c.sk : 1;
    return Q8K_OK;
}

extern "C" int q8k_mm_last_round_columns(int bs_a, int bs_b, int M, int N, int K, int resid, int* columns) {
    using q8k::set_error_detail;
    Q8K_REQUIRE(columns != nullptr && bs_a >= 1 && bs_b >= 1 && M > 0 && N > 0 && K > 0 && (int64_t)bs_a * M <= 0x7fffffffLL,
                Q8K_ERR_INVALID_ARG, "mm_last_round_columns: null result or bad shape");
    const int batch = q8k::fold_batch(bs_a, bs_b, M);
    *columns = q8k::pair_last_round_columns(M, N, K, batch, resid != 0);
    return Q8K_OK;
}

extern "C" int q8k_q8_mm(const void* a, const void* b, const float* bias, const float* a_scales,
                         const float* b_scales, void* out, int out_dtype, int bs_a, int bs_b, int M, int N,
                         int K, int fuse_gelu, int* dev_status, void* stream) {
    return q8k::gemm_8bit(true, a, b, bias, a_scales, b_scales, out, out_dtype, bs_a, bs_b, M, N, K, fuse_gelu,
                          dev_status, stream);
}

extern "C" int q8k_mm_gate_residual(int int8, const void* a, const void* b, const float* bias, const float* a_scales,
                                    const float* b_scales, const void* gate, const void* resid, int64_t rows_per_gate,
                                    void* out, int bs_a, int bs_b, int M, int N, int K, int* dev_status, void* stream) {
    if (resid == nullptr) {
        q8k::set_error_detail("mm_gate_residual: null residual");
        return Q8K_ERR_INVALID_ARG;
    }
    return q8k::gemm_8bit(int8 != 0, a, b, bias, a_scales, b_scales, out, Q8K_DT_BF16, bs_a, bs_b, M, N, K, 0, dev_status,
                          stream, resid, gate, rows_per_gate);
}

extern "C" int q8k_fp8_mm(const void* a, const void* b, const float* bias, const float* a_scales,
                          const float* b_scales, void* out, int out_dtype, int bs_a, int bs_b, int M, int N,
                          int K, int fuse_gelu, int* dev_status, void* stream) {
    return q8k::gemm_8bit(false, a, b, bias, a_scales, b_scales, out, out_dtype, bs_a, bs_b, M, N, K, fuse_gelu,
                          dev_status, stream);
}
