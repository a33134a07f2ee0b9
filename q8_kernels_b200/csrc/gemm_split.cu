// 8-bit GEMM for problems that 256 x 256 pair tiles cannot spread over the device: 128 x bn output tiles,
// for int8 optionally with the K range split over the CTAs of a cluster.
//
//   C[b] = act((A[b] . B[b]^T) * (sa[m] * sb[n]) + bias[n])      (operands and epilogue as in gemm_pair.cu)
//
// Why: a 128-token projection (M = 128, N = K = 2048) has 16 tiles of 128 x 128; on 16 CTAs each streams 512 KB
// through one SM's L2 port (about 91 GB/s of TMA traffic), and the rest of the device idles.  Here the tile width
// is chosen so that the tiles fill the device once, and where that is not enough a cluster of sk CTAs owns one
// tile: CTA r accumulates its share of K in TMEM, then the partial tiles are exchanged through distributed shared
// memory (every CTA receives all sk partials of its bn / sk columns), summed and finished by the CTA that owns the
// columns.  The sum of the int32 partials is exact.  fp8 keeps one fp32 accumulator per element (sk = 1), so that its
// bits do not depend on the split, i.e. on the other rows and columns of the call.
//
// One tile per CTA.  Roles (10 warps):
//   warp 0     TMA producer (plain loads, no multicast; of A only the rows that exist)
//   warp 1     TMEM allocation; one thread issues tcgen05.mma (M = 128, N = bn, K = 32)
//   warps 2-9  epilogue; column scales and bias are fetched while the main loop runs
// All waits are bounded.  A CTA that finds the status word set skips its loads, MMAs and stores but keeps to the
// cluster barriers, so the CTAs of a cluster need not agree.
//
// Bound by the latency of one short main loop: launch, set-up and drain take about 4 us, a 128-byte K slab 0.165 us.
// Measured (CUDA graph, weights from HBM; the 128 x 128-tile kernel or the pair kernel before): int8 M = 128, N = K = 2048
// 9.5 -> 5.2 us (bn 32), M = 77, N = 10240, K = 4096 15.4 -> 11.6 us (42 MB of weights: 0.55 of the copy rate), M = 128,
// N = 2048, K = 8192 23.1 -> 9.0 us (bn 64, sk 4), M = 512 26.0 -> 13.7 us (bn 128, sk 2).  Tried: independent accumulators for
// the four MMAs of a slab (no difference), clusters of eight (the exchange costs 5 us).  Where the line to the pair
// kernel lies: choose_split in gemm.cu.

#include "gemm_common.cuh"

namespace q8k {

constexpr int kSplitMaxStages = 8;
constexpr int kSplitMaxBN = 256;
constexpr int kSplitABytes = kGemmBM * kGemmBK;
struct SplitSmem {                           // behind the operand ring, whose length is chosen per launch
    static constexpr int kNumBars = 2 * kSplitMaxStages + 1;
    static constexpr int kTmemPtrOffset = kNumBars * 8;
    static constexpr int kAbortOffset = kTmemPtrOffset + 4;
    static constexpr int kColScaleOffset = (kAbortOffset + 4 + 15) & ~15;
    static constexpr int kBiasOffset = kColScaleOffset + kSplitMaxBN * 4;
    static constexpr int kTotal = kBiasOffset + kSplitMaxBN * 4;
};
struct SplitParams {
    GemmParams g;
    uint32_t idesc;
    int bn, sk;                              // tile columns (a multiple of 16, with sk = 4 of 32); CTAs per tile (fp8: 1)
    int stages;
    int stage_bytes;                         // 16 KB of A and bn rows of B
    int load_bytes;                          // what one stage's TMA boxes bring
};

__device__ __forceinline__ void st_cluster_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// NC (a multiple of 8) adjacent columns of one row: scale, bias, GELU, cast, gate / residual, 16-byte (e4m3: 8-byte)
// stores.  n is the first column; columns from p.N on are left out (N % 16 == 0: eight are all in or all out).
template <bool INT8, bool GELU, bool OUT_E4M3, bool RESID, int NC>
__device__ __forceinline__ void finish_row(const GemmParams& p, const uint32_t (&acc)[NC], float sa, int64_t out_row,
                                           int64_t gate_row, int n, const float* col_scale, const float* bias) {
#pragma unroll
    for (int g = 0; g < NC / 8; ++g) {
        if (n + g * 8 < p.N) {
            float2 y[4];
#pragma unroll
            for (int j = 0; j < 4; ++j)
                y[j] = epilogue_pair<INT8, GELU>(acc[g * 8 + 2 * j], acc[g * 8 + 2 * j + 1], make_float2(sa, sa),
                                                 col_scale + g * 8 + 2 * j, bias + g * 8 + 2 * j);
            const int64_t o = out_row + n + g * 8;
            if constexpr (OUT_E4M3) {
                uint2 w;
                w.x = (uint32_t)float2_to_e4m3x2_sat(y[0].x, y[0].y) | ((uint32_t)float2_to_e4m3x2_sat(y[1].x, y[1].y) << 16);
                w.y = (uint32_t)float2_to_e4m3x2_sat(y[2].x, y[2].y) | ((uint32_t)float2_to_e4m3x2_sat(y[3].x, y[3].y) << 16);
                *reinterpret_cast<uint2*>(reinterpret_cast<uint8_t*>(p.out) + o) = w;
            } else {
                uint32_t w[4];
                uint4 rs = make_uint4(0, 0, 0, 0), gt = make_uint4(0, 0, 0, 0);
                if constexpr (RESID) {
                    rs = *reinterpret_cast<const uint4*>(p.resid + o);
                    if (p.gate != nullptr) gt = *reinterpret_cast<const uint4*>(p.gate + gate_row + n + g * 8);
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    __nv_bfloat162 b2 = __floats2bfloat162_rn(y[j].x, y[j].y);
                    if constexpr (RESID) {                      // the roundings of the separate ops: see gemm_pair.cu
                        const uint32_t gw = j == 0 ? gt.x : (j == 1 ? gt.y : (j == 2 ? gt.z : gt.w));
                        const uint32_t rw = j == 0 ? rs.x : (j == 1 ? rs.y : (j == 2 ? rs.z : rs.w));
                        if (p.gate != nullptr) b2 = __hmul2_rn(*reinterpret_cast<const __nv_bfloat162*>(&gw), b2);
                        b2 = __hadd2_rn(b2, *reinterpret_cast<const __nv_bfloat162*>(&rw));
                    }
                    w[j] = *reinterpret_cast<uint32_t*>(&b2);
                }
                *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.out) + o) = make_uint4(w[0], w[1], w[2], w[3]);
            }
        }
    }
}

template <int COLS> __device__ __forceinline__ void split_tmem(bool alloc, uint32_t arg) {
    if (alloc) ptx::tmem_alloc<COLS>(arg);
    else ptx::tmem_dealloc<COLS>(arg);
}
__device__ __forceinline__ void split_tmem_any(int bn, bool alloc, uint32_t arg) {   // whole warp, convergent
    if (bn <= 32) split_tmem<32>(alloc, arg);
    else if (bn <= 64) split_tmem<64>(alloc, arg);
    else if (bn <= 128) split_tmem<128>(alloc, arg);
    else split_tmem<256>(alloc, arg);
}

template <bool INT8, bool GELU, bool OUT_E4M3, bool RESID>
__global__ void __launch_bounds__(kGemmThreads, 2)
gemm_8bit_split_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                       const __grid_constant__ SplitParams sp) {
    using L = SplitSmem;
    const GemmParams& p = sp.g;
    const int bn = sp.bn, sk = INT8 ? sp.sk : 1, stages = sp.stages;

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t smem_base = ptx::smem_u32(smem);            // the same offset in every CTA of the cluster
    uint8_t* tail = smem + stages * sp.stage_bytes;
    const uint32_t bar_base = ptx::smem_u32(tail);
    auto full_bar = [&](int s) { return bar_base + 8u * s; };
    auto empty_bar = [&](int s) { return bar_base + 8u * (kSplitMaxStages + s); };
    const uint32_t acc_bar = bar_base + 8u * (2 * kSplitMaxStages);
    volatile uint32_t* tmem_ptr_smem = reinterpret_cast<volatile uint32_t*>(tail + L::kTmemPtrOffset);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tail + L::kAbortOffset);
    float* col_scale_smem = reinterpret_cast<float*>(tail + L::kColScaleOffset);
    float* bias_smem = reinterpret_cast<float*>(tail + L::kBiasOffset);
    __shared__ int prior_failure;

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int rank = sk > 1 ? (int)ptx::cluster_ctarank() : 0;
    const int tile = blockIdx.x / sk;
    const int n_blk = tile % p.n_tiles;
    const int m_blk = (tile / p.n_tiles) % p.m_tiles;
    const int batch = tile / (p.n_tiles * p.m_tiles);
    const int k_iters = (p.K + kGemmBK - 1) / kGemmBK;
    const int k_begin = k_iters * rank / sk;                   // k_iters >= sk: nobody's share is empty
    const int k_count = k_iters * (rank + 1) / sk - k_begin;
    const int n0 = n_blk * bn;

    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
            ptx::mbar_init(full_bar(s), 1);
            ptx::mbar_init(empty_bar(s), 1);
        }
        ptx::mbar_init(acc_bar, 1);
        *abort_flag = 0;
        ptx::fence_barrier_init();
        ptx::fence_proxy_async_smem();
        ptx::prefetch_tensormap(&tmap_a);
        ptx::prefetch_tensormap(&tmap_b);
    }
    if (warp == 1) {
        split_tmem_any(bn, true, ptx::smem_u32(const_cast<uint32_t*>(tmem_ptr_smem)));
        ptx::tmem_relinquish_alloc_permit();
    }
    pdl_wait();                                                // everything above overlaps the kernel before
    if (threadIdx.x == 0) prior_failure = p.status != nullptr ? *reinterpret_cast<volatile int*>(p.status) : 0;
    ptx::tcgen05_fence_before_sync();
    __syncthreads();
    ptx::tcgen05_fence_after_sync();
    pdl_release();                                             // this CTA holds its TMEM: the next kernel may move in behind it
    const uint32_t tmem_base = *tmem_ptr_smem;
    bool ok = prior_failure == 0;

    // epilogue coordinates (warps 2..9): warp w may touch TMEM lanes [32 * (w % 4), +32); warps 2-5 take the even
    // groups of 16 columns, warps 6-9 the odd ones
    const int quarter = warp & 3;
    const int half = (warp - 2) >> 2;
    const int row_in = quarter * 32 + lane;

    if (warp == 0) {
        if (ok && ptx::elect_one()) {
            const int a_row = (p.batch_a ? batch * p.M : 0) + m_blk * kGemmBM;
            const int b_row = (p.batch_b ? batch * p.N : 0) + n0;
            int s = 0;
            uint32_t ph = 1;                                   // empty_bar phase to wait for: the first round passes
            for (int i = 0; i < k_count; ++i) {
                if (!ptx::mbar_wait(empty_bar(s), ph, abort_flag)) { ok = false; break; }
                ptx::mbar_arrive_expect_tx(full_bar(s), (uint32_t)sp.load_bytes);
                const uint32_t a_dst = smem_base + s * sp.stage_bytes;
                ptx::tma_load_2d(a_dst, &tmap_a, full_bar(s), (k_begin + i) * kGemmBK, a_row);
                ptx::tma_load_2d(a_dst + kSplitABytes, &tmap_b, full_bar(s), (k_begin + i) * kGemmBK, b_row);
                if (++s == stages) { s = 0; ph ^= 1u; }
            }
            if (!ok && p.status != nullptr) atomicExch(p.status, Q8K_STATUS_TIMEOUT | (1 << 8));
        }
        __syncwarp();
    } else if (warp == 1) {
        if (ok && ptx::elect_one()) {
            int s = 0;
            uint32_t ph = 0;
            for (int i = 0; i < k_count; ++i) {
                if (!ptx::mbar_wait(full_bar(s), ph, abort_flag)) { ok = false; break; }
                ptx::tcgen05_fence_after_sync();
                const uint32_t a_addr = smem_base + s * sp.stage_bytes;
                const uint64_t a_desc = ptx::make_kmajor_desc(a_addr, 128);
                const uint64_t b_desc = ptx::make_kmajor_desc(a_addr + kSplitABytes, 128);
#pragma unroll
                for (int k = 0; k < kGemmBK / 32; ++k) {
                    const uint32_t accumulate = (i > 0 || k > 0) ? 1u : 0u;
                    if constexpr (INT8) ptx::mma_i8(tmem_base, a_desc + 2 * k, b_desc + 2 * k, sp.idesc, accumulate);
                    else ptx::mma_f8f6f4(tmem_base, a_desc + 2 * k, b_desc + 2 * k, sp.idesc, accumulate);
                }
                ptx::tcgen05_commit(empty_bar(s));
                if (++s == stages) { s = 0; ph ^= 1u; }
            }
            if (ok) ptx::tcgen05_commit(acc_bar);
            else if (p.status != nullptr) atomicExch(p.status, Q8K_STATUS_TIMEOUT | (2 << 8));
        }
        __syncwarp();
    } else if (ok) {
        for (int c = threadIdx.x - 64; c < bn; c += kGemmEpilogueThreads) {
            const int n = n0 + c;
            const bool in = n < p.N;
            col_scale_smem[c] = in ? p.b_scales[(p.batch_b ? (int64_t)batch * p.N : 0) + n] : 0.f;
            bias_smem[c] = (in && p.bias != nullptr) ? p.bias[n] : 0.f;
        }
        asm volatile("bar.sync 1, 256;" ::: "memory");
    }
    const int row = m_blk * kGemmBM + (sk > 1 ? (int)(threadIdx.x - 64) & 127 : row_in);
    const bool row_ok = warp >= 2 && row < p.M;
    const float sa = row_ok ? p.a_scales[(p.batch_a ? (int64_t)batch * p.M : 0) + row] : 0.f;
    if (warp >= 2 && ok) {
        ok = ptx::mbar_wait(acc_bar, 0, abort_flag);
        ok = __all_sync(0xffffffffu, ok);                      // keep the warp convergent for tcgen05.ld
        ptx::tcgen05_fence_after_sync();
        if (!ok && p.status != nullptr && threadIdx.x == 64) atomicExch(p.status, Q8K_STATUS_TIMEOUT | (3 << 8));
    }

    const int64_t out_row = ((int64_t)batch * p.M + row) * p.N;
    const int64_t gate_row = RESID ? (((int64_t)batch * p.M + row) / p.rows_per_gate) * p.N : 0;
    const uint32_t t_row = tmem_base + ((uint32_t)(quarter * 32) << 16);

    if (sk == 1) {
        if (warp >= 2 && ok) {
#pragma unroll 1
            for (int cl = half * 16; cl < bn; cl += 32) {
                uint32_t r[16];
                ptx::tmem_ld_32x32b_x16(t_row + cl, r);
                ptx::tmem_wait_ld();
                if (row_ok)
                    finish_row<INT8, GELU, OUT_E4M3, RESID, 16>(p, r, sa, out_row, gate_row, n0 + cl, col_scale_smem + cl, bias_smem + cl);
                __syncwarp();
            }
        }
    } else {
        const int cpc = bn / sk;                               // columns that each CTA finishes: a multiple of 8
        // every CTA's MMAs have retired: its ring may be written by the others
        ptx::cluster_sync_all();
        if (warp >= 2 && ok) {
            // partial tile -> the owners of the columns: [rank][4-column group][row], 16 bytes per row
#pragma unroll 1
            for (int cl = half * 16; cl < bn; cl += 32) {
                uint32_t r[16];
                ptx::tmem_ld_32x32b_x16(t_row + cl, r);
                ptx::tmem_wait_ld();
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int col = cl + q * 4;
                    const int owner = col / cpc;
                    const uint32_t dst = smem_base + (uint32_t)(((rank * cpc + col - owner * cpc) / 4 * kGemmBM + row_in) * 16);
                    st_cluster_v4(ptx::mapa_shared(dst, (uint32_t)owner), r[4 * q], r[4 * q + 1], r[4 * q + 2], r[4 * q + 3]);
                }
            }
        }
        __syncwarp();
        ptx::cluster_sync_all();
        if (warp >= 2 && ok && row_ok) {
            const int hh = (int)(threadIdx.x - 64) >> 7;       // two threads per row: groups of eight columns in turn
            const int rl = (int)(threadIdx.x - 64) & 127;
#pragma unroll 1
            for (int c8 = hh * 8; c8 < cpc; c8 += 16) {
                uint32_t acc[8];
                for (int r = 0; r < sk; ++r) {
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const uint4 w = *reinterpret_cast<const uint4*>(smem + ((((r * cpc + c8) >> 2) + q) * kGemmBM + rl) * 16);
                        const uint32_t v[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            if (r == 0) acc[4 * q + j] = v[j];
                            else acc[4 * q + j] += v[j];
                        }
                    }
                }
                const int cl = rank * cpc + c8;
                finish_row<INT8, GELU, OUT_E4M3, RESID, 8>(p, acc, sa, out_row, gate_row, n0 + cl, col_scale_smem + cl, bias_smem + cl);
            }
        }
    }

    if (threadIdx.x == 0 && *abort_flag != 0) {
        // a wait was abandoned: give copies still in flight time to land before the CTA gives up its shared memory
        const unsigned long long t0 = ptx::globaltimer_ns();
        while (ptx::globaltimer_ns() - t0 < 50000ull) {}
    }
    ptx::tcgen05_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        ptx::tcgen05_fence_after_sync();
        split_tmem_any(bn, false, tmem_base);
    }
}

// ------------------------------------------------------------------ host side
template <bool INT8, bool GELU, bool OUT_E4M3, bool RESID>
static int launch_split(const CUtensorMap& ta, const CUtensorMap& tb, const SplitParams& sp, int smem, cudaStream_t st) {
    auto kern = gemm_8bit_split_kernel<INT8, GELU, OUT_E4M3, RESID>;
    static std::atomic<uint64_t> smem_done{0};
    if (int rc = allow_dynamic_smem((const void*)kern, 226 * 1024, smem_done)) return rc;
    Q8K_CUDA_OK(launch_dependent(kern, (unsigned)sp.g.total_tiles * (unsigned)sp.sk, kGemmThreads, smem, st, sp.sk, ta, tb, sp));
    return Q8K_OK;
}

int launch_gemm_split(bool int8, bool gelu, bool out_e4m3, bool resid, const void* a, const void* b, const GemmParams& p,
                      int bs_a, int bs_b, int bn, int sk, cudaStream_t st) {
    const char* op = int8 ? "q8_mm" : "fp8_mm";
    const int a_rows = split_a_rows(p.M);
    CUtensorMap ta, tb;
    {
        const uint64_t dims[2] = {(uint64_t)p.K, (uint64_t)bs_a * (uint64_t)p.M};
        const uint64_t strides[1] = {(uint64_t)p.K};
        const uint32_t box[2] = {(uint32_t)kGemmBK, (uint32_t)a_rows};
        if (int rc = make_byte_tensor_map(&ta, a, 2, dims, strides, box, 128, op)) return rc;
    }
    {
        const uint64_t dims[2] = {(uint64_t)p.K, (uint64_t)bs_b * (uint64_t)p.N};
        const uint64_t strides[1] = {(uint64_t)p.K};
        const uint32_t box[2] = {(uint32_t)kGemmBK, (uint32_t)bn};
        if (int rc = make_byte_tensor_map(&tb, b, 2, dims, strides, box, 128, op)) return rc;
    }
    SplitParams sp;
    sp.g = p;
    sp.idesc = int8 ? ptx::make_idesc_s8(kGemmBM, bn) : ptx::make_idesc_e4m3(kGemmBM, bn);
    sp.bn = bn;
    sp.sk = sk;
    sp.stage_bytes = kSplitABytes + bn * kGemmBK;
    sp.load_bytes = (a_rows + bn) * kGemmBK;
    const int64_t m_tiles = (p.M + kGemmBM - 1) / kGemmBM, n_tiles = (p.N + bn - 1) / bn;
    const int64_t total = m_tiles * n_tiles * (bs_a > bs_b ? bs_a : bs_b);
    Q8K_REQUIRE(total * sk <= 0x7fffffffLL, Q8K_ERR_TOO_LARGE, "%s: too many tiles", op);
    sp.g.m_tiles = (int)m_tiles;
    sp.g.n_tiles = (int)n_tiles;
    sp.g.total_tiles = (int)total;
    // A grid that fits the device once gets a deep ring; otherwise two CTAs share an SM.  No more stages than slabs (one for
    // K <= 128), and with sk > 1 room for the exchange of 128 x bn words.
    const int budget = total * sk <= gemm_num_sms() ? 208 * 1024 : 104 * 1024;
    int stages = budget / sp.stage_bytes;
    const int per_cta = ((p.K + kGemmBK - 1) / kGemmBK + sk - 1) / sk;
    if (stages > per_cta) stages = per_cta;
    const int least = sk > 1 ? (kGemmBM * bn * 4 + sp.stage_bytes - 1) / sp.stage_bytes : 1;
    if (stages < least) stages = least;
    if (stages > kSplitMaxStages) stages = kSplitMaxStages;
    sp.stages = stages;
    const int smem = stages * sp.stage_bytes + SplitSmem::kTotal + 1024;   // slack to align the base to 1024 B
#define Q8K_SPLIT(I8)                                                                     \
    do {                                                                                  \
        if (resid) return launch_split<I8, false, false, true>(ta, tb, sp, smem, st);     \
        if (gelu) return out_e4m3 ? launch_split<I8, true, true, false>(ta, tb, sp, smem, st)    \
                                  : launch_split<I8, true, false, false>(ta, tb, sp, smem, st);  \
        return out_e4m3 ? launch_split<I8, false, true, false>(ta, tb, sp, smem, st)      \
                        : launch_split<I8, false, false, false>(ta, tb, sp, smem, st);    \
    } while (0)
    if (int8) Q8K_SPLIT(true);
    Q8K_SPLIT(false);
#undef Q8K_SPLIT
}

}  // namespace q8k
