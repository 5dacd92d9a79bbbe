// Two-SM bf16 GEMM with the operand roles swapped: out (M, N) = x (M, K) . w (N, K)^T (+ bias) with 256 weight rows on the M side of the MMA
// (128 per CTA of the pair) and `nb` activation rows, any multiple of 16 up to 256, on its N side; and the same with SwiGLU on top.
//
// For products of some hundred rows, the prompts of generation.  The kernel of gemm2.cu has 256 x 256 tiles only: 777 rows are four row tiles, the last with
// 9 rows of its own, and the tiles of a product fill whole rounds of the 74 pairs only by chance.  Here the rows are spread evenly over the row tiles
// and their number is chosen so that the last round is full (pick_rows).  Loads are what bounds these products: a pair reads (256 + nb) rows for
// 256 nb products, so that small nb cost more per product; the rule weighs both.  Measured figures stand with the dispatch (ops/kernels.py, _swapped).
//
// SwiGLU: w holds 2 N rows, out = (x . w1^T) * silu(x . w2^T).  Lanes 0..63 of a CTA are rows of w1, lanes 64..127 the same rows of w2; the two warps that
// hold the factors of an output exchange half of them through shared memory and finish half of the rows each.  Unlike the plain product it is taken for
// any number of rows, since the launch and the pass over the factors that it saves grow with them (ops/kernels.py, decoder_forward).
//
// Structure as in gemm2.cu: warp 0 TMA producer, warp 1 MMA issuer (leader CTA), sixteen epilogue warps, double-buffered accumulator.  A tensor memory lane is an
// output column and a column is a row of the output, so an epilogue warp turns 32 columns x 16 rows round through its own shared memory (one
// 2-byte store per value, 64 contiguous bytes per warp) and one TMA store.
#include "common.cuh"
#include "decoder_ops.h"
#include "pdl.cuh"
#include "two_sm.cuh"

namespace {

constexpr int WR = 128;                       // weight rows per CTA
constexpr int BK = 64;
constexpr int W_BYTES = WR * BK * 2;          // 16 KB
constexpr int MAX_NB = 256, NB_STEP = 16;
constexpr int MAX_STAGES = 8;
constexpr int THREADS = 576;                  // TMA warp + MMA warp + 16 epilogue warps
constexpr int CHUNK = 16;                     // output rows per epilogue step
constexpr int STAGE_OUT = 32 * CHUNK * 2;     // 1 KB: a warp's staging buffer, two of them per warp (SwiGLU: two halves of one, the other for the exchange)
constexpr int OUT_BYTES = 16 * 2 * STAGE_OUT;
constexpr int SMEM_MAX = 225 * 1024;
constexpr int TMEM_COLS = 512;

struct Args {
    const bf16* bias;          // N entries or null
    int M, N, K;
    int nb, m_tiles, n_tiles, num_kb, stages;
    int early_w;               // no kernel directly in front of this one writes the weights: they are read before it has completed
    unsigned int* status;
};

template <bool SWIGLU>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 1)
gemm2t_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmD, const Args g) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int stage_bytes = W_BYTES + (g.nb / 2) * (BK * 2);         // a multiple of 1024: nb / 2 is one of 8
    uint8_t* out_smem = smem + g.stages * stage_bytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(out_smem + OUT_BYTES);
    uint64_t* full = bars;                        // [MAX_STAGES]  used in the leader CTA: bytes of both CTAs' loads
    uint64_t* empty = bars + MAX_STAGES;          // [MAX_STAGES]  one per CTA, raised by the leader's commit
    uint64_t* acc_full = bars + 2 * MAX_STAGES;   // [2]           one per CTA, raised by the leader's commit
    uint64_t* acc_empty = acc_full + 2;           // [2]           used in the leader CTA: all epilogue warps of the pair arrive
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();              // 0 = leader
    const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
    const int total = g.m_tiles * g.n_tiles;

    if (threadIdx.x == 0) {
        for (int s = 0; s < g.stages; s++) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; b++) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 2 * 16); }
        *abort_flag = 0;
        mbar_fence_init();
        tma_prefetch_desc(&tmW); tma_prefetch_desc(&tmX); tma_prefetch_desc(&tmD);
    }
    cluster_sync_all();                                   // both CTAs' barriers exist before anyone signals them
    if (warp == 1) { tmem_alloc_2sm(tmem_slot, TMEM_COLS); tmem_relinquish_2sm(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    // output columns of a pair's tile and of a CTA's share; the row tiles of one weight tile run side by side, so that it is read from DRAM once
    constexpr int COLS = SWIGLU ? 128 : 256, CTA_COLS = COLS / 2;
    auto col0 = [&](int w) { return (w / g.m_tiles) * COLS + (int)rank * CTA_COLS; };
    auto row0 = [&](int w) { return (w % g.m_tiles) * g.nb; };

    auto load_w = [&](int n0, int kb, int stage) {
        uint8_t* dst = smem + stage * stage_bytes;
        const uint32_t lead_full = map_to_cta(smem_u32(&full[stage]), 0);
        if (rank == 0) mbar_expect_tx(&full[stage], 2 * stage_bytes);              // bytes of both CTAs
        if (SWIGLU) {
            tma_load_2d_2sm(dst, &tmW, lead_full, kb * BK, n0);                    // boxes {64 k, 64 rows}
            tma_load_2d_2sm(dst + W_BYTES / 2, &tmW, lead_full, kb * BK, g.N + n0);
        } else {
            tma_load_2d_2sm(dst, &tmW, lead_full, kb * BK, n0);                    // box {64 k, 128 rows}
        }
    };
    int early = g.early_w && pair < total ? min(g.stages, g.num_kb) : 0;          // stages filled with weights while the kernel before drains
    if (warp == 0 && lane == 0)
        for (int kb = 0; kb < early; kb++) load_w(col0(pair), kb, kb);
    __syncwarp();
    pdl_wait();

    if (warp == 0) {
        if (lane == 0) {
            int stage = 0; uint32_t phase = 0;
            bool fail = false;
            for (int w = pair; w < total && !fail; w += npairs) {
                const int n0 = col0(w), m0 = row0(w) + (int)rank * (g.nb / 2);
                for (int kb = 0; kb < g.num_kb; kb++) {
                    if (kb >= early) {
                        if (!mbar_wait(&empty[stage], phase ^ 1, abort_flag, g.status, 0xD00 + stage)) { fail = true; break; }
                        load_w(n0, kb, stage);
                    }
                    tma_load_2d_2sm(smem + stage * stage_bytes + W_BYTES, &tmX, map_to_cta(smem_u32(&full[stage]), 0), kb * BK, m0);    // box {64 k, nb / 2 rows}
                    if (++stage == g.stages) { stage = 0; phase ^= 1; }
                }
                early = 0;
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            const bool leader = elect_one();
            const uint32_t idesc = umma_idesc_bf16(256, 0, 0, 0) | ((uint32_t)(g.nb >> 3) << 17);
            const uint64_t dw0 = umma_desc_sw128(smem_u32(smem), 16, 1024), dx0 = umma_desc_sw128(smem_u32(smem + W_BYTES), 16, 1024);
            int stage = 0; uint32_t phase = 0;
            int it = 0;
            bool ok = true;
            for (int w = pair; w < total && ok; w += npairs, it++) {
                const int buf = it & 1;
                ok = __all_sync(0xffffffffu, mbar_wait(&acc_empty[buf], ((it >> 1) & 1) ^ 1, abort_flag, g.status, 0xD20 + buf)) != 0;
                tc_fence_after();
                for (int kb = 0; kb < g.num_kb && ok; kb++) {
                    ok = __all_sync(0xffffffffu, mbar_wait(&full[stage], phase, abort_flag, g.status, 0xD10 + stage)) != 0;
                    if (!ok) break;
                    tc_fence_after();
                    const uint64_t at = (uint64_t)(stage * (stage_bytes >> 4));
                    if (leader) {
                        #pragma unroll
                        for (int k = 0; k < BK / 16; k++)
                            umma_ss_2sm(tmem_base + buf * 256, dw0 + at + 2 * k, dx0 + at + 2 * k, idesc, (kb | k) > 0);
                        umma_commit_2sm(&empty[stage]);
                        if (kb == g.num_kb - 1) umma_commit_2sm(&acc_full[buf]);
                    }
                    if (++stage == g.stages) { stage = 0; phase ^= 1; }
                }
            }
        }
    } else {
        const int ew = warp - 2, q = warp & 3, grp = ew >> 2;
        uint8_t* wbuf = out_smem + ew * 2 * STAGE_OUT;
        const uint32_t lead_acc_empty = map_to_cta(smem_u32(&acc_empty[0]), 0);
        int it = 0;
        uint32_t n_out = 0;
        for (int w = pair; w < total; w += npairs, it++) {
            const int buf = it & 1;
            const bool ok = mbar_wait(&acc_full[buf], (it >> 1) & 1, abort_flag, g.status, 0xD30 + buf);
            tc_fence_after();
            const int n0 = col0(w) + (SWIGLU ? q & 1 : q) * 32, m0 = row0(w);
            float bias = 0.f;
            if (!SWIGLU && g.bias != nullptr && n0 + lane < g.N) bias = __bfloat162float(g.bias[n0 + lane]);
            for (int c = grp * CHUNK; c < g.nb; c += 4 * CHUNK) {
                uint32_t v[CHUNK];
                tmem_ld16(tmem_base + ((uint32_t)(q * 32) << 16) + buf * 256 + c, v);
                tmem_ld_wait();
                uint8_t* ob = wbuf + (n_out & 1) * (SWIGLU ? STAGE_OUT / 2 : STAGE_OUT);
                if (lane == 0) tma_store_wait_read<1>();          // the store issued two steps ago has read this buffer
                __syncwarp();
                bf16* o = reinterpret_cast<bf16*>(ob);
                const int r0 = SWIGLU ? (q >> 1) * (CHUNK / 2) : 0;       // SwiGLU: this warp finishes rows r0 .. r0 + 7
                if (SWIGLU) {
                    // warp q (w1) and warp q + 2 (w2) of the group: each gives the other its values of the rows that the other finishes
                    float* mine = reinterpret_cast<float*>(wbuf + STAGE_OUT);
                    const float* theirs = reinterpret_cast<const float*>(out_smem + (ew ^ 2) * 2 * STAGE_OUT + STAGE_OUT);
                    const bool second = q >= 2;
                    const int bar = 1 + grp * 2 + (q & 1);
                    #pragma unroll
                    for (int e = 0; e < CHUNK / 2; e++) mine[e * 32 + lane] = __uint_as_float(second ? v[e] : v[CHUNK / 2 + e]);
                    asm volatile("bar.sync %0, 64;" ::"r"(bar) : "memory");
                    float x[CHUNK / 2];
                    #pragma unroll
                    for (int e = 0; e < CHUNK / 2; e++) x[e] = theirs[e * 32 + lane];
                    asm volatile("bar.sync %0, 64;" ::"r"(bar) : "memory");      // both have read: the next step may write
                    #pragma unroll
                    for (int e = 0; e < CHUNK / 2; e++) {
                        const float own = __uint_as_float(second ? v[CHUNK / 2 + e] : v[e]), got = x[e];
                        const float x1 = second ? got : own, x2 = second ? own : got;
                        o[e * 32 + lane] = __float2bfloat16_rn(x1 * x2 / (1.0f + __expf(-x2)));
                    }
                } else {
                    #pragma unroll
                    for (int e = 0; e < CHUNK; e++) o[e * 32 + lane] = __float2bfloat16_rn(__uint_as_float(v[e]) + bias);
                }
                fence_async_smem();
                __syncwarp();
                if (lane == 0) {
                    if (ok && n0 < g.N && m0 + c + r0 < g.M) tma_store_2d(&tmD, ob, n0, m0 + c + r0);
                    tma_store_commit();                            // one group per step, also an empty one: the wait above counts steps
                }
                n_out++;
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(lead_acc_empty + buf * 8);      // this warp's part of the accumulator is read
            if (!SWIGLU && __any_sync(0xffffffffu, *abort_flag)) break;        // (SwiGLU: two warps meet at barriers, both go through all tiles)
        }
        if (lane == 0) tma_store_wait<0>();
    }

    pdl_trigger();
    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {
        long long t0 = clock64();
        while (clock64() - t0 < 2000000ll) { __nanosleep(1000); }
    }
    cluster_sync_all();                                   // nobody may still signal a barrier of a CTA that has left
    tc_fence_after();
    if (warp == 1) tmem_dealloc_2sm(tmem_base, TMEM_COLS);
}

// Row tiles of a product and the rows of each: the number of tiles that takes the pairs the least time.  A k-block of a tile takes as long as its
// 256 + nb rows take to arrive.
void pick_rows(int M, int n_tiles, int pairs, int& m_tiles, int& nb) {
    long long best = -1;
    for (int t = CEIL_DIV(M, MAX_NB); t <= CEIL_DIV(M, 64); t++) {
        const int rows = CEIL_DIV(CEIL_DIV(M, t), NB_STEP) * NB_STEP;
        const int tiles = CEIL_DIV(M, rows);
        const long long cost = CEIL_DIV((long long)tiles * n_tiles, pairs) * (256 + rows);
        if (best < 0 || cost < best) { best = cost; m_tiles = tiles; nb = rows; }
    }
}

template <bool SWIGLU>
int launch_gemm2t(bf16* out, const bf16* x, const bf16* w, const bf16* bias, int M, int N, int K, int ldx, int ldw, int ldo, int rows, int early_w,
                  cudaStream_t stream) {
    if (M <= 0 || N <= 0 || K <= 0) return 0;
    if ((K % 8) || (N % 8) || (ldx % 8) || (ldw % 8) || (ldo % 8) || ldx < K || ldw < K || ldo < N) return -1;
    if (SWIGLU && (N % 128)) return -1;
    int sms = llmc_device_sm_count(); if (sms <= 0) sms = 148;
    Args g;
    g.early_w = early_w;
    g.bias = bias; g.M = M; g.N = N; g.K = K; g.status = llmc_status_ptr();
    g.n_tiles = CEIL_DIV(N, SWIGLU ? 128 : 256);
    g.num_kb = CEIL_DIV(K, BK);
    if (rows > 0) {
        if (rows % NB_STEP || rows > MAX_NB) return -1;
        g.nb = rows; g.m_tiles = CEIL_DIV(M, rows);
    } else {
        pick_rows(M, g.n_tiles, sms / 2, g.m_tiles, g.nb);
    }
    const int stage_bytes = W_BYTES + (g.nb / 2) * (BK * 2);
    g.stages = (SMEM_MAX - 1024 - OUT_BYTES - 512) / stage_bytes;
    if (g.stages > MAX_STAGES) g.stages = MAX_STAGES;
    CUtensorMap tmW, tmX, tmD;
    int rc;
    {
        uint64_t dims[2] = {(uint64_t)K, (uint64_t)N * (SWIGLU ? 2 : 1)}, strides[2] = {2, (uint64_t)ldw * 2};
        uint32_t box[2] = {BK, SWIGLU ? WR / 2 : WR};
        if ((rc = llmc_get_tensormap(&tmW, w, 2, 2, dims, strides, box, 3))) return rc;
        uint64_t dimx[2] = {(uint64_t)K, (uint64_t)M}, strx[2] = {2, (uint64_t)ldx * 2};
        uint32_t boxx[2] = {BK, (uint32_t)(g.nb / 2)};
        if ((rc = llmc_get_tensormap(&tmX, x, 2, 2, dimx, strx, boxx, 3))) return rc;
        uint64_t dimd[2] = {(uint64_t)N, (uint64_t)M}, strd[2] = {2, (uint64_t)ldo * 2};
        uint32_t boxd[2] = {32, SWIGLU ? CHUNK / 2 : CHUNK};
        if ((rc = llmc_get_tensormap(&tmD, out, 2, 2, dimd, strd, boxd, 0))) return rc;
    }
    const int total = g.m_tiles * g.n_tiles;
    const int grid = 2 * (total < sms / 2 ? total : sms / 2);
    const int smem = 1024 + g.stages * stage_bytes + OUT_BYTES + 512;
    static bool configured = false;
    if (!configured) {
        CUDA_CHECK(cudaFuncSetAttribute(gemm2t_kernel<SWIGLU>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_MAX));
        configured = true;
    }
    CUDA_CHECK(launch_pdl(gemm2t_kernel<SWIGLU>, dim3(grid), dim3(THREADS), smem, stream, 0, tmW, tmX, tmD, g));
    return 0;
}

}  // namespace

// out (M, N) = x (M, K) . w (N, K)^T (+ bias).  K, N and the row strides are multiples of 8, the pointers 16-byte aligned.  rows: activation rows of a tile, a
// multiple of 16 up to 256 (0: pick_rows).
extern "C" int llmc_gemm2t(bf16* out, const bf16* x, const bf16* w, const bf16* bias, int M, int N, int K, int ldx, int ldw, int ldo, int rows,
                           cudaStream_t stream) {
    return launch_gemm2t<false>(out, x, w, bias, M, N, K, ldx, ldw, ldo, rows, 0, stream);
}

// The same behind a kernel that does not write w (csrc/decoder.cu): an early launch fills the stages with weights while that kernel drains.  What other
// kernels before it wrote is complete: it triggers the launch after its own wait (pdl.cuh).
extern "C" int llmc_gemm2t_chained(bf16* out, const bf16* x, const bf16* w, int M, int N, int K, int ldx, int ldw, int ldo, cudaStream_t stream) {
    return launch_gemm2t<false>(out, x, w, nullptr, M, N, K, ldx, ldw, ldo, 0, 1, stream);
}

// out (M, N) = (x . w1^T) * silu(x . w2^T) with w = [w1; w2] of 2 N rows; N a multiple of 128
extern "C" int llmc_gemm2t_swiglu(bf16* out, const bf16* x, const bf16* w, int M, int N, int K, int ldx, int ldw, int ldo, int rows, cudaStream_t stream) {
    return launch_gemm2t<true>(out, x, w, nullptr, M, N, K, ldx, ldw, ldo, rows, 0, stream);
}
extern "C" int llmc_gemm2t_swiglu_chained(bf16* out, const bf16* x, const bf16* w, int M, int N, int K, int ldx, int ldw, int ldo, cudaStream_t stream) {
    return launch_gemm2t<true>(out, x, w, nullptr, M, N, K, ldx, ldw, ldo, 0, 1, stream);
}
