// Products with few rows: out (M, N) = x (M, K) . w (N, K)^T (+ bias), M <= 128, and the same with SwiGLU on top.  These are the
// products of decoding steps and short prompts.  They are bound by streaming the weights once, so the roles of the tcgen05 operands
// are swapped: 128 weight rows are the M side of the MMA and the activation rows, padded to a multiple of 16, its N side (a 128-row
// activation tile would be padding, and 256 weight rows per tile leave most SMs without work: 16 tiles for N = 4096).
//
// K is split over the CTAs of a cluster (1, 2, 4 or 8 of them), so that a product with few weight tiles still has enough CTAs in
// flight to reach the memory rate.  Every CTA accumulates its K slice in TMEM, puts the fp32 partial tile into its own shared memory,
// and after one cluster barrier each CTA adds its share of the rows over all CTAs of the cluster through distributed shared memory,
// in the order of the slices: deterministic, no workspace, no second launch.
//
// The kernel is launched with programmatic stream serialization: while the kernel before it drains, its CTAs set up and ask for the
// first kilobyte of each weight row of their slice in L2 (a hint only: nothing is read before the predecessor has completed).
//
// Alone, after an L2 flush, the 128 x 256 tiles of the training GEMM in brackets: 32 x 4096 x 14336 (M x N x K) 36 us (101),
// 32 x 6144 x 4096 23 us (38), 32 x 28672 x 4096 58 us (69), 100 x 2048 x 7168 23 us (52).  Inside a replayed decoding step (4 rows, 4 layers
// of 2048 channels, LM head of 128256 rows) this kernel takes the step to 277 us; a weight-streaming kernel on warp-level MMAs with the same
// early launch and prefetch, used for the products of at most 8 rows, left it at 290 us.
//
// Warps of a CTA: 0 TMA producer, 1 MMA issuer, 2-5 epilogue.  Two CTAs fit an SM.
#include "common.cuh"
#include "pdl.cuh"

namespace {

constexpr int WR = 128;                       // weight rows per tile
constexpr int BK = 64;                        // K elements per stage: one 128-byte swizzled row
constexpr int W_BYTES = WR * BK * 2;          // 16 KB
constexpr int MAX_STAGES = 6;
constexpr int SMEM_BUDGET = 112 * 1024;       // two CTAs per SM
constexpr int THREADS = 192;
constexpr int PREFETCH_BYTES = 1024;          // of each weight row: 296 resident CTAs x 128 KB stay well inside L2
constexpr int MAX_M = 128;

struct Args {
    bf16* out;
    const bf16* bias;          // N entries or null
    const bf16* w;             // for the prefetch
    int M, N, K, ldo, ldw;
    int nb;                    // activation rows of a tile: M rounded up to 16
    int stages, num_kb, kb_per_split;
    int vec_out;               // out rows start on 4-byte boundaries
    unsigned int* status;
};

DEVINL uint32_t cluster_size() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(r)); return r; }
DEVINL uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
DEVINL void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
DEVINL float2 ld_peer2(uint32_t addr, uint32_t rank) {
    uint32_t ra; float2 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(ra) : "memory");
    return v;
}
DEVINL void prefetch_l2(const void* p, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// SWIGLU: w holds 2 N rows; tile t covers rows 64 t .. of the first half and the same rows of the second half, and
// out = first * silu(second).  Otherwise tile t covers rows 128 t ..
template <bool SWIGLU>
__global__ void __launch_bounds__(THREADS, 2)
stream_gemm_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const Args g) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int stage_bytes = W_BYTES + g.nb * (BK * 2);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + g.stages * stage_bytes);
    uint64_t* full = bars;                       // [MAX_STAGES]
    uint64_t* empty = bars + MAX_STAGES;         // [MAX_STAGES]
    uint64_t* acc_full = bars + 2 * MAX_STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t S = cluster_size(), rank = cluster_rank();
    const int tile = blockIdx.x / S;
    constexpr int ROWS = SWIGLU ? WR / 2 : WR;   // output columns of a tile
    const int n0 = tile * ROWS;
    const int kb0 = rank * g.kb_per_split, kb1 = min(g.num_kb, kb0 + g.kb_per_split);
    const uint32_t tmem_cols = g.nb <= 32 ? 32 : g.nb <= 64 ? 64 : 128;

    if (threadIdx.x == 0) {
        for (int s = 0; s < g.stages; s++) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        mbar_init(acc_full, 1);
        *abort_flag = 0;
        mbar_fence_init();
        tma_prefetch_desc(&tmW); tma_prefetch_desc(&tmX);
    }
    if (warp == 1) { tmem_alloc(tmem_slot, tmem_cols); tmem_relinquish(); }
    if (warp >= 2 && kb0 < kb1) {
        const int r = threadIdx.x - 64;
        const int row = SWIGLU ? (r < 64 ? n0 + r : g.N + n0 + r - 64) : n0 + r;
        const bool in = SWIGLU ? n0 + (r & 63) < g.N : row < g.N;
        const int bytes = min(min(kb1 * BK, g.K) - kb0 * BK, PREFETCH_BYTES / 2) * 2;      // K is a multiple of 8: whole 16-byte units
        if (in) prefetch_l2(g.w + (size_t)row * g.ldw + kb0 * BK, bytes);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_wait();
    pdl_trigger();

    if (warp == 0) {
        if (lane == 0) {
            for (int kb = kb0; kb < kb1; kb++) {
                const int it = kb - kb0, st = it % g.stages;
                if (!mbar_wait_relaxed(&empty[st], ((it / g.stages) & 1) ^ 1, abort_flag, g.status, 0x900)) break;
                uint8_t* dst = smem + st * stage_bytes;
                mbar_expect_tx(&full[st], stage_bytes);
                if (SWIGLU) {
                    tma_load_2d(dst, &tmW, &full[st], kb * BK, n0);                                   // boxes {64 k, 64 rows}
                    tma_load_2d(dst + W_BYTES / 2, &tmW, &full[st], kb * BK, g.N + n0);
                } else {
                    tma_load_2d(dst, &tmW, &full[st], kb * BK, n0);                                   // box {64 k, 128 rows}
                }
                tma_load_2d(dst + W_BYTES, &tmX, &full[st], kb * BK, 0);                              // box {64 k, nb rows}
            }
        }
    } else if (warp == 1) {
        const bool leader = elect_one();
        const uint32_t idesc = umma_idesc_bf16(WR, 0, 0, 0) | ((uint32_t)(g.nb >> 3) << 17);
        bool ok = true;
        for (int kb = kb0; kb < kb1 && ok; kb++) {
            const int it = kb - kb0, st = it % g.stages;
            ok = __all_sync(0xffffffffu, mbar_wait_relaxed(&full[st], (it / g.stages) & 1, abort_flag, g.status, 0x910)) != 0;
            if (!ok) break;
            tc_fence_after();
            const uint64_t dw = umma_desc_sw128(smem_u32(smem + st * stage_bytes), 16, 1024);
            const uint64_t dx = umma_desc_sw128(smem_u32(smem + st * stage_bytes + W_BYTES), 16, 1024);
            if (leader) {
                #pragma unroll
                for (int kk = 0; kk < BK / 16; kk++) umma_ss(tmem_base, dw + 2 * kk, dx + 2 * kk, idesc, (it | kk) > 0);
                umma_commit(&empty[st]);
                if (kb == kb1 - 1) umma_commit(acc_full);
            }
        }
    } else {
        // partial tile -> shared memory as [activation row][weight row]: the stage buffers are free once the last MMA has completed
        float* part = reinterpret_cast<float*>(smem);
        const int r = (warp & 3) * 32 + lane;                 // weight row = TMEM lane
        if (kb0 < kb1) {
            const bool ok = mbar_wait(acc_full, 0, abort_flag, g.status, 0x920);
            tc_fence_after();
            for (int c = 0; c < g.nb; c += 16) {
                uint32_t v[16];
                tmem_ld16(tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + c, v);
                tmem_ld_wait();
                #pragma unroll
                for (int e = 0; e < 16; e++) part[(c + e) * WR + r] = ok ? __uint_as_float(v[e]) : 0.f;
            }
            tc_fence_before();
        } else {
            for (int c = 0; c < g.nb; c++) part[c * WR + r] = 0.f;      // more CTAs in the cluster than K blocks
        }
    }
    __syncwarp();
    cluster_sync();                                           // every partial tile of the cluster is in place
    if (warp >= 2) {
        constexpr int PAIRS = ROWS / 2, GROUPS = 128 / PAIRS;           // column pairs of a tile; rows handled side by side
        const int tid = threadIdx.x - 64;
        const int pi = tid % PAIRS, grp = tid / PAIRS;
        const int n = n0 + 2 * pi;
        const uint32_t base = smem_u32(smem) + pi * 8;
        float b0 = 0.f, b1 = 0.f;
        if (!SWIGLU && g.bias != nullptr) {
            if (n < g.N) b0 = __bfloat162float(g.bias[n]);
            if (n + 1 < g.N) b1 = __bfloat162float(g.bias[n + 1]);
        }
        for (int m = (int)rank * GROUPS + grp; m < g.M; m += (int)S * GROUPS) {
            float2 v = make_float2(0.f, 0.f), u = make_float2(0.f, 0.f);
            for (uint32_t s = 0; s < S; s++) {
                const float2 p = ld_peer2(base + m * (WR * 4), s);
                v.x += p.x; v.y += p.y;
                if (SWIGLU) {
                    const float2 p2 = ld_peer2(base + m * (WR * 4) + (WR / 2) * 4, s);
                    u.x += p2.x; u.y += p2.y;
                }
            }
            if (SWIGLU) {
                v.x *= u.x / (1.0f + __expf(-u.x));
                v.y *= u.y / (1.0f + __expf(-u.y));
            } else { v.x += b0; v.y += b1; }
            bf16* o = g.out + (size_t)m * g.ldo + n;
            if (n + 1 < g.N && g.vec_out) {
                *reinterpret_cast<uint32_t*>(o) = pack_bf16x2(v.x, v.y);
            } else {
                if (n < g.N) o[0] = __float2bfloat16_rn(v.x);
                if (n + 1 < g.N) o[1] = __float2bfloat16_rn(v.y);
            }
        }
    }
    __syncwarp();
    cluster_sync();                                           // no CTA leaves while a peer may still read its shared memory
    tc_fence_after();
    if (warp == 1) tmem_dealloc(tmem_base, tmem_cols);
}

// CTAs per weight tile: as many as keep all of them resident at once (two per SM) and leave each at least four K blocks
int pick_split(int tiles, int num_kb, int sms) {
    int s = 1;
    while (s < 8 && tiles * s * 2 <= 2 * sms && num_kb >= s * 2 * 4) s *= 2;
    return s;
}

template <bool SWIGLU>
int launch_stream(bf16* out, const bf16* x, const bf16* w, const bf16* bias, int M, int N, int K, int ldx, int ldw, int ldo, cudaStream_t stream) {
    if (M <= 0 || M > MAX_M || N <= 0 || K <= 0 || (K % 8) || (ldx % 8) || (ldw % 8) || ldx < K || ldw < K || ldo < N) return -1;
    Args g;
    g.out = out; g.bias = bias; g.w = w; g.M = M; g.N = N; g.K = K; g.ldo = ldo; g.ldw = ldw;
    g.nb = (M + 15) & ~15;
    g.num_kb = CEIL_DIV(K, BK);
    const int stage_bytes = W_BYTES + g.nb * (BK * 2);
    g.stages = (SMEM_BUDGET - 2048) / stage_bytes;
    if (g.stages > MAX_STAGES) g.stages = MAX_STAGES;
    g.vec_out = (ldo % 2 == 0) && (reinterpret_cast<uintptr_t>(out) & 3) == 0;
    g.status = llmc_status_ptr();
    CUtensorMap tmW, tmX;
    {
        uint64_t dims[2] = {(uint64_t)K, (uint64_t)(SWIGLU ? 2 * (uint64_t)N : (uint64_t)N)};
        uint64_t strides[2] = {2, (uint64_t)ldw * 2};
        uint32_t box[2] = {BK, SWIGLU ? WR / 2 : WR};
        int rc = llmc_get_tensormap(&tmW, w, 2, 2, dims, strides, box, 3);
        if (rc) return rc;
        uint64_t dimx[2] = {(uint64_t)K, (uint64_t)M};
        uint64_t strx[2] = {2, (uint64_t)ldx * 2};
        uint32_t boxx[2] = {BK, (uint32_t)g.nb};
        rc = llmc_get_tensormap(&tmX, x, 2, 2, dimx, strx, boxx, 3);
        if (rc) return rc;
    }
    int sms = llmc_device_sm_count(); if (sms <= 0) sms = 148;
    const int tiles = CEIL_DIV(N, SWIGLU ? WR / 2 : WR);
    const int S = pick_split(tiles, g.num_kb, sms);
    g.kb_per_split = CEIL_DIV(g.num_kb, S);
    const int smem = g.stages * stage_bytes + 1024 + 256;
    static bool configured = false;
    if (!configured) {
        CUDA_CHECK(cudaFuncSetAttribute(stream_gemm_kernel<SWIGLU>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BUDGET));
        configured = true;
    }
    CUDA_CHECK(launch_pdl(stream_gemm_kernel<SWIGLU>, dim3(tiles * S), dim3(THREADS), smem, stream, S, tmW, tmX, g));
    return 0;
}

}  // namespace

// out (M, N) = x (M, K) . w (N, K)^T (+ bias) for M <= 128; K and the row strides of x and w are multiples of 8 elements.
extern "C" int llmc_stream_gemm(bf16* out, const bf16* x, const bf16* w, const bf16* bias, int M, int N, int K, int ldx, int ldw, int ldo,
                                cudaStream_t stream) {
    return launch_stream<false>(out, x, w, bias, M, N, K, ldx, ldw, ldo, stream);
}

// out (M, N) = (x . w1^T) * silu(x . w2^T) with w = [w1; w2] of 2 N rows, M <= 128; N a multiple of 64
extern "C" int llmc_stream_gemm_swiglu(bf16* out, const bf16* x, const bf16* w, int M, int N, int K, int ldx, int ldw, int ldo, cudaStream_t stream) {
    if (N % 64) return -1;
    return launch_stream<true>(out, x, w, nullptr, M, N, K, ldx, ldw, ldo, stream);
}

// The same product for the at most 8 rows of a decoding step
extern "C" int llmc_skinny_gemm(bf16* out, const bf16* x, const bf16* w, int M, int N, int K, int ldx, int ldw, int ldo, cudaStream_t stream) {
    if (M > 8) return -1;
    return launch_stream<false>(out, x, w, nullptr, M, N, K, ldx, ldw, ldo, stream);
}
