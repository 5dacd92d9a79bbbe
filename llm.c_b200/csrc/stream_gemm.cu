// Products with few tiles: out (M, N) = x (M, K) . w (N, K)^T (+ bias), x . w (K, N), and the first with SwiGLU on top.  These are the products
// of decoding steps, short prompts and small training batches.
// The roles of the tcgen05 operands are swapped: 128 weight rows are the M side of the MMA and up to 256 activation rows, padded to a
// multiple of 16, its N side.  A product of at most 128 rows then has no padded rows, and weight tiles of 128 instead of 256 columns
// leave fewer SMs without work.
//
// K is split over the CTAs of a cluster (1, 2, 4 or 8 of them), so that a product with few weight tiles still has enough CTAs in
// flight to reach the memory rate.  Every CTA accumulates its K slice in TMEM, puts the fp32 partial tile into its own shared memory,
// and after one cluster barrier each CTA adds its share of the rows over all CTAs of the cluster through distributed shared memory,
// in the order of the slices: deterministic, no workspace, no second launch.
//
// The kernel is launched with programmatic stream serialization: while the kernel before it drains, its CTAs set up and ask for the
// first kilobyte of each weight row of their slice in L2 (a hint only).  Behind a kernel that does not write the weights (the chained entry
// points) they fill their stages with them; nothing else is read before the predecessor has completed.
//
// Alone, after an L2 flush, the 128 x 256 tiles of the training GEMM in brackets: 32 x 4096 x 14336 (M x N x K) 36 us (101),
// 32 x 6144 x 4096 23 us (38), 32 x 28672 x 4096 58 us (69), 100 x 2048 x 7168 23 us (52).  Inside a replayed decoding step (4 rows, 4 layers
// of 2048 channels, LM head of 128256 rows) this kernel took the step to 277 us; a weight-streaming kernel on warp-level MMAs with the same
// early launch and prefetch, used for the products of at most 8 rows, left it at 290 us (at 284 us for the LM head alone), although launched
// by itself it is faster (4 x 28672 x 4096 50 us against 59; skinny_gemm_kernel in decode.cu).  More rows (input gradients, in a chain, the training GEMM's tiles in
// brackets): 256 x 768 x 768 4.9 us (6.3), 256 x 768 x 3072 7.9 us (16.3), 256 x 768 x 50304 44 us (291 after an L2 flush).  Forward products of some hundred rows
// cut the same way against the tiles of gemm2t.cu: 256 x 768 x 768 5.1 us (6.2), 256 x 768 x 3072 7.9 (14.1), 512 x 2048 x 2048 11.2 (11.7).
//
// Warps of a CTA: 0 TMA producer, 1 MMA issuer, 2-5 epilogue.  Two CTAs fit an SM.
#include "common.cuh"
#include "decoder_ops.h"
#include "pdl.cuh"

namespace {

constexpr int WR = 128;                       // weight rows (output columns) per tile
constexpr int BK = 64;                        // K elements per stage: one 128-byte swizzled row
constexpr int W_BYTES = WR * BK * 2;          // 16 KB
constexpr int MAX_NB = 256;                   // activation rows per tile
constexpr int MAX_STAGES = 6;
constexpr int SMEM_TWO = 112 * 1024;          // two CTAs per SM (at most 128 activation rows: 16 to 32 KB per stage)
constexpr int SMEM_ONE = 224 * 1024;          // one CTA per SM (up to 48 KB per stage)
constexpr int THREADS = 192;
constexpr int PREFETCH_BYTES = 1024;          // of each weight row: 296 resident CTAs x 128 KB stay well inside L2
constexpr int MAX_SPLIT = 8;

enum Mode : int { STORE = 0, SWIGLU = 1 };

struct Args {
    bf16* out;
    float* out32; int cols32;  // in place of out (null: out): the bf16 results as fp32, the first cols32 columns, in rows of as many
    int* advance;              // a counter to add 1 to (null: none)
    const bf16* bias;          // N entries or null (STORE)
    const bf16* w;             // for the prefetch
    int M, N, K, ldo, ldw;
    int nb;                    // activation rows of a tile, a multiple of 16
    int stages, num_kb, kb_per_split;
    int vec_out;               // rows of out start on 8-byte boundaries
    int early_w;               // no kernel directly in front of this one writes the weights: they are read before it has completed
    unsigned int* status;
};

DEVINL uint32_t cluster_size() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(r)); return r; }
DEVINL uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
DEVINL void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
DEVINL float4 ld_peer4(uint32_t addr, uint32_t rank) {
    uint32_t ra; float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(ra) : "memory");
    return v;
}
// sum over the cluster's partial tiles in slice order; all loads are on their way before the first is added
DEVINL void sum_peers(float (&f)[4], uint32_t addr, uint32_t S) {
    float4 p[MAX_SPLIT];
    #pragma unroll
    for (uint32_t s = 0; s < MAX_SPLIT; s++) if (s < S) p[s] = ld_peer4(addr, s);
    f[0] = p[0].x; f[1] = p[0].y; f[2] = p[0].z; f[3] = p[0].w;
    #pragma unroll
    for (uint32_t s = 1; s < MAX_SPLIT; s++) if (s < S) { f[0] += p[s].x; f[1] += p[s].y; f[2] += p[s].z; f[3] += p[s].w; }
}
DEVINL float round_bf16(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
DEVINL void prefetch_l2(const void* p, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// W_MN: the weights are stored (K, N) (an input gradient); otherwise (N, K).
// SWIGLU: w holds 2 N rows; tile t covers rows 64 t .. of the first half and the same rows of the second half, and
// out = first * silu(second).  Otherwise tile t covers output columns 128 t ..
template <int MODE, bool W_MN>
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
    constexpr int COLS = MODE == SWIGLU ? WR / 2 : WR;   // output columns of a tile
    const int n0 = tile * COLS;
    const int m0 = blockIdx.y * g.nb;
    const int kb0 = rank * g.kb_per_split, kb1 = min(g.num_kb, kb0 + g.kb_per_split);
    const uint32_t tmem_cols = g.nb <= 32 ? 32 : g.nb <= 64 ? 64 : g.nb <= 128 ? 128 : 256;

    if (threadIdx.x == 0) {
        for (int s = 0; s < g.stages; s++) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        mbar_init(acc_full, 1);
        *abort_flag = 0;
        mbar_fence_init();
        tma_prefetch_desc(&tmW); tma_prefetch_desc(&tmX);
    }
    if (warp == 1) { tmem_alloc(tmem_slot, tmem_cols); tmem_relinquish(); }
    if (warp >= 2 && kb0 < kb1 && blockIdx.y == 0) {
        const int r = threadIdx.x - 64;
        if (W_MN) {
            // rows of w are K: the tile's columns of the slice's first rows
            const uint32_t bytes = 2 * min(WR, g.N - n0);      // N is a multiple of 8: whole 16-byte units
            for (int i = 0; i < PREFETCH_BYTES / (2 * WR); i++) {
                const int k = kb0 * BK + i * 128 + r;
                if (k < min(kb1 * BK, g.K)) prefetch_l2(g.w + (size_t)k * g.ldw + n0, bytes);
            }
        } else {
            const int row = MODE == SWIGLU ? (r < 64 ? n0 + r : g.N + n0 + r - 64) : n0 + r;
            const bool in = MODE == SWIGLU ? n0 + (r & 63) < g.N : row < g.N;
            const int bytes = min(min(kb1 * BK, g.K) - kb0 * BK, PREFETCH_BYTES / 2) * 2;      // K is a multiple of 8: whole 16-byte units
            if (in) prefetch_l2(g.w + (size_t)row * g.ldw + kb0 * BK, bytes);
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    auto load_w = [&](int kb, int st) {
        uint8_t* dst = smem + st * stage_bytes;
        mbar_expect_tx(&full[st], stage_bytes);
        if (W_MN) {
            tma_load_2d(dst, &tmW, &full[st], n0, kb * BK);                                   // boxes {64 n, 64 k}
            tma_load_2d(dst + W_BYTES / 2, &tmW, &full[st], n0 + 64, kb * BK);
        } else if (MODE == SWIGLU) {
            tma_load_2d(dst, &tmW, &full[st], kb * BK, n0);                                   // boxes {64 k, 64 rows}
            tma_load_2d(dst + W_BYTES / 2, &tmW, &full[st], kb * BK, g.N + n0);
        } else {
            tma_load_2d(dst, &tmW, &full[st], kb * BK, n0);                                   // box {64 k, 128 rows}
        }
    };
    auto load_x = [&](int kb, int st) { tma_load_2d(smem + st * stage_bytes + W_BYTES, &tmX, &full[st], kb * BK, m0); };       // box {64 k, nb rows}
    const int early = g.early_w ? min(g.stages, kb1 - kb0) : 0;       // stages filled with weights while the kernel before drains
    if (warp == 0 && lane == 0)
        for (int it = 0; it < early; it++) load_w(kb0 + it, it);
    __syncwarp();
    pdl_wait();
    pdl_trigger();
    if (g.advance != nullptr && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 64) *g.advance += 1;

    if (warp == 0) {
        if (lane == 0) {
            for (int it = 0; it < early; it++) load_x(kb0 + it, it);
            for (int kb = kb0 + early; kb < kb1; kb++) {
                const int it = kb - kb0, st = it % g.stages;
                if (!mbar_wait_relaxed(&empty[st], ((it / g.stages) & 1) ^ 1, abort_flag, g.status, 0x900)) break;
                load_w(kb, st);
                load_x(kb, st);
            }
        }
    } else if (warp == 1) {
        const bool leader = elect_one();
        const uint32_t idesc = umma_idesc_bf16(WR, 0, W_MN, 0) | ((uint32_t)(g.nb >> 3) << 17);
        bool ok = true;
        for (int kb = kb0; kb < kb1 && ok; kb++) {
            const int it = kb - kb0, st = it % g.stages;
            ok = __all_sync(0xffffffffu, mbar_wait_relaxed(&full[st], (it / g.stages) & 1, abort_flag, g.status, 0x910)) != 0;
            if (!ok) break;
            tc_fence_after();
            const uint64_t dw = umma_desc_sw128(smem_u32(smem + st * stage_bytes), W_MN ? BK * 128 : 16, 1024);
            const uint64_t dx = umma_desc_sw128(smem_u32(smem + st * stage_bytes + W_BYTES), 16, 1024);
            if (leader) {
                // 16 K elements: 32 bytes along a K-major row, 16 rows of 128 bytes of an N-major tile
                #pragma unroll
                for (int kk = 0; kk < BK / 16; kk++) umma_ss(tmem_base, dw + (W_MN ? 128 : 2) * kk, dx + 2 * kk, idesc, (it | kk) > 0);
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
        // four adjacent columns per thread; the rows are dealt to the CTAs of the cluster
        constexpr int QUADS = COLS / 4, GROUPS = 128 / QUADS;
        const int tid = threadIdx.x - 64;
        const int qd = tid % QUADS, grp = tid / QUADS;
        const int n = n0 + 4 * qd;
        const uint32_t base = smem_u32(smem) + qd * 16;
        const int rows = min(g.nb, g.M - m0);
        float bias[4] = {0.f, 0.f, 0.f, 0.f};
        if (MODE == STORE && g.bias != nullptr) {
            #pragma unroll
            for (int e = 0; e < 4; e++) if (n + e < g.N) bias[e] = __bfloat162float(g.bias[n + e]);
        }
        const bool vec = g.vec_out && n + 3 < g.N;
        for (int m = (int)rank * GROUPS + grp; m < rows; m += (int)S * GROUPS) {
            const size_t at = (size_t)(m0 + m) * g.ldo + n;
            float f[4];
            sum_peers(f, base + m * (WR * 4), S);
            if (MODE == SWIGLU) {
                float u[4];
                sum_peers(u, base + m * (WR * 4) + (WR / 2) * 4, S);
                #pragma unroll
                for (int e = 0; e < 4; e++) f[e] *= u[e] / (1.0f + __expf(-u[e]));
            } else {
                #pragma unroll
                for (int e = 0; e < 4; e++) f[e] += bias[e];
            }
            if (MODE == STORE && g.out32 != nullptr) {
                #pragma unroll
                for (int e = 0; e < 4; e++) if (n + e < g.cols32) g.out32[(size_t)(m0 + m) * g.cols32 + n + e] = round_bf16(f[e]);
            } else if (vec) {
                *reinterpret_cast<uint2*>(g.out + at) = make_uint2(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]));
            } else {
                #pragma unroll
                for (int e = 0; e < 4; e++) if (n + e < g.N) g.out[at + e] = __float2bfloat16_rn(f[e]);
            }
        }
    }
    // after an abandoned wait copies may still be on their way into this CTA's shared memory: give them time to land before it is freed
    if (*abort_flag) {
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000ll) { __nanosleep(1000); }
    }
    __syncwarp();
    cluster_sync();                                           // no CTA leaves while a peer may still read its shared memory
    tc_fence_after();
    if (warp == 1) tmem_dealloc(tmem_base, tmem_cols);
}

// The same product with so many weight tiles that every CTA gets several (the LM head of a decoding step), K unsplit: CTAs stay and their TMA
// warp runs on into the next tile while the epilogue warps, on one of two accumulators, finish the one before.  With a CTA per tile the loads of
// every tile start with the set-up of its CTA and end with its epilogue: 4 x 50304 x 768 17.0 us against 12.8, 100 x 50304 x 768 29 against 16,
// 16 x 128256 x 2048 86.5 against 83.8, 64 x 128256 x 4096 183 against 173 (6.1 TB/s).  The output leaves from the registers: a lane is an output
// column.
__global__ void __launch_bounds__(THREADS, 2)
stream_wide_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const Args g) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int stage_bytes = W_BYTES + g.nb * (BK * 2);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + g.stages * stage_bytes);
    uint64_t* full = bars;                       // [MAX_STAGES]
    uint64_t* empty = bars + MAX_STAGES;         // [MAX_STAGES]
    uint64_t* acc_full = bars + 2 * MAX_STAGES;  // [2]
    uint64_t* acc_empty = acc_full + 2;          // [2]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tiles = CEIL_DIV(g.N, WR);
    const int acc_cols = g.nb <= 16 ? 16 : g.nb <= 32 ? 32 : g.nb <= 64 ? 64 : 128;

    if (threadIdx.x == 0) {
        for (int s = 0; s < g.stages; s++) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; b++) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 4); }
        *abort_flag = 0;
        mbar_fence_init();
        tma_prefetch_desc(&tmW); tma_prefetch_desc(&tmX);
    }
    if (warp == 1) { tmem_alloc(tmem_slot, 2 * acc_cols); tmem_relinquish(); }
    if (warp >= 2) {
        // the first tile's rows into L2 while the kernel before drains
        const int row = blockIdx.x * WR + (int)threadIdx.x - 64;
        if (row < g.N) prefetch_l2(g.w + (size_t)row * g.ldw, 2 * min(g.K, PREFETCH_BYTES / 2));
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    auto load_w = [&](int tile, int kb, int st) {
        mbar_expect_tx(&full[st], stage_bytes);
        tma_load_2d(smem + st * stage_bytes, &tmW, &full[st], kb * BK, tile * WR);            // box {64 k, 128 rows}
    };
    int early = g.early_w ? min(g.stages, g.num_kb) : 0;              // stages filled with weights while the kernel before drains
    if (warp == 0 && lane == 0)
        for (int kb = 0; kb < early; kb++) load_w(blockIdx.x, kb, kb);
    __syncwarp();
    pdl_wait();
    pdl_trigger();
    if (g.advance != nullptr && blockIdx.x == 0 && threadIdx.x == 64) *g.advance += 1;

    if (warp == 0) {
        if (lane == 0) {
            int st = 0; uint32_t ph = 1;
            bool ok = true;
            for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
                for (int kb = 0; kb < g.num_kb; kb++) {
                    if (kb >= early) {
                        ok = mbar_wait_relaxed(&empty[st], ph, abort_flag, g.status, 0x930);
                        if (!ok) break;
                        load_w(tile, kb, st);
                    }
                    tma_load_2d(smem + st * stage_bytes + W_BYTES, &tmX, &full[st], kb * BK, 0);       // box {64 k, nb rows}
                    if (++st == g.stages) { st = 0; ph ^= 1; }
                }
                early = 0;
            }
        }
    } else if (warp == 1) {
        const bool leader = elect_one();
        const uint32_t idesc = umma_idesc_bf16(WR, 0, 0, 0) | ((uint32_t)(g.nb >> 3) << 17);
        int st = 0; uint32_t ph = 0;
        int it = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x, it++) {
            const int buf = it & 1;
            ok = __all_sync(0xffffffffu, mbar_wait_relaxed(&acc_empty[buf], ((it >> 1) & 1) ^ 1, abort_flag, g.status, 0x938)) != 0;
            for (int kb = 0; kb < g.num_kb && ok; kb++) {
                ok = __all_sync(0xffffffffu, mbar_wait_relaxed(&full[st], ph, abort_flag, g.status, 0x931)) != 0;
                if (!ok) break;
                tc_fence_after();
                const uint64_t dw = umma_desc_sw128(smem_u32(smem + st * stage_bytes), 16, 1024);
                const uint64_t dx = umma_desc_sw128(smem_u32(smem + st * stage_bytes + W_BYTES), 16, 1024);
                if (leader) {
                    #pragma unroll
                    for (int kk = 0; kk < BK / 16; kk++) umma_ss(tmem_base + buf * acc_cols, dw + 2 * kk, dx + 2 * kk, idesc, (kb | kk) > 0);
                    umma_commit(&empty[st]);
                    if (kb == g.num_kb - 1) umma_commit(&acc_full[buf]);
                }
                if (++st == g.stages) { st = 0; ph ^= 1; }
            }
        }
    } else {
        int it = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x, it++) {
            const int buf = it & 1;
            ok = mbar_wait_relaxed(&acc_full[buf], (it >> 1) & 1, abort_flag, g.status, 0x932);
            ok = __all_sync(0xffffffffu, ok) != 0;
            tc_fence_after();
            const int n = tile * WR + (warp & 3) * 32 + lane;
            const float bias = g.bias != nullptr && n < g.N ? __bfloat162float(g.bias[n]) : 0.f;
            for (int c = 0; c < g.nb && ok; c += 16) {
                uint32_t v[16];
                tmem_ld16(tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + buf * acc_cols + c, v);
                tmem_ld_wait();
                if (g.out32 != nullptr) {
                    #pragma unroll
                    for (int e = 0; e < 16; e++)
                        if (c + e < g.M && n < g.cols32) g.out32[(size_t)(c + e) * g.cols32 + n] = round_bf16(__uint_as_float(v[e]) + bias);
                } else {
                    #pragma unroll
                    for (int e = 0; e < 16; e++)
                        if (c + e < g.M && n < g.N) g.out[(size_t)(c + e) * g.ldo + n] = __float2bfloat16_rn(__uint_as_float(v[e]) + bias);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[buf]);
        }
    }
    __syncthreads();
    // after an abandoned wait copies may still be on their way into this CTA's shared memory: give them time to land before it is freed
    if (*abort_flag) {
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000ll) { __nanosleep(1000); }
    }
    __syncthreads();
    tc_fence_after();
    if (warp == 1) tmem_dealloc(tmem_base, 2 * acc_cols);
}

// CTAs per weight tile: as many as are resident at once and have some K blocks each; the wider the tile, the more blocks a slice must have to
// be worth its share of the reduction.  A cluster lives in one GPC, so an eighth of the SMs is not counted on: 36 clusters of 4 on 148 SMs ran
// in two waves.
int pick_split(int tiles, int num_kb, int nb, int sms) {
    const int slots = (nb <= 128 ? 2 : 1) * (sms * 7 / 8), min_kb = nb <= 128 ? 4 : 8;
    int s = 1;
    while (s < MAX_SPLIT && tiles * s * 2 <= slots && num_kb >= s * 2 * min_kb) s *= 2;
    return s;
}

// How a product is cut: row tiles of nb rows, K in S slices.
struct Plan { int nb, mtiles, S; };
int rows_of(int M, int mtiles) { return (CEIL_DIV(M, mtiles) + 15) & ~15; }       // M spread evenly over its tiles

Plan wide_plan(int M, int tiles, int num_kb, int sms) {
    const int nb = rows_of(M, CEIL_DIV(M, MAX_NB)), mtiles = CEIL_DIV(M, nb);
    return {nb, mtiles, pick_split(tiles * mtiles, num_kb, nb, sms)};
}

// Input gradients of more than 128 rows, and forward products cut like them: tiles of about 64 rows (48 at M = 129) or more, as many as leave room for four slices of K each, or as few as
// the 256 rows of a tile allow.  With the small ones a CTA's share of the reduction and its set-up are short; with the large ones fewer CTAs read the same
// weights and K can be cut into more slices.  So shallow products take the small ones and deep ones the large ones.  Estimated in ns from the k-blocks of
// a slice and the rows of a tile, coefficients fitted to 536 products (M 129 to 1024, N 384 to 4096, K 768 to 128256, each way of cutting), 5 and 8 %
// rms off; the way taken is at most 9 % behind the other, by more than 3 % in 16 of them.  CTAs of small tiles take longer where two share an SM; 15 clusters of 8 large tiles fit
// the chip at once, 16 do not.  us, small / large tiles: 256 x 768 x 768 5.0 / 9.3, 256 x 768 x 3072 7.9 / 12.5, 1024 x 768 x 3072 11.7 / 13.3,
// 384 x 768 x 6144 14.9 / 13.1, 256 x 1600 x 14336 27.5 / 21.9, 512 x 2048 x 14336 33 / 31, 384 x 768 x 50304 79 / 43, 512 x 2048 x 128256 304 / 245,
// but 256 x 2048 x 14336 28 / 40 (16 clusters of 8).  Forward products of K = 6144 and more take small tiles only where the estimate is 4 % ahead: 269 x 448 x 14208 16.5 /
// 15.6, 521 x 1152 x 7360 17.7 / 17.2 with estimates 3 and 2 % ahead, 561 x 1024 x 6336 16.1 / 16.3 with 7 %; 15 clusters 641 x 576 x 6784 15.6 / 13.5.
Plan gradient_plan(int M, int tiles, int num_kb, int sms, bool forward) {
    const int slots = 2 * (sms * 7 / 8);
    const Plan wide = wide_plan(M, tiles, num_kb, sms);
    int t = CEIL_DIV(M, 64);
    while (t > 1 && tiles * t * 4 > slots) t--;
    if (CEIL_DIV(M, t) > 128) return wide;
    int S = 1;
    while (S < 4 && num_kb >= S * 2 * 3) S *= 2;
    if (S == 4 && tiles * t * 8 <= slots && num_kb >= 48) S = 8;
    Plan narrow = {rows_of(M, t), 0, S};
    narrow.mtiles = CEIL_DIV(M, narrow.nb);
    const long long kb_n = CEIL_DIV(num_kb, S), kb_w = CEIL_DIV(num_kb, wide.S);
    const bool shared_sms = tiles * narrow.mtiles * S > sms * 7 / 8;
    const long long cost_n = kb_n * (295 + (shared_sms ? 63 + narrow.nb * 87 / 100 : 0)) + 44 * narrow.nb + 2300;
    const int rounds = wide.S == 8 && tiles * wide.mtiles * 19 > 2 * sms ? 2 : 1;
    const long long cost_w = rounds * (kb_w * (297 + wide.nb * 31 / 100) + 24 * wide.nb + 4200);
    return cost_n + (forward && num_kb >= 96 ? cost_n / 25 : 0) <= cost_w ? narrow : wide;
}

// form: 0 a forward product, 1 an input gradient, 2 a forward product cut like one
Plan make_plan(int M, int N, int K, bool swiglu, int form) {
    int sms = llmc_device_sm_count(); if (sms <= 0) sms = 148;
    const int tiles = CEIL_DIV(N, swiglu ? WR / 2 : WR), num_kb = CEIL_DIV(K, BK);
    return form && M > 128 ? gradient_plan(M, tiles, num_kb, sms, form == 2) : wide_plan(M, tiles, num_kb, sms);
}

template <int MODE, bool W_MN>
int launch_stream(bf16* out, const bf16* x, const bf16* w, const bf16* bias, int M, int N, int K, int ldx, int ldw, int ldo, int early_w, cudaStream_t stream,
                  bool sliced = false, float* out32 = nullptr, int cols32 = 0, int* advance = nullptr) {
    if (M <= 0 || N <= 0 || K <= 0 || (K % 8) || (ldx % 8) || (ldw % 8) || ldx < K || ldw < (W_MN ? N : K) || ldo < N) return -1;
    if (W_MN && (N % 8)) return -1;
    Args g;
    g.early_w = early_w;
    g.out32 = out32; g.cols32 = cols32; g.advance = advance;
    g.out = out; g.bias = bias; g.w = w; g.M = M; g.N = N; g.K = K; g.ldo = ldo; g.ldw = ldw;
    const Plan plan = make_plan(M, N, K, MODE == SWIGLU, W_MN ? 1 : sliced ? 2 : 0);
    const int tiles = CEIL_DIV(N, MODE == SWIGLU ? WR / 2 : WR), mtiles = plan.mtiles, S = plan.S;
    int sms = llmc_device_sm_count(); if (sms <= 0) sms = 148;
    g.nb = plan.nb;
    g.num_kb = CEIL_DIV(K, BK);
    const int stage_bytes = W_BYTES + g.nb * (BK * 2);
    const bool two = g.nb <= 128;
    g.stages = ((two ? SMEM_TWO : SMEM_ONE) - 2048) / stage_bytes;
    if (g.stages > MAX_STAGES) g.stages = MAX_STAGES;
    g.vec_out = (ldo % 4 == 0) && (reinterpret_cast<uintptr_t>(out) & 7) == 0;
    g.status = llmc_status_ptr();
    CUtensorMap tmW, tmX;
    {
        uint64_t dims[2] = {(uint64_t)K, (uint64_t)(MODE == SWIGLU ? 2 * (uint64_t)N : (uint64_t)N)};
        uint32_t box[2] = {BK, MODE == SWIGLU ? WR / 2 : WR};
        if (W_MN) { dims[0] = (uint64_t)N; dims[1] = (uint64_t)K; box[0] = 64; box[1] = BK; }
        uint64_t strides[2] = {2, (uint64_t)ldw * 2};
        int rc = llmc_get_tensormap(&tmW, w, 2, 2, dims, strides, box, 3);
        if (rc) return rc;
        uint64_t dimx[2] = {(uint64_t)K, (uint64_t)M};
        uint64_t strx[2] = {2, (uint64_t)ldx * 2};
        uint32_t boxx[2] = {BK, (uint32_t)g.nb};
        rc = llmc_get_tensormap(&tmX, x, 2, 2, dimx, strx, boxx, 3);
        if (rc) return rc;
    }
    if (MODE == STORE && !W_MN && mtiles == 1 && two && tiles > 2 * sms) {
        static bool configured_wide = false;
        const int smem = g.stages * stage_bytes + 1024 + 256;
        if (!configured_wide) {
            CUDA_CHECK(cudaFuncSetAttribute(stream_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_TWO));
            configured_wide = true;
        }
        CUDA_CHECK(launch_pdl(stream_wide_kernel, dim3(2 * sms), dim3(THREADS), smem, stream, 0, tmW, tmX, g));
        return 0;
    }
    g.kb_per_split = CEIL_DIV(g.num_kb, S);
    const int smem = g.stages * stage_bytes + 1024 + 256;
    static bool configured = false;
    if (!configured) {
        CUDA_CHECK(cudaFuncSetAttribute(stream_gemm_kernel<MODE, W_MN>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_ONE));
        configured = true;
    }
    CUDA_CHECK(launch_pdl(stream_gemm_kernel<MODE, W_MN>, dim3(tiles * S, mtiles), dim3(THREADS), smem, stream, S, tmW, tmX, g));
    return 0;
}

}  // namespace

// How a plain product of these sizes is cut
extern "C" void llmc_stream_gemm_plan(int M, int N, int K, int form, int* rows, int* slices) {
    const Plan p = make_plan(M, N, K, false, form);
    *rows = p.nb; *slices = p.S;
}

// out (M, N) = x (M, K) . w (N, K)^T (+ bias), form 0 or 2 (make_plan), or x . w (K, N), form 1.  K, the row strides of x and w and, in form 1, N are multiples of 8.
extern "C" int llmc_stream_gemm(bf16* out, const bf16* x, const bf16* w, const bf16* bias, int M, int N, int K, int ldx, int ldw, int ldo, int form,
                                cudaStream_t stream) {
    if (M <= 0 || N <= 0 || K <= 0) return 0;        // an empty product leaves out as it is, like the other two kernels'
    if (form == 1) return launch_stream<STORE, true>(out, x, w, bias, M, N, K, ldx, ldw, ldo, 0, stream);
    return launch_stream<STORE, false>(out, x, w, bias, M, N, K, ldx, ldw, ldo, 0, stream, form == 2);
}

// The same behind a kernel that does not write w (csrc/decoder.cu): an early launch fills the stages with weights while that kernel drains.  What other
// kernels before it wrote is complete: it triggers the launch after its own wait (pdl.cuh).
extern "C" int llmc_stream_gemm_chained(bf16* out, const bf16* x, const bf16* w, int M, int N, int K, int ldx, int ldw, int ldo, int form,
                                        cudaStream_t stream) {
    if (M <= 0 || N <= 0 || K <= 0) return 0;
    return launch_stream<STORE, false>(out, x, w, nullptr, M, N, K, ldx, ldw, ldo, 1, stream, form == 2);
}

// out (M, N) = (x . w1^T) * silu(x . w2^T) with w = [w1; w2] of 2 N rows, M <= 128; N a multiple of 64
extern "C" int llmc_stream_gemm_swiglu(bf16* out, const bf16* x, const bf16* w, int M, int N, int K, int ldx, int ldw, int ldo, cudaStream_t stream) {
    if (N % 64 || M > 128) return -1;
    return launch_stream<SWIGLU, false>(out, x, w, nullptr, M, N, K, ldx, ldw, ldo, 0, stream);
}
extern "C" int llmc_stream_gemm_swiglu_chained(bf16* out, const bf16* x, const bf16* w, int M, int N, int K, int ldx, int ldw, int ldo, cudaStream_t stream) {
    if (N % 64 || M > 128) return -1;
    return launch_stream<SWIGLU, false>(out, x, w, nullptr, M, N, K, ldx, ldw, ldo, 1, stream);
}

// The last product of a decoding pass: its bf16 results as fp32, the first `cols` columns in rows of as many, and, where a counter is given, 1 added to it (the
// position of a replayed step).  In launches of their own the conversion and the addition took 7 us of a step of 4 rows and 15 of one of 32 (128256 columns).
extern "C" int llmc_stream_gemm_logits(float* out, int cols, const bf16* x, const bf16* w, int M, int N, int K, int ldx, int ldw, int* advance, cudaStream_t stream) {
    if (M <= 0 || N <= 0 || K <= 0 || cols <= 0 || cols > N) return -1;
    return launch_stream<STORE, false>(nullptr, x, w, nullptr, M, N, K, ldx, ldw, N, 1, stream, false, out, cols, advance);
}
