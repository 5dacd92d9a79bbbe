// Causal flash attention backward for sm_100a on the packed (B, T, 3, NH, HS) layout, head sizes 72..128 (multiples of 8; a
// narrower head runs as a 128-wide one whose missing channels TMA fills with zeros, with the products cut to whole 16-channel steps).
//
// Deterministic by construction: no atomics, every output element has one writer and a fixed summation order.  Three launches:
//   1. delta[b,h,t] = sum_d O[b,t,h,d] * dO[b,t,h,d]
//   2. dK / dV: the key tile (K_j, V_j) stays in shared memory, the query tiles i >= j stream past it.  The score tiles are formed
//      TRANSPOSED (keys on the TMEM lanes): S^T = K Q^T, dP^T = V dO^T, so that P^T and dS^T, written back to tensor memory as
//      bf16 over the scores they came from, are the A operands of dV += P^T dO and dK += dS^T Q.
//   3. dQ: the query tile (Q_i, dO_i) stays, the key tiles j <= i stream; S = Q K^T, dP = dO V^T, dQ += dS K_j with dS in TMEM.
//
// Why two passes with S and dP formed twice and not one: with 128 channels a tile pair's dQ contribution is 64 KB of fp32.  Summing
// these in a fixed order through memory (what attention_bwd1.cu does at 64 channels) would write and read them at the rate of
// HBM, which takes longer than the two extra products; and dV, dK, dQ and both score tiles together do not fit 512 TMEM columns.
// Neither holds at 72 and 80 channels (2 x 128 + 3 x 80 = 496 columns, 40 KB a pair): one pass is possible there and is not built.
//
// Both passes are bound by the softmax warps (16 exponentials per clock and SM: 1024 cycles for a 128 x 128 tile, plus the TMEM
// loads and stores around them) with the tensor pipe close behind (2048 / 1536 cycles a pair).  So nothing but that is left to the
// softmax warps: no operand goes through shared memory (the kernel this one replaces staged P and dS there, with one stage of
// streamed tiles), S of the next pair is issued before dS of this one is finished, the outputs leave through four warps of
// their own.  All three launches, the kernels before these in brackets: B=16 T=2048 NH=8 HS=128 509 us (978), B=2 T=4096 NH=32 HS=128
// 855 us (1723), B=3 T=1000 NH=32 HS=80 112 us (235); 521 / 880 / 113 with scalar instead of paired fp32 arithmetic in the softmax.
//
// Work items are one fixed tile of one head, heaviest first, dealt to the persistent CTAs in alternating direction (CTA c gets items
// c, 2G-1-c, 2G+c, ...), which evens out the decreasing sizes; a plain round-robin gives CTA 0 the longest item of every round.
//
// Roles inside a CTA (512 threads):
//   warp 0       TMA producer (fixed tiles single-buffered, each of the two released by the last product that reads it, one pair
//                before the item ends; X0, which a pair needs from its first product to its last, in a ring of three, X1, which is
//                free again by the middle of its pair, in one buffer: with both in a two-stage ring S waited for loads)
//   warp 1       issuer of the products; program order keeps a score tile from overwriting the bf16 operand that aliases it
//   warps 4-11   softmax: thread = row of the score tile x 64-column half
//   warps 12-15  drain: accumulators -> bf16 -> shared memory -> TMA store; in the dK / dV pass also the per-query statistics table
//
// TMEM columns: S [0,128) (P^T bf16 in the first 32 columns of each half)   dP [128,256) (dS bf16 likewise)
//               dK/dV pass: dV [256,384) dK [384,512)      dQ pass: dQ [256,384), second S buffer [384,512)
//
// Capability parity: attention_backward_cudnn (llmc/cudnn_att.cpp:256-288) and attention_backward of llmc/attention.cuh in the
// reference, which also demands reproducible gradients of cuDNN (llmc/cudnn_att.cpp:186-191).
#include "common.cuh"

int llmc_attn_qkv_map(CUtensorMap* tm, const bf16* qkv, int B, int T, int NH, int hs, int rows);   // attention_fwd.cu

namespace {

constexpr int BT = 128;                             // tile rows (queries and keys)
constexpr int CHUNK_BYTES = BT * 64 * 2;            // 16 KB: 128 rows x 64 channels, one 128-byte-swizzled TMA box
constexpr int TILE_BYTES = 2 * CHUNK_BYTES;
constexpr int X0STAGES = 3;                         // ring of the streamed tiles X0; X1 has one buffer
constexpr int THREADS = 512;
constexpr int TMEM_COLS = 512;
constexpr int STAT_BYTES = 2 * 2 * BT * 4;          // [2 buffers][lse, delta][128 queries]
constexpr int SMEM = 2 * TILE_BYTES + (X0STAGES + 1) * TILE_BYTES + TILE_BYTES + STAT_BYTES + 256;
static_assert(SMEM <= 232448, "shared memory of one CTA");

struct Args {
    const float* lse;    // (B, NH, T)
    const float* delta;  // (B, NH, T)
    int T, NH, BH;
    int ks;              // 16-channel steps of the head: ceil(hs / 16)
    float scale, scale_log2e;
    unsigned int* status;
};

// delta: 8 lanes per (b, t, h) row of hs channels, CH 16-byte pieces of it each at most; narrow heads take two rows per thread.  Bound by memory.  us, the 64-bit
// divisions, blocks of 256 threads and one row per thread of before in brackets: 64 x 1024 x 12 heads of 64 30.2 (43.6; 35.4 with one row, 34.4 with four), 3 x 1000 x 32 x 80
// 7.3 (8.9; 7.6 with two rows), 2 x 4096 x 32 x 128 19.9 (23.6; 21.0).  With sums collected in shared memory, so that tokens of a head leave together, 57 to 130.
constexpr int DELTA_THREADS = 128;
__host__ __device__ constexpr int delta_rows(int ch) { return ch == 1 ? 2 : 1; }
template <int CH>
__global__ void __launch_bounds__(DELTA_THREADS)
delta_kernel(float* __restrict__ delta, const bf16* __restrict__ out, const bf16* __restrict__ dout,
             unsigned rows, unsigned T, unsigned NH, int hs) {
    constexpr int ROWS = delta_rows(CH), GROUPS = DELTA_THREADS / 8;
    const int part = threadIdx.x & 7;
    const unsigned row0 = blockIdx.x * (GROUPS * ROWS) + (threadIdx.x >> 3);
    bf16x8 o[ROWS][CH], d[ROWS][CH];
    #pragma unroll
    for (int k = 0; k < ROWS; k++) {
        const unsigned row = min(row0 + k * GROUPS, rows - 1);
        const size_t at = (size_t)row * hs;
        #pragma unroll
        for (int i = 0; i < CH; i++) {
            const int p = part + 8 * i;
            if (i == 0 || p < (hs >> 3)) { o[k][i] = ld128cs(out + at + p * 8); d[k][i] = ld128cs(dout + at + p * 8); }
        }
    }
    #pragma unroll
    for (int k = 0; k < ROWS; k++) {
        const unsigned row = row0 + k * GROUPS;
        float acc = 0.f;
        #pragma unroll
        for (int i = 0; i < CH; i++)
            if (i == 0 || part + 8 * i < (hs >> 3)) {
                #pragma unroll
                for (int e = 0; e < 8; e++) acc += __bfloat162float(o[k][i][e]) * __bfloat162float(d[k][i][e]);
            }
        acc += __shfl_xor_sync(0xffffffffu, acc, 1);
        acc += __shfl_xor_sync(0xffffffffu, acc, 2);
        acc += __shfl_xor_sync(0xffffffffu, acc, 4);
        if (row < rows && part == 0) {
            const unsigned bt = row / NH, h = row - bt * NH, b = bt / T, t = bt - b * T;
            delta[((size_t)b * NH + h) * T + t] = acc;
        }
    }
}

DEVINL void tmem_st8(uint32_t taddr, const uint32_t* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}

// The sequence of tile pairs of one CTA.  f: the item's fixed tile (key tile in the dK / dV pass, query tile in the dQ pass),
// x: the streamed tile, x0..x1 its range.
template <bool DKV>
struct Walk {
    int round, cta, grid, total, BH, nt, NH;
    int w, bh, b, h, f, x, x0, x1;
    DEVINL void start(int cta_, int grid_, int BH_, int nt_, int NH_) {
        cta = cta_; grid = grid_; BH = BH_; nt = nt_; NH = NH_; total = BH_ * nt_; round = 0;
        bh = b = h = f = x = x0 = x1 = 0;
        w = cta;
        if (w < total) item();
    }
    DEVINL bool valid() const { return w < total; }
    DEVINL void item() {
        const int rank = w / BH;
        bh = w - rank * BH; b = bh / NH; h = bh - b * NH;
        if (DKV) { f = rank; x0 = f; x1 = nt - 1; }
        else { f = nt - 1 - rank; x0 = 0; x1 = f; }
        x = x0;
    }
    DEVINL bool first() const { return x == x0; }
    DEVINL bool last() const { return x == x1; }
    DEVINL void next() {                      // valid() turns false past the last pair
        if (++x <= x1) return;
        round++;
        w = round * grid + ((round & 1) ? grid - 1 - cta : cta);
        if (w < total) item();
    }
};

template <bool DKV>
__global__ void __launch_bounds__(THREADS, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tmQKV, const __grid_constant__ CUtensorMap tmDO,
                const __grid_constant__ CUtensorMap tmDQKV, const Args a) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sF = smem;                                // fixed tiles F0 (K_j / Q_i), F1 (V_j / dO_i)
    uint8_t* sX0 = sF + 2 * TILE_BYTES;                // [X0STAGES] streamed tiles X0 (Q_i / K_j)
    uint8_t* sX1 = sX0 + X0STAGES * TILE_BYTES;        // streamed tile X1 (dO_i / V_j)
    uint8_t* sOut = sX1 + TILE_BYTES;                  // an accumulator tile on its way out (two TMA boxes)
    float* sStat = reinterpret_cast<float*>(sOut + TILE_BYTES);     // [2][2][128]
    uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(sStat) + STAT_BYTES);
    uint64_t* f_full = bars + 0;      // [F0, F1]
    uint64_t* f_empty = bars + 2;     // [F0, F1]
    uint64_t* x0_full = bars + 21;    // [3]
    uint64_t* x0_empty = bars + 24;   // [3]
    uint64_t* x1_full = bars + 4;
    uint64_t* x1_empty = bars + 5;
    uint64_t* s_full = bars + 8;      // [2] S(t) complete, t & 1                           (1 commit)
    uint64_t* dp_full = bars + 10;    // dP(t) complete                                     (1 commit)
    uint64_t* p_ready = bars + 11;    // P^T(t) is in TMEM                                  (8 arrivals)
    uint64_t* ds_ready = bars + 12;   // dS(t) is in TMEM, S(t) has been read               (8 arrivals)
    uint64_t* acc_full = bars + 13;   // [2] accumulator of the item complete               (1 commit)
    uint64_t* acc_empty = bars + 15;  // [2] the drain warps have read it                   (4 arrivals)
    uint64_t* st_full = bars + 17;    // [2] statistics table of a pair written             (4 arrivals)
    uint64_t* st_empty = bars + 19;   // [2] ... and read by every softmax warp             (8 arrivals)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 27);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const int nt = CEIL_DIV(a.T, BT);

    if (threadIdx.x == 0) {
        if ((smem_u32(smem) & 1023u) != 0) record_error(a.status, ST_BAD_ARG, 0x28);
        for (int i = 0; i < 2; i++) {
            mbar_init(&f_full[i], 1); mbar_init(&f_empty[i], 1); mbar_init(&s_full[i], 1);
            mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], 4); mbar_init(&st_full[i], 4); mbar_init(&st_empty[i], 8);
        }
        for (int i = 0; i < X0STAGES; i++) { mbar_init(&x0_full[i], 1); mbar_init(&x0_empty[i], 1); }
        mbar_init(x1_full, 1); mbar_init(x1_empty, 1); mbar_init(dp_full, 1); mbar_init(p_ready, 8); mbar_init(ds_ready, 8);
        *abort_flag = 0;
        mbar_fence_init();
        tma_prefetch_desc(&tmQKV); tma_prefetch_desc(&tmDO); tma_prefetch_desc(&tmDQKV);
    }
    if (warp == 1) { tmem_alloc(tmem_slot, TMEM_COLS); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tS = tmem_base, tdP = tmem_base + 128, tAcc0 = tmem_base + 256, tAcc1 = tmem_base + 384;
    constexpr uint32_t S_BUF = DKV ? 0 : 384;           // distance of the second S buffer (the dK / dV pass has one)

    Walk<DKV> wk;
    wk.start(blockIdx.x, gridDim.x, a.BH, nt, a.NH);

    if (warp == 0) {
        // ---------------------------------------------------------------- TMA producer
        if (lane == 0) {
            auto load = [&](uint8_t* dst, const CUtensorMap* tm, uint64_t* bar, int head, int tile, int b) {
                tma_load_4d(dst, tm, bar, 0, head, tile * BT, b);
                tma_load_4d(dst + CHUNK_BYTES, tm, bar, 64, head, tile * BT, b);
            };
            uint32_t t = 0;
            int item = 0;
            for (; wk.valid(); wk.next(), t++) {
                if (wk.first()) {
                    if (!mbar_wait_relaxed(&f_empty[0], (item & 1) ^ 1, abort_flag, a.status, 0x681)) break;
                    mbar_expect_tx(&f_full[0], TILE_BYTES);
                    load(sF, &tmQKV, &f_full[0], DKV ? a.NH + wk.h : wk.h, wk.f, wk.b);
                    if (!mbar_wait_relaxed(&f_empty[1], (item & 1) ^ 1, abort_flag, a.status, 0x682)) break;
                    mbar_expect_tx(&f_full[1], TILE_BYTES);
                    load(sF + TILE_BYTES, DKV ? &tmQKV : &tmDO, &f_full[1], DKV ? 2 * a.NH + wk.h : wk.h, wk.f, wk.b);
                    item++;
                }
                const uint32_t st = t % X0STAGES;
                if (!mbar_wait_relaxed(&x0_empty[st], ((t / X0STAGES) & 1) ^ 1, abort_flag, a.status, 0x680)) break;
                mbar_expect_tx(&x0_full[st], TILE_BYTES);
                load(sX0 + st * TILE_BYTES, &tmQKV, &x0_full[st], DKV ? wk.h : a.NH + wk.h, wk.x, wk.b);
                if (!mbar_wait_relaxed(x1_empty, (t & 1) ^ 1, abort_flag, a.status, 0x683)) break;
                mbar_expect_tx(x1_full, TILE_BYTES);
                load(sX1, DKV ? &tmDO : &tmQKV, x1_full, DKV ? wk.h : 2 * a.NH + wk.h, wk.x, wk.b);
            }
        }
    } else if (warp == 1) {
        // ---------------------------------------------------------------- issuer: the whole warp in uniform control flow, one elected
        // lane executes the tcgen05 instructions; wait results go through a warp vote so that the branches on them are uniform
        if (wk.valid()) {
            const bool leader = elect_one();
#define WAIT_ALL(bar, parity, code) (__all_sync(0xffffffffu, mbar_wait_relaxed(bar, parity, abort_flag, a.status, code)) != 0)
            constexpr uint32_t idesc_s = umma_idesc_bf16(BT, BT, 0, 0);                // both operands K-major
            const uint32_t idesc_acc = umma_idesc_bf16(BT, 0, 0, 1) | ((uint32_t)(a.ks * 2) << 17);      // A from TMEM, B N-major, N = 16 ks
            constexpr uint32_t TILE_UNITS = TILE_BYTES / 16, CHUNK_UNITS = CHUNK_BYTES / 16;
            const uint64_t dF0 = umma_desc_sw128(smem_u32(sF), 16, 1024), dF1 = umma_desc_sw128(smem_u32(sF + TILE_BYTES), 16, 1024);
            const uint64_t dX0 = umma_desc_sw128(smem_u32(sX0), 16, 1024), dX1 = umma_desc_sw128(smem_u32(sX1), 16, 1024);
            const uint64_t nX0 = umma_desc_sw128(smem_u32(sX0), CHUNK_BYTES, 1024), nX1 = umma_desc_sw128(smem_u32(sX1), CHUNK_BYTES, 1024);
            const int ks = a.ks;
            // score product: 16 channels = 32 bytes = 2 address units per step, 4 steps per 64-channel chunk
            auto issue_score = [&](uint32_t d, uint64_t f, uint64_t x, uint64_t* bar) {
                if (leader) {
                    #pragma unroll
                    for (int kk = 0; kk < 8; kk++)
                        if (kk < ks) umma_ss(d, f + (kk >> 2) * CHUNK_UNITS + (kk & 3) * 2, x + (kk >> 2) * CHUNK_UNITS + (kk & 3) * 2, idesc_s, kk > 0);
                    umma_commit(bar);
                }
            };
            // accumulating product: A = bf16 operand over its score tile (16 rows of B = 8 columns per step, each 64-row half at its own half
            // of the tile), B = streamed tile N-major (16 rows = 2048 bytes = 128 units per step)
            auto issue_acc = [&](uint32_t d, uint32_t ta, uint64_t x, uint32_t acc) {
                if (leader) {
                    #pragma unroll
                    for (int kk = 0; kk < BT / 16; kk++) umma_ts(d, ta + (kk >> 2) * 64 + (kk & 3) * 8, x + 128 * kk, idesc_acc, acc | (kk > 0));
                }
            };
            uint32_t t = 0;
            int item = 0;              // item of pair t
            bool ok = WAIT_ALL(&f_full[0], 0, 0x690) && WAIT_ALL(&x0_full[0], 0, 0x691);
            tc_fence_after();
            if (ok) { issue_score(tS, dF0, dX0, &s_full[0]); if (leader && wk.last()) umma_commit(&f_empty[0]); }
            ok = ok && WAIT_ALL(&f_full[1], 0, 0x692) && WAIT_ALL(x1_full, 0, 0x692);
            tc_fence_after();
            if (ok) {
                issue_score(tdP, dF1, dX1, dp_full);
                if (leader && !DKV) umma_commit(x1_empty);
                if (leader && wk.last()) umma_commit(&f_empty[1]);
            }
            while (ok) {
                Walk<DKV> nx = wk; nx.next();
                const bool have_next = nx.valid();
                const uint32_t st = t % X0STAGES, nst = (t + 1) % X0STAGES, sb = (t + 1) & 1;
                const uint64_t xo = (uint64_t)(st * TILE_UNITS), nxo = (uint64_t)(nst * TILE_UNITS);
                const int nitem = have_next && nx.first() ? item + 1 : item;
                const uint32_t acc = wk.first() ? 0u : 1u;
                if (DKV) {
                    // ---- dV(t) += P^T dO_i
                    ok = WAIT_ALL(p_ready, t & 1, 0x693);
                    if (ok && wk.first() && item > 0) ok = WAIT_ALL(&acc_empty[0], (item - 1) & 1, 0x694);
                    if (!ok) break;
                    tc_fence_after();
                    issue_acc(tAcc0, tS, nX1, acc);
                    if (leader) {
                        umma_commit(x1_empty);
                        if (wk.last()) umma_commit(&acc_full[0]);
                    }
                }
                // ---- S(t+1): into the tile P^T(t) was read from just before (dK / dV pass), or into the other S buffer, which the
                //      softmax warps have read before they announced dS(t-1)
                if (have_next) {
                    if (nx.first()) ok = WAIT_ALL(&f_full[0], nitem & 1, 0x695);
                    ok = ok && WAIT_ALL(&x0_full[nst], ((t + 1) / X0STAGES) & 1, 0x696);
                    if (!ok) break;
                    tc_fence_after();
                    issue_score(tS + sb * S_BUF, dF0, dX0 + nxo, &s_full[sb]);
                    if (leader && nx.last()) umma_commit(&f_empty[0]);
                }
                // ---- dK(t) += dS^T Q_i   or   dQ(t) += dS K_j
                ok = WAIT_ALL(ds_ready, t & 1, 0x697);
                if (ok && wk.first() && item > 0) ok = WAIT_ALL(&acc_empty[DKV ? 1 : 0], (item - 1) & 1, 0x698);
                if (!ok) break;
                tc_fence_after();
                issue_acc(DKV ? tAcc1 : tAcc0, tdP, nX0 + xo, acc);
                if (leader) {
                    umma_commit(&x0_empty[st]);
                    if (wk.last()) umma_commit(&acc_full[DKV ? 1 : 0]);
                }
                // ---- dP(t+1): after the product above in program order, so it cannot overwrite dS(t) early
                if (have_next) {
                    if (nx.first()) ok = WAIT_ALL(&f_full[1], nitem & 1, 0x699);
                    ok = ok && WAIT_ALL(x1_full, (t + 1) & 1, 0x69a);
                    if (!ok) break;
                    tc_fence_after();
                    issue_score(tdP, dF1, dX1, dp_full);
                    if (leader) {
                        if (!DKV) umma_commit(x1_empty);
                        if (nx.last()) umma_commit(&f_empty[1]);
                    }
                }
                if (!have_next) break;
                wk = nx; item = nitem; t++;
            }
#undef WAIT_ALL
        }
    } else if (warp >= 4 && warp < 12) {
        // ---------------------------------------------------------------- softmax: thread = row r of the score tile x column half hf
        const int q = warp & 3;                        // TMEM lane quarter
        const int hf = (warp - 4) >> 2;
        const int r = q * 32 + lane;
        const uint32_t lane_off = (uint32_t)(q * 32) << 16;
        const float log2e = 1.4426950408889634f;
        bool ok = true;
        uint32_t t = 0;
        float row_lse = 0.f, row_delta = 0.f;          // dQ pass: statistics of this thread's query row, negated like those of the table
        const uint64_t sl2 = f2_pack(a.scale_log2e, a.scale_log2e), sc2 = f2_pack(a.scale, a.scale);
        for (; wk.valid(); wk.next(), t++) {
            const bool diag = wk.x == wk.f;
            const float* stat = sStat + (t & 1) * (2 * BT) + hf * 64;       // dK / dV pass: -lse * log2(e) of this half's queries; -delta * scale 128 floats further
            if (!DKV && wk.first()) {
                const int tq = wk.f * BT + r;
                row_lse = -INFINITY; row_delta = 0.f;
                if (tq < a.T) { row_lse = -(a.lse[(size_t)wk.bh * a.T + tq] * log2e); row_delta = -(a.delta[(size_t)wk.bh * a.T + tq] * a.scale); }
            }
            ok = mbar_wait(&s_full[t & 1], (t >> 1) & 1, abort_flag, a.status, 0x6a0) && ok;
            if (DKV) ok = mbar_wait(&st_full[t & 1], (t >> 1) & 1, abort_flag, a.status, 0x6a1) && ok;
            tc_fence_after();
            // ---- P = exp2(S * scale * log2(e) - LSE * log2(e)), causal, in two passes of 32 columns (with all 64 scores next to the 64
            //      results the register file is so full that every exponential waits for its predecessor)
            const uint32_t tSt = tS + (DKV ? 0u : (t & 1) * S_BUF) + lane_off + hf * 64;
            float p[64];
            #pragma unroll
            for (int h2 = 0; h2 < 2; h2++) {
                uint32_t sv[32];
                tmem_ld32(tSt + h2 * 32, sv);
                tmem_ld_wait();
                #pragma unroll
                for (int e4 = 0; e4 < 8; e4++) {
                    float4 l4 = make_float4(row_lse, row_lse, row_lse, row_lse);
                    if (DKV) l4 = *reinterpret_cast<const float4*>(stat + h2 * 32 + e4 * 4);
                    const float2 x0 = f2_unpack(f2_fma(f2_pack_u(sv[e4 * 4 + 0], sv[e4 * 4 + 1]), sl2, f2_pack(l4.x, l4.y)));
                    const float2 x1 = f2_unpack(f2_fma(f2_pack_u(sv[e4 * 4 + 2], sv[e4 * 4 + 3]), sl2, f2_pack(l4.z, l4.w)));
                    p[h2 * 32 + e4 * 4 + 0] = ex2_fast(x0.x); p[h2 * 32 + e4 * 4 + 1] = ex2_fast(x0.y);
                    p[h2 * 32 + e4 * 4 + 2] = ex2_fast(x1.x); p[h2 * 32 + e4 * 4 + 3] = ex2_fast(x1.y);
                }
            }
            // the diagonal tile needs a mask (query >= key).  Keys past T need none beyond it, as no query before T sees them.  Queries past T
            // have LSE = +inf, which leaves 0 except where an infinite key made their zero rows' score NaN.
            if (diag) {
                #pragma unroll
                for (int e = 0; e < 64; e++) if (DKV ? hf * 64 + e < r : hf * 64 + e > r) p[e] = 0.f;
            }
            if (DKV && (wk.x + 1) * BT > a.T) {
                #pragma unroll
                for (int e = 0; e < 64; e++) if (wk.x * BT + hf * 64 + e >= a.T) p[e] = 0.f;
            }
            if (DKV) {
                uint32_t pk[32];
                #pragma unroll
                for (int e = 0; e < 32; e++) pk[e] = pack_bf16x2(p[2 * e], p[2 * e + 1]);
                tmem_st16(tSt, pk);
                tmem_st16(tSt + 16, pk + 16);
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(p_ready);
            }
            // ---- dS = P * (dP * scale - delta * scale), in four chunks of 16 columns: bf16 inside this half's own columns of the dP tile
            //      (a chunk's bf16 lands on fp32 columns that are already in registers)
            ok = mbar_wait(dp_full, t & 1, abort_flag, a.status, 0x6a3) && ok;
            tc_fence_after();
            #pragma unroll
            for (int c = 0; c < 4; c++) {
                uint32_t dv[16];
                tmem_ld16(tdP + lane_off + hf * 64 + c * 16, dv);
                tmem_ld_wait();
                uint32_t dd[8];
                #pragma unroll
                for (int e4 = 0; e4 < 4; e4++) {
                    float4 d4 = make_float4(row_delta, row_delta, row_delta, row_delta);
                    if (DKV) d4 = *reinterpret_cast<const float4*>(stat + BT + c * 16 + e4 * 4);
                    const float* pe = p + c * 16 + e4 * 4;
                    const float2 s0 = f2_unpack(f2_mul(f2_pack(pe[0], pe[1]), f2_fma(f2_pack_u(dv[e4 * 4 + 0], dv[e4 * 4 + 1]), sc2, f2_pack(d4.x, d4.y))));
                    const float2 s1 = f2_unpack(f2_mul(f2_pack(pe[2], pe[3]), f2_fma(f2_pack_u(dv[e4 * 4 + 2], dv[e4 * 4 + 3]), sc2, f2_pack(d4.z, d4.w))));
                    dd[e4 * 2] = pack_bf16x2(s0.x, s0.y);
                    dd[e4 * 2 + 1] = pack_bf16x2(s1.x, s1.y);
                }
                tmem_st8(tdP + lane_off + hf * 64 + c * 8, dd);
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) { mbar_arrive(ds_ready); if (DKV) mbar_arrive(&st_empty[t & 1]); }
        }
    } else if (warp >= 12) {
        // ---------------------------------------------------------------- drain warps (128 threads): thread = row rr of a tile
        const int q = warp & 3;
        const int rr = q * 32 + lane;
        const uint32_t lane_off = (uint32_t)(q * 32) << 16;
        const float log2e = 1.4426950408889634f;
        const bool issuer = warp == 12 && lane == 0;
        bool ok = true;
        bool staged = false;
        uint32_t t = 0;
        int item = 0;
        // dK / dV pass: statistics of query rr of a pair's query tile -> table (tt & 1): LSE in log2 units, delta times the scale;
        // queries past the end of the sequence get LSE = +inf, so that their P^T column is zero
        auto put_stats = [&](const Walk<DKV>& pr, uint32_t tt) {
            const int tq = pr.x * BT + rr;
            float l = INFINITY, d = 0.f;
            if (tq < a.T) { l = a.lse[(size_t)pr.bh * a.T + tq] * log2e; d = a.delta[(size_t)pr.bh * a.T + tq] * a.scale; }
            ok = mbar_wait_relaxed(&st_empty[tt & 1], ((tt >> 1) & 1) ^ 1, abort_flag, a.status, 0x6b0) && ok;
            float* tab = sStat + (tt & 1) * (2 * BT);
            tab[rr] = -l; tab[BT + rr] = -d;
            __syncwarp();
            if (lane == 0) mbar_arrive(&st_full[tt & 1]);
        };
        // accumulator tile -> bf16 in the layout of two 128-byte-swizzled TMA boxes -> bulk stores (rows past T and channels past the
        // head are clipped by TMA); warps writing rows themselves would touch 32 cache lines per instruction
        auto drain = [&](int which, uint32_t tAcc, int head, int f, int b) {
            ok = mbar_wait_relaxed(&acc_full[which], item & 1, abort_flag, a.status, 0x6b2) && ok;
            tc_fence_after();
            if (staged) { if (issuer) tma_store_wait_read<0>(); asm volatile("bar.sync 1, 128;" ::: "memory"); }
            #pragma unroll
            for (int c = 0; c < 4; c++) {
                if (c * 2 < a.ks) {
                    uint32_t v[32];
                    tmem_ld32(tAcc + lane_off + c * 32, v);
                    tmem_ld_wait();
                    uint8_t* orow = sOut + (c >> 1) * CHUNK_BYTES + rr * 128;
                    #pragma unroll
                    for (int u = 0; u < 4; u++) {
                        uint4 o;
                        o.x = pack_bf16x2(__uint_as_float(v[8 * u]), __uint_as_float(v[8 * u + 1]));
                        o.y = pack_bf16x2(__uint_as_float(v[8 * u + 2]), __uint_as_float(v[8 * u + 3]));
                        o.z = pack_bf16x2(__uint_as_float(v[8 * u + 4]), __uint_as_float(v[8 * u + 5]));
                        o.w = pack_bf16x2(__uint_as_float(v[8 * u + 6]), __uint_as_float(v[8 * u + 7]));
                        *reinterpret_cast<uint4*>(orow + ((((c & 1) * 4 + u) ^ (rr & 7)) * 16)) = o;
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[which]);
            fence_async_smem();
            asm volatile("bar.sync 1, 128;" ::: "memory");
            if (issuer && ok) {
                tma_store_4d(&tmDQKV, sOut, 0, head, f * BT, b);
                tma_store_4d(&tmDQKV, sOut + CHUNK_BYTES, 64, head, f * BT, b);
                tma_store_commit();
            }
            staged = true;
        };
        if (DKV && wk.valid()) put_stats(wk, 0);
        for (; wk.valid(); t++) {
            const int b = wk.b, h = wk.h, f = wk.f;
            const bool last = wk.last();
            wk.next();
            if (DKV && wk.valid()) put_stats(wk, t + 1);        // the next pair's table, one pair ahead
            if (last) {
                drain(0, tAcc0, DKV ? 2 * a.NH + h : h, f, b);
                if (DKV) drain(1, tAcc1, a.NH + h, f, b);
                item++;
            }
        }
        if (issuer) tma_store_wait<0>();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (*abort_flag) {
        long long t0 = clock64();
        while (clock64() - t0 < 2000000ll) { __nanosleep(1000); }
        __syncthreads();
    }
    if (warp == 1) tmem_dealloc(tmem_base, TMEM_COLS);
}

}  // namespace

// delta[b,h,t] = sum_d O[b,t,h,d] * dO[b,t,h,d] (shared with the single-pass kernel of attention_bwd1.cu)
int llmc_attention_delta(float* delta, const bf16* out, const bf16* dout, int B, int T, int NH, int hs, cudaStream_t stream) {
    const long long rows = (long long)B * T * NH;
    if (rows > 0xf0000000ll) return -1;
    const int ch = hs <= 64 ? 1 : 2;
    const unsigned grid = (unsigned)CEIL_DIV(rows, DELTA_THREADS / 8 * delta_rows(ch));
    if (ch == 1) delta_kernel<1><<<grid, DELTA_THREADS, 0, stream>>>(delta, out, dout, rows, T, NH, hs);
    else delta_kernel<2><<<grid, DELTA_THREADS, 0, stream>>>(delta, out, dout, rows, T, NH, hs);
    CUDA_CHECK(cudaGetLastError());
    return 0;
}

// dqkv (B,T,3,NH,HS) = gradient of causal attention; delta: scratch of B*NH*T floats.  Head sizes: multiples of 8, 72..128.
// The entry point llmc_attention_bwd (attention_bwd1.cu) sends every head size but 64 here.
int llmc_attention_bwd_two_pass(bf16* dqkv, float* delta, const bf16* dout, const bf16* qkv, const bf16* out, const float* lse,
                                int B, int T, int NH, int hs, cudaStream_t stream) {
    if (hs <= 64 || hs > 128 || (hs % 8)) { fprintf(stderr, "[llmc_b200] attention backward: head size %d not supported (multiples of 8 from 64 to 128)\n", hs); return -1; }
    CUtensorMap tmQKV, tmDO, tmDQKV;
    int rc = llmc_attn_qkv_map(&tmQKV, qkv, B, T, NH, hs, BT);
    if (rc) return rc;
    {
        uint64_t dims[4] = {(uint64_t)hs, (uint64_t)NH, (uint64_t)T, (uint64_t)B};
        uint64_t strides[4] = {2, (uint64_t)hs * 2, (uint64_t)NH * hs * 2, (uint64_t)T * NH * hs * 2};
        uint32_t box[4] = {64, 1, 128, 1};
        if ((rc = llmc_get_tensormap(&tmDO, dout, 2, 4, dims, strides, box, 3))) return rc;
    }
    if ((rc = llmc_attn_qkv_map(&tmDQKV, dqkv, B, T, NH, hs, BT))) return rc;
    if ((rc = llmc_attention_delta(delta, out, dout, B, T, NH, hs, stream))) return rc;
    Args a;
    a.lse = lse; a.delta = delta; a.T = T; a.NH = NH; a.BH = B * NH;
    a.ks = CEIL_DIV(hs, 16);
    a.scale = 1.0f / sqrtf((float)hs);
    a.scale_log2e = a.scale * 1.4426950408889634f;
    a.status = llmc_status_ptr();
    const int nt = CEIL_DIV(T, BT);
    int sms = llmc_device_sm_count(); if (sms <= 0) sms = 148;
    const int grid = B * NH * nt < sms ? B * NH * nt : sms;
    static bool configured = false;
    if (!configured) {
        CUDA_CHECK(cudaFuncSetAttribute(attn_bwd_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
        CUDA_CHECK(cudaFuncSetAttribute(attn_bwd_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
        configured = true;
    }
    attn_bwd_kernel<true><<<grid, THREADS, SMEM, stream>>>(tmQKV, tmDO, tmDQKV, a);
    CUDA_CHECK(cudaGetLastError());
    attn_bwd_kernel<false><<<grid, THREADS, SMEM, stream>>>(tmQKV, tmDO, tmDQKV, a);
    CUDA_CHECK(cudaGetLastError());
    return 0;
}
