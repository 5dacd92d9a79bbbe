// Causal flash attention backward for sm_100a, head size 64, on the packed (B, T, 3, NH, HS) layout: ONE pass over the
// (key tile j, query tile i) pairs with the five products of the algorithm and nothing recomputed.
//
// The score tiles are formed TRANSPOSED (key rows on the TMEM lanes, queries along the columns), so that the two products
// that accumulate over the query loop take their A operand straight from tensor memory:
//
//   S^T  = K_j Q_i^T          dP^T = V_j dO_i^T                    (SS products, 128 x 128 fp32 in TMEM)
//   P^T  = exp(S^T scale - LSE_q)     dS^T = P^T (dP^T - delta_q) scale      (softmax threads; bf16 back into TMEM,
//                                                                             dS^T also to shared memory)
//   dV_j += P^T dO_i          dK_j += dS^T Q_i                     (TS products: A from TMEM, B = the streamed tile)
//   dQ_i(j) = dS K_j                                               (SS product: A = dS^T read M-major from shared memory)
//
// Shared-memory bandwidth is what bounds such a kernel at 64-wide heads (a 128 x 64 x 16 product with both operands in
// shared memory reads 6 KB for 32 cycles of arithmetic); keeping P^T and dS^T in tensor memory removes a third of that
// traffic and all of the P stores.
//
// A work item is (batch, head, g) with the two key tiles {g, nt-1-g}: nt + 1 pairs whatever g, so a static round-robin over
// the persistent CTAs is balanced.  dK_j / dV_j leave the CTA once per key tile.  What item g contributes to dQ_i is written as
// fp32 to a slot of its own in a workspace (the second key tile is added to what the first left there by a reducing bulk copy
// of the same CTA, ordered after the first); a second kernel adds the slots of a query tile in the order of g and rounds once.
// With many heads of few tiles (whole_heads) a CTA takes all units of a head instead and sums dQ_i in one slot: what the slot holds is fetched into the
// staging buffer behind the pair before, the drain warps add to it there, and the last key tile's sum is rounded and written for good.
// No atomics, no ordering between CTAs: the gradients are bit-reproducible, which the reference also demands of cuDNN
// (llmc/cudnn_att.cpp:186-191), and no CTA ever waits for another one.
//
// What bounds it: the chain S^T -> exponentials -> dP^T -> dS^T -> dK, dQ of one pair, about 2900 cycles, of which the tensor
// pipe works 1450; three things keep the chain short.  S^T(t+1) is issued before dV(t), so that its 64 columns are there when a
// softmax warp returns for them; the two warps of a scheduler take turns at the exponentials, so that one of them loads, packs
// and stores while the other has the unit to itself; and accumulators are read into registers and handed back before the
// staging buffer is waited for.  64 x 1024 x 12 heads: 632 us before, 603 with those, 556 with one slot per item instead of
// one per pair (a quarter less workspace to write and to add; tiles of one sequence alone need no second kernel), 523 with the row sums at the copy rate and the
// issuer on uniform registers, 459 with whole heads (a pair then moves 336 KB through shared memory, 2600 of its about 3300 cycles).
// Fetching K_j / V_j of later key tiles into L2 ahead of their loads was slower (566): the loads of 148 CTAs that change
// their head together wait for memory bandwidth, not for latency.
//
// Roles inside a CTA (512 threads):
//   warp 0       TMA producer: K_j, V_j resident (double buffered across key tiles); Q_i, dO_i through a 3-stage ring.
//   warp 1       issuer of all five products, in the order S^T(t+1), dV(t), dK(t), dQ(t), dP^T(t+1): program order is what
//                keeps dP^T of the next pair from overwriting the bf16 dS^T operand that aliases its TMEM columns.
//   warps 2-3    producers of the per-query statistics table.
//   warps 4-11   softmax: thread = key row x 64-query half.  Nothing is exchanged between threads (the row statistics of the
//                forward pass are per query = per column, read from a small shared table).
//   warps 12-15  drain: the pair's dQ contribution from TMEM to the workspace, and at the end of a key tile dV_j / dK_j to
//                global memory through a staging buffer and TMA stores.
//
// TMEM columns: S^T [0,128)  dP^T [128,256) (dS^T bf16 aliases the first 32 columns of each 64-column half)
//               dV [256,320)  dK [320,384)  dQ [384,448)  P^T bf16 [448,512).
//
// Head sizes above 64 use the two-pass kernels of attention_bwd.cu.
//
// Capability parity: attention_backward_cudnn (llmc/cudnn_att.cpp:256-288) and attention_backward of llmc/attention.cuh.
#include "common.cuh"
#include "pdl.cuh"

int llmc_attn_qkv_map(CUtensorMap* tm, const bf16* qkv, int B, int T, int NH, int hs, int rows);   // attention_fwd.cu
int llmc_attention_bwd_two_pass(bf16* dqkv, float* delta, const bf16* dout, const bf16* qkv, const bf16* out, const float* lse,
                                int B, int T, int NH, int hs, cudaStream_t stream);      // attention_bwd.cu
int llmc_attention_delta(float* delta, const bf16* out, const bf16* dout, int B, int T, int NH, int hs, cudaStream_t stream);

namespace {

constexpr int BT = 128;                             // tile rows (queries and keys)
constexpr int HS = 64;
constexpr int TILE_BYTES = BT * HS * 2;             // 16 KB: one 128-byte-swizzled TMA box
constexpr int PAIR_BYTES = 2 * TILE_BYTES;
constexpr int DS_BYTES = BT * BT * 2;               // 32 KB
constexpr int RB = 2;                               // resident (K_j, V_j) buffers
constexpr int XSTAGES = 3;                          // ring of streamed (Q_i, dO_i) pairs
constexpr int THREADS = 512;
constexpr int TMEM_COLS = 512;
constexpr int STAT_BYTES = 2 * 2 * BT * 4;          // [2 buffers][lse, delta][128 queries]
constexpr int SMEM = RB * PAIR_BYTES + XSTAGES * PAIR_BYTES + DS_BYTES + PAIR_BYTES + STAT_BYTES + 256;
constexpr int TURN_BAR = 3;                         // named barriers 3..10: [scheduler][query half] turns at the exponentials
constexpr int SLOT_FLOATS = BT * HS;                // one dQ contribution
static_assert(SMEM <= 232448, "shared memory of one CTA");

struct Args {
    bf16* dqkv;          // (B, T, 3, NH, 64)
    float* dq_ws;        // [B*NH][slots][16 column groups][128 rows][4] fp32: slot_of(i) + g holds what unit g adds to query tile i; WHOLE: [CTAs][nt] such slots
    const float* lse;    // (B, NH, T)
    const float* delta;  // (B, NH, T); null (one tile per sequence): computed here from out and dout
    const bf16* out;     // (B, T, NH, 64)
    const bf16* dout;
    int T, NH;
    int item0, items;    // this launch takes items item0 .. items - 1
    float scale, scale_log2e;
    int early;           // the next kernel may start while this one runs
    unsigned int* status;
    long long* trace;    // optional: [4 roles][8 events][TRACE_PAIRS] clock64() stamps of CTA 0 (null in normal runs)
};
constexpr int TRACE_PAIRS = 64;

DEVINL void tmem_st8(uint32_t taddr, const uint32_t* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}

template <int N> struct Groups { static constexpr int value = N; };

// Slots of the query tiles before i: tile k has one per unit g <= min(k, G - 1) that reaches it.
__host__ __device__ inline int slot_of(int i, int G) { return i <= G ? i * (i + 1) / 2 : G * (G + 1) / 2 + (i - G) * G; }

// The sequence of pairs of one CTA: items w (round-robin), their one or two key tiles, the query tiles i >= j of each.
// WHOLE: an item is a head, all its units in the order of g.
template <bool WHOLE>
struct Walk {
    int w, total, G, nt, stride, NH;
    int bh, b, h, g, seg, j, i;
    DEVINL void start(int first, int total_, int G_, int nt_, int stride_, int NH_) {
        w = first; total = total_; G = G_; nt = nt_; stride = stride_; NH = NH_;
        bh = b = h = g = seg = j = i = 0;
        if (w < total) item();
    }
    DEVINL bool valid() const { return w < total; }
    DEVINL void item() {
        if (WHOLE) { bh = w; g = 0; } else { bh = w / G; g = w - bh * G; }
        b = bh / NH; h = bh - b * NH; seg = 0; j = g; i = j;
    }
    DEVINL bool first_of_tile() const { return i == j; }
    DEVINL bool last_of_tile() const { return i == nt - 1; }
    DEVINL void next() {                      // valid() turns false past the last pair
        if (++i < nt) return;
        if (seg == 0 && 2 * g != nt - 1) { seg = 1; j = nt - 1 - g; i = j; return; }
        if (WHOLE && ++g < G) { seg = 0; j = g; i = j; return; }
        w += stride;
        if (w < total) item();
    }
};

// SHORT: one tile of at most 96 queries, whose row sums wait for as many loads as there are queries.  (In one kernel the second loop costs the
// registers of the first: 5 % of every size.)  us, the other form first: 128 sequences of 16 x 25 heads 107, 79, 64 of 40 x 25 heads 57, 46, 4 of 64 x 12
// heads 7.7, 7.4.  Three loads save too little of four unless the CTAs have several items each: 128 of 80 x 25 heads 116, 107, 4 of 80 x 12 heads 7.9, 8.4.
constexpr int SHORT_T = 64, SHORT_T_MANY = 96;
enum { SPLIT = 0, SHORT_SPLIT = 1, WHOLE_HEADS = 2 };
template <int MODE>
__global__ void __launch_bounds__(THREADS, 1)
attn_bwd1_kernel(const __grid_constant__ CUtensorMap tmQKV, const __grid_constant__ CUtensorMap tmDO,
                 const __grid_constant__ CUtensorMap tmDQKV, const Args a) {
    constexpr bool SHORT = MODE == SHORT_SPLIT, WHOLE = MODE == WHOLE_HEADS;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sRes = smem;                              // [RB][K_j, V_j]
    uint8_t* sStr = sRes + RB * PAIR_BYTES;            // [XSTAGES][Q_i, dO_i]
    uint8_t* sdS = sStr + XSTAGES * PAIR_BYTES;        // dS^T: 128 key rows x 128 queries, two 64-query chunks of 128-byte rows
    uint8_t* sOut = sdS + DS_BYTES;                    // dV_j, dK_j on their way out (two TMA boxes)
    float* sStat = reinterpret_cast<float*>(sOut + PAIR_BYTES);     // [2][2][128]
    uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(sStat) + STAT_BYTES);
    uint64_t* res_full = bars + 0;    // [2]
    uint64_t* res_empty = bars + 2;   // [2]
    uint64_t* x_full = bars + 4;      // [3]
    uint64_t* x_empty = bars + 7;     // [3]
    uint64_t* s_full = bars + 10;     // S^T(t) complete                            (1 commit)
    uint64_t* s_empty = bars + 11;    // every softmax warp has S^T(t) in registers  (8 arrivals)
    uint64_t* dp_full = bars + 12;    // dP^T(t) complete                           (1 commit)
    uint64_t* p_ready = bars + 13;    // P^T(t) is in TMEM                           (8 arrivals)
    uint64_t* p_empty = bars + 14;    // dV(t) has read P^T(t)                       (1 commit)
    uint64_t* ds_ready = bars + 15;   // dS^T(t) is in TMEM and in shared memory     (8 arrivals)
    uint64_t* ds_empty = bars + 16;   // dK(t), dQ(t) have read dS^T(t)              (1 commit)
    uint64_t* dq_full = bars + 17;    // dQ(t) complete                              (1 commit)
    uint64_t* dq_empty = bars + 18;   // the drain warps hold dQ(t) in registers     (4 arrivals)
    uint64_t* acc_full = bars + 19;   // dV_j, dK_j complete                         (1 commit)
    uint64_t* acc_empty = bars + 20;  // the drain warps hold them                   (4 arrivals)
    uint64_t* st_full = bars + 21;    // [2] statistics table of a pair written      (2 arrivals)
    uint64_t* st_empty = bars + 23;   // [2] ... and read by every softmax warp      (8 arrivals)
    uint64_t* part_full = bars + 25;  // WHOLE: what a query tile has so far is in the staging buffer
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 26);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const int nt = CEIL_DIV(a.T, BT);
    const int G = (nt + 1) >> 1;                      // key-tile groups {g, nt-1-g}
    const int nslots = slot_of(nt, G);

    if (threadIdx.x == 0) {
        if ((smem_u32(smem) & 1023u) != 0) record_error(a.status, ST_BAD_ARG, 0x28);
        for (int i = 0; i < 2; i++) { mbar_init(&res_full[i], 1); mbar_init(&res_empty[i], 1); mbar_init(&st_full[i], 2); mbar_init(&st_empty[i], 8); }
        for (int i = 0; i < XSTAGES; i++) { mbar_init(&x_full[i], 1); mbar_init(&x_empty[i], 1); }
        mbar_init(s_full, 1); mbar_init(s_empty, 8); mbar_init(dp_full, 1); mbar_init(p_ready, 8); mbar_init(p_empty, 1);
        mbar_init(ds_ready, 8); mbar_init(ds_empty, 1); mbar_init(dq_full, 1); mbar_init(dq_empty, 4);
        mbar_init(acc_full, 1); mbar_init(acc_empty, 4); mbar_init(part_full, 1);
        *abort_flag = 0;
        mbar_fence_init();
        tma_prefetch_desc(&tmQKV); tma_prefetch_desc(&tmDO); tma_prefetch_desc(&tmDQKV);
    }
    if (warp == 1) { tmem_alloc(tmem_slot, TMEM_COLS); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t tS = tmem_base, tdP = tmem_base + 128, tdV = tmem_base + 256, tdK = tmem_base + 320, tdQ = tmem_base + 384,
                   tP = tmem_base + 448;
    pdl_wait();
    if (a.early) pdl_trigger();

    // time stamps of CTA 0's first TRACE_PAIRS pairs, one thread per role, for the timeline tool (llmc_attention_bwd_set_trace)
#define TRACE(role, ev) do { if (a.trace != nullptr && blockIdx.x == 0 && t < TRACE_PAIRS) a.trace[((role) * 8 + (ev)) * TRACE_PAIRS + t] = clock64(); } while (0)

    Walk<WHOLE> wk;
    wk.start(a.item0 + blockIdx.x, a.items, G, nt, gridDim.x, a.NH);

    if (warp == 0) {
        // ---------------------------------------------------------------- TMA producer
        if (lane == 0) {
            int xst = 0; uint32_t xph = 0;
            int kvt = 0;
            for (; wk.valid(); wk.next()) {
                if (wk.first_of_tile()) {
                    const int rb = kvt & 1;
                    if (!mbar_wait_relaxed(&res_empty[rb], ((kvt >> 1) & 1) ^ 1, abort_flag, a.status, 0x681)) break;
                    uint8_t* rdst = sRes + rb * PAIR_BYTES;
                    mbar_expect_tx(&res_full[rb], PAIR_BYTES);
                    tma_load_4d(rdst, &tmQKV, &res_full[rb], 0, a.NH + wk.h, wk.j * BT, wk.b);                    // K_j
                    tma_load_4d(rdst + TILE_BYTES, &tmQKV, &res_full[rb], 0, 2 * a.NH + wk.h, wk.j * BT, wk.b);   // V_j
                    kvt++;
                }
                if (!mbar_wait_relaxed(&x_empty[xst], xph ^ 1, abort_flag, a.status, 0x680)) break;
                uint8_t* dst = sStr + xst * PAIR_BYTES;
                mbar_expect_tx(&x_full[xst], PAIR_BYTES);
                tma_load_4d(dst, &tmQKV, &x_full[xst], 0, wk.h, wk.i * BT, wk.b);                                 // Q_i
                tma_load_4d(dst + TILE_BYTES, &tmDO, &x_full[xst], 0, wk.h, wk.i * BT, wk.b);                     // dO_i
                if (++xst == XSTAGES) { xst = 0; xph ^= 1; }
            }
        }
    } else if (warp == 1) {
        // ---------------------------------------------------------------- issuer of the five products
        // The whole warp runs this code in uniform control flow and one elected lane executes the tcgen05 instructions.  With a
        // single lane inside a divergent branch every descriptor has to be moved from that lane's registers to uniform registers,
        // which costs the issuing thread about 90 cycles per product (measured) -- more than a 128 x 64 x 16 product runs.
        // Wait results go through a warp vote so that the compiler knows the branches on them to be uniform.
        if (wk.valid()) {
            const bool leader = elect_one();
#define WAIT_ALL(bar, parity, code) (__all_sync(0xffffffffu, mbar_wait_relaxed(bar, parity, abort_flag, a.status, code, 32)) != 0)
            constexpr uint32_t idesc_s = umma_idesc_bf16(BT, BT, 0, 0);      // S^T, dP^T: both operands K-major
            constexpr uint32_t idesc_ts = umma_idesc_bf16(BT, HS, 0, 1);     // dV, dK: A from TMEM, B N-major
            constexpr uint32_t idesc_q = umma_idesc_bf16(BT, HS, 1, 1);      // dQ: A = dS^T read M-major, B = K_j N-major
            // Descriptors of buffer 0 of each kind are built once; the others follow by addition (the start address sits in the
            // low bits of a descriptor, in 16-byte units).
            const uint64_t dQk0 = umma_desc_sw128(smem_u32(sStr), 16, 1024), dOk0 = umma_desc_sw128(smem_u32(sStr + TILE_BYTES), 16, 1024);
            const uint64_t dQn0 = umma_desc_sw128(smem_u32(sStr), TILE_BYTES, 1024), dOn0 = umma_desc_sw128(smem_u32(sStr + TILE_BYTES), TILE_BYTES, 1024);
            const uint64_t dKk0 = umma_desc_sw128(smem_u32(sRes), 16, 1024), dVk0 = umma_desc_sw128(smem_u32(sRes + TILE_BYTES), 16, 1024);
            const uint64_t dKn0 = umma_desc_sw128(smem_u32(sRes), TILE_BYTES, 1024);
            const uint64_t dSm = umma_desc_sw128(smem_u32(sdS), BT * 128, 1024);     // dS^T as an M-major A operand
            constexpr uint32_t PAIR_UNITS = PAIR_BYTES / 16;
            // S^T and dP^T of one pair: A = resident K_j / V_j, B = streamed Q_i / dO_i; 16 channels = 32 bytes = 2 address units per step
            auto issue_s = [&](int rb, int st) {
                const uint64_t ka = dKk0 + (uint32_t)rb * PAIR_UNITS, qb = dQk0 + (uint32_t)st * PAIR_UNITS;
                if (leader) {
                    #pragma unroll
                    for (int kk = 0; kk < HS / 16; kk++) umma_ss(tS, ka + 2 * kk, qb + 2 * kk, idesc_s, kk > 0);
                    umma_commit(s_full);
                }
            };
            auto issue_dp = [&](int rb, int st) {
                const uint64_t va = dVk0 + (uint32_t)rb * PAIR_UNITS, ob = dOk0 + (uint32_t)st * PAIR_UNITS;
                if (leader) {
                    #pragma unroll
                    for (int kk = 0; kk < HS / 16; kk++) umma_ss(tdP, va + 2 * kk, ob + 2 * kk, idesc_s, kk > 0);
                    umma_commit(dp_full);
                }
            };
            uint32_t t = 0;
            int st = 0;                // ring stage of pair t
            uint32_t xph = 0;          // parity of the ring round of pair t
            int kvt = 0;               // key-tile counter of pair t
            // prologue: S^T(0), dP^T(0)
            bool ok = WAIT_ALL(&res_full[0], 0, 0x690) && WAIT_ALL(&x_full[0], 0, 0x691);
            tc_fence_after();
            if (ok) { issue_s(0, 0); issue_dp(0, 0); }
            while (ok) {
                // pair t = wk; the pair after it, if any
                Walk<WHOLE> nx = wk; nx.next();
                const bool have_next = nx.valid();
                const int rb = kvt & 1;
                const int nst = st + 1 == XSTAGES ? 0 : st + 1;
                const uint32_t nph = st + 1 == XSTAGES ? xph ^ 1 : xph;
                const int nkvt = have_next && nx.first_of_tile() ? kvt + 1 : kvt;
                const int nrb = nkvt & 1;
                const uint32_t acc = wk.first_of_tile() ? 0u : 1u;
                // ---- S^T(t+1), as soon as the second half's warps hold S^T(t): the first half's are through with pair t by then
                if (leader) TRACE(0, 0);
                if (have_next) {
                    if (nx.first_of_tile()) ok = WAIT_ALL(&res_full[nrb], (nkvt >> 1) & 1, 0x694);
                    ok = ok && WAIT_ALL(&x_full[nst], nph, 0x695);
                    ok = ok && WAIT_ALL(s_empty, t & 1, 0x696);
                    if (!ok) break;
                    tc_fence_after();
                    issue_s(nrb, nst);
                }
                // ---- dV(t) += P^T dO_i : A = P^T in TMEM (16 queries = 8 columns per step), B = dO_i N-major (16 rows = 2048 bytes)
                ok = WAIT_ALL(p_ready, t & 1, 0x692);
                if (ok && wk.first_of_tile() && kvt > 0) ok = WAIT_ALL(acc_empty, (kvt - 1) & 1, 0x693);
                if (!ok) break;
                tc_fence_after();
                if (leader) TRACE(0, 1);
                {
                    const uint64_t ob = dOn0 + (uint32_t)st * PAIR_UNITS;
                    if (leader) {
                        #pragma unroll
                        for (int kk = 0; kk < BT / 16; kk++) umma_ts(tdV, tP + kk * 8, ob + 128 * kk, idesc_ts, acc | (kk > 0));
                        umma_commit(p_empty);
                    }
                }
                if (leader) TRACE(0, 2);
                // ---- dK(t) += dS^T Q_i (A = dS^T in TMEM: queries 0..63 in columns [0,32) of the dP^T tile, 64..127 in [64,96));
                //      dQ(t) = dS K_j (A = dS^T in shared memory read M-major: 16 key rows = 2048 bytes per step)
                ok = WAIT_ALL(ds_ready, t & 1, 0x697);
                if (ok && t > 0) ok = WAIT_ALL(dq_empty, (t - 1) & 1, 0x698);
                if (!ok) break;
                tc_fence_after();
                if (leader) TRACE(0, 3);
                {
                    const uint64_t qb = dQn0 + (uint32_t)st * PAIR_UNITS, kb = dKn0 + (uint32_t)rb * PAIR_UNITS;
                    if (leader) {
                        #pragma unroll
                        for (int kk = 0; kk < BT / 16; kk++)
                            umma_ts(tdK, tdP + (kk >> 2) * 64 + (kk & 3) * 8, qb + 128 * kk, idesc_ts, acc | (kk > 0));
                        if (wk.last_of_tile()) umma_commit(acc_full);
                        #pragma unroll
                        for (int kk = 0; kk < BT / 16; kk++) umma_ss(tdQ, dSm + 128 * kk, kb + 128 * kk, idesc_q, kk > 0);
                        umma_commit(dq_full);
                        umma_commit(ds_empty);
                        umma_commit(&x_empty[st]);
                        if (wk.last_of_tile()) umma_commit(&res_empty[rb]);
                    }
                }
                // ---- dP^T(t+1): after dK(t) in program order, so it cannot overwrite dS^T(t) early
                if (have_next) issue_dp(nrb, nst);
                if (leader) TRACE(0, 4);
                if (!have_next) break;
                wk = nx; st = nst; xph = nph; kvt = nkvt; t++;
            }
#undef WAIT_ALL
        }
    } else if (warp < 4) {
        // ---------------------------------------------------------------- statistics of a pair's 128 queries -> table (t & 1), 64 by each of the
        // two warps: the LSE in log2 units and delta = sum_d O dO times the scale; queries past the end of the sequence get LSE = +inf, so
        // that their P^T column is zero
        const float log2e = 1.4426950408889634f;
        if constexpr (SHORT) {
            // at most 96 queries: each warp takes every other group of 16, and none that the sequence does not have
            auto few = [&](auto groups) {
                constexpr int NG = decltype(groups)::value;
                const int w0 = (warp - 2) * 16;
                bool ok = true;
                uint32_t t = 0;
                for (; wk.valid() && ok; wk.next(), t++) {
                    float l[2], d[16];
                    #pragma unroll
                    for (int k = 0; k < 2; k++) {
                        const int q = w0 + (2 * k + (lane >> 4)) * 32 + (lane & 15);
                        l[k] = q < a.T ? a.lse[(size_t)wk.bh * a.T + q] * log2e : INFINITY;
                    }
                    #pragma unroll
                    for (int part = 0; part < NG; part++) {
                        bf16x8 o[4], g[4];
                        #pragma unroll
                        for (int k = 0; k < 4; k++) {
                            const int q = min(w0 + part * 32 + k * 4 + (lane >> 3), a.T - 1);
                            const size_t at = (((size_t)wk.b * a.T + q) * a.NH + wk.h) * HS + (lane & 7) * 8;
                            o[k] = ld128cs(a.out + at); g[k] = ld128(a.dout + at);
                        }
                        #pragma unroll
                        for (int k = 0; k < 4; k++) {
                            float acc = 0.f;
                            #pragma unroll
                            for (int e = 0; e < 8; e++) acc += __bfloat162float(o[k][e]) * __bfloat162float(g[k][e]);
                            acc += __shfl_xor_sync(0xffffffffu, acc, 1);
                            acc += __shfl_xor_sync(0xffffffffu, acc, 2);
                            acc += __shfl_xor_sync(0xffffffffu, acc, 4);
                            d[part * 4 + k] = w0 + part * 32 + k * 4 + (lane >> 3) < a.T ? acc * a.scale : 0.f;
                        }
                    }
                    #pragma unroll
                    for (int k = NG * 4; k < 16; k++) d[k] = 0.f;
                    ok = __all_sync(0xffffffffu, mbar_wait_relaxed(&st_empty[t & 1], ((t >> 1) & 1) ^ 1, abort_flag, a.status, 0x6b0)) != 0;
                    float* tab = sStat + (t & 1) * (2 * BT) + w0;
                    #pragma unroll
                    for (int k = 0; k < 2; k++) tab[(2 * k + (lane >> 4)) * 32 + (lane & 15)] = l[k];
                    if ((lane & 7) == 0) {
                        #pragma unroll
                        for (int k = 0; k < 16; k++) tab[BT + (k >> 2) * 32 + (k & 3) * 4 + (lane >> 3)] = d[k];
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&st_full[t & 1]);
                }
            };
            if (a.T <= 32) few(Groups<1>()); else if (a.T <= 64) few(Groups<2>()); else few(Groups<3>());
        } else {
            const int w0 = (warp - 2) * 64;                 // the warp's queries of the tile
            bool ok = true;
            uint32_t t = 0;
            for (; wk.valid() && ok; wk.next(), t++) {
                const int tq0 = wk.i * BT + w0;
                float l[2], d[16];
                const size_t row = (size_t)wk.bh * a.T + tq0 + lane;
                #pragma unroll
                for (int k = 0; k < 2; k++) l[k] = tq0 + k * 32 + lane < a.T ? a.lse[row + k * 32] * log2e : INFINITY;
                if (a.delta != nullptr) {
                    #pragma unroll
                    for (int k = 0; k < 2; k++) d[k] = tq0 + k * 32 + lane < a.T ? a.delta[row + k * 32] * a.scale : 0.f;
                } else {
                    // 8 lanes per query, 4 queries per step; no branch around the loads, so that they are on their way at once
                    #pragma unroll
                    for (int part = 0; part < 4; part++) {
                        bf16x8 o[4], g[4];
                        #pragma unroll
                        for (int k = 0; k < 4; k++) {
                            const int tq = min(tq0 + part * 16 + k * 4 + (lane >> 3), a.T - 1);
                            const size_t at = (((size_t)wk.b * a.T + tq) * a.NH + wk.h) * HS + (lane & 7) * 8;
                            o[k] = ld128cs(a.out + at); g[k] = ld128(a.dout + at);
                        }
                        #pragma unroll
                        for (int k = 0; k < 4; k++) {
                            float acc = 0.f;
                            #pragma unroll
                            for (int e = 0; e < 8; e++) acc += __bfloat162float(o[k][e]) * __bfloat162float(g[k][e]);
                            acc += __shfl_xor_sync(0xffffffffu, acc, 1);
                            acc += __shfl_xor_sync(0xffffffffu, acc, 2);
                            acc += __shfl_xor_sync(0xffffffffu, acc, 4);
                            d[part * 4 + k] = tq0 + part * 16 + k * 4 + (lane >> 3) < a.T ? acc * a.scale : 0.f;
                        }
                    }
                }
                ok = __all_sync(0xffffffffu, mbar_wait_relaxed(&st_empty[t & 1], ((t >> 1) & 1) ^ 1, abort_flag, a.status, 0x6b0)) != 0;
                float* tab = sStat + (t & 1) * (2 * BT) + w0;
                tab[lane] = l[0]; tab[32 + lane] = l[1];
                if (a.delta != nullptr) {
                    tab[BT + lane] = d[0]; tab[BT + 32 + lane] = d[1];
                } else if ((lane & 7) == 0) {
                    #pragma unroll
                    for (int k = 0; k < 16; k++) tab[BT + k * 4 + (lane >> 3)] = d[k];
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&st_full[t & 1]);
            }
        }
    } else if (warp < 12) {
        // ---------------------------------------------------------------- softmax: thread = key row r x query half hf
        const int q = warp & 3;                        // TMEM lane quarter
        const int hf = (warp - 4) >> 2;                // query half
        const int r = q * 32 + lane;                   // key row of the tile
        const uint32_t lane_off = (uint32_t)(q * 32) << 16;
        bool ok = true;
        if (hf == 1) turn_pass(TURN_BAR + 2 * q);      // the first half has the first turn
        uint32_t t = 0;
        for (; wk.valid(); wk.next(), t++) {
            const int i = wk.i, j = wk.j;
            const float* stat = sStat + (t & 1) * (2 * BT) + hf * 64;       // lse * log2(e) of this half's queries; delta * scale 128 floats further
            if (threadIdx.x == 128) TRACE(1, 0);
            ok = mbar_wait(s_full, t & 1, abort_flag, a.status, 0x6a0) && ok;
            tc_fence_after();
            if (threadIdx.x == 128) TRACE(1, 1);
            ok = mbar_wait(&st_full[t & 1], (t >> 1) & 1, abort_flag, a.status, 0x6a1) && ok;
            // ---- P^T = exp2(S^T * scale * log2(e) - LSE * log2(e)); causal: query >= key
            float p[64];
            // only the diagonal tile and a ragged last key tile need masks; both conditions are the same for the whole warp
            const bool masked = (i == j) || (j * BT + BT > a.T);
            {
                uint32_t sv[64];
                tmem_ld32(tS + lane_off + hf * 64, sv);
                tmem_ld32(tS + lane_off + hf * 64 + 32, sv + 32);
                tmem_ld_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(s_empty);
                float sl = a.scale_log2e;
                turn_wait(TURN_BAR + 2 * q + hf, sl);
                if (threadIdx.x == 128) TRACE(1, 6);
                const uint64_t sl2 = f2_pack(sl, sl);
                #pragma unroll
                for (int e = 0; e < 64; e += 4) {
                    const float4 l4 = *reinterpret_cast<const float4*>(stat + e);
                    const float2 x0 = f2_unpack(f2_fma(f2_pack_u(sv[e], sv[e + 1]), sl2, f2_pack(-l4.x, -l4.y)));
                    const float2 x1 = f2_unpack(f2_fma(f2_pack_u(sv[e + 2], sv[e + 3]), sl2, f2_pack(-l4.z, -l4.w)));
                    p[e] = ex2_fast(x0.x); p[e + 1] = ex2_fast(x0.y); p[e + 2] = ex2_fast(x1.x); p[e + 3] = ex2_fast(x1.y);
                }
                turn_pass(TURN_BAR + 2 * q + (hf ^ 1), p[63]);
            }
            if (masked) {
                const int lo = j * BT + r >= a.T ? 64 : (i == j ? r - hf * 64 : 0);      // first query of this half that counts for this key
                #pragma unroll
                for (int e = 0; e < 64; e++) p[e] = e < lo ? 0.f : p[e];
            }
            if (t > 0) ok = mbar_wait(p_empty, (t - 1) & 1, abort_flag, a.status, 0x6a2) && ok;      // dV(t-1) has read P^T(t-1)
            tc_fence_after();
            if (threadIdx.x == 128) TRACE(1, 7);
            {
                uint32_t pk[32];
                #pragma unroll
                for (int e = 0; e < 32; e++) pk[e] = pack_bf16x2(p[2 * e], p[2 * e + 1]);
                tmem_st16(tP + lane_off + hf * 32, pk);
                tmem_st16(tP + lane_off + hf * 32 + 16, pk + 16);
            }
            if (threadIdx.x == 128) TRACE(1, 2);
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_ready);
            if (threadIdx.x == 128) TRACE(1, 3);
            // ---- dS^T = P^T * (dP^T * scale - delta * scale), in four chunks of 16 queries: bf16 to TMEM (inside this half's own
            //      columns of the dP^T tile: a chunk's bf16 lands on fp32 columns that are already in registers) and to shared memory
            ok = mbar_wait(dp_full, t & 1, abort_flag, a.status, 0x6a3) && ok;
            if (t > 0) ok = mbar_wait(ds_empty, (t - 1) & 1, abort_flag, a.status, 0x6a4) && ok;     // dK / dQ (t-1) have read dS^T(t-1)
            tc_fence_after();
            if (threadIdx.x == 128) TRACE(1, 4);
            uint8_t* drow = sdS + hf * (BT * 128) + r * 128;
            const uint64_t sc2 = f2_pack(a.scale, a.scale);
            uint32_t dv[2][16];
            tmem_ld16(tdP + lane_off + hf * 64, dv[0]);
            #pragma unroll
            for (int c = 0; c < 4; c++) {
                tmem_ld_wait();
                if (c < 3) tmem_ld16(tdP + lane_off + hf * 64 + (c + 1) * 16, dv[(c + 1) & 1]);
                const uint32_t* dc = dv[c & 1];
                uint32_t dd[8];
                #pragma unroll
                for (int e = 0; e < 16; e += 4) {
                    const float4 d4 = *reinterpret_cast<const float4*>(stat + BT + c * 16 + e);
                    dd[e / 2] = pack_bf16x2(f2_mul(f2_pack(p[c * 16 + e], p[c * 16 + e + 1]), f2_fma(f2_pack_u(dc[e], dc[e + 1]), sc2, f2_pack(-d4.x, -d4.y))));
                    dd[e / 2 + 1] = pack_bf16x2(f2_mul(f2_pack(p[c * 16 + e + 2], p[c * 16 + e + 3]), f2_fma(f2_pack_u(dc[e + 2], dc[e + 3]), sc2, f2_pack(-d4.z, -d4.w))));
                }
                tmem_st8(tdP + lane_off + hf * 64 + c * 8, dd);
                // 16 queries = 32 bytes = two 16-byte units 2c, 2c+1 of this row, 128-byte swizzle
                *reinterpret_cast<uint4*>(drow + (((2 * c) ^ (r & 7)) * 16)) = make_uint4(dd[0], dd[1], dd[2], dd[3]);
                *reinterpret_cast<uint4*>(drow + (((2 * c + 1) ^ (r & 7)) * 16)) = make_uint4(dd[4], dd[5], dd[6], dd[7]);
            }
            tmem_st_wait();
            tc_fence_before();
            fence_async_smem();
            __syncwarp();
            if (lane == 0) { mbar_arrive(ds_ready); mbar_arrive(&st_empty[t & 1]); }
            if (threadIdx.x == 128) TRACE(1, 5);
        }
        if (hf == 0) turn_wait(TURN_BAR + 2 * q);      // the last turn passed on by the second half
    } else {
        // ---------------------------------------------------------------- drain warps (128 threads): thread = row rr of a tile
        const int q = warp & 3;
        const int rr = q * 32 + lane;
        const uint32_t lane_off = (uint32_t)(q * 32) << 16;
        const bool issuer = warp == 12 && lane == 0;
        bool ok = true;
        bool staged = false;
        uint32_t t = 0, parts = 0;
        int kvt = 0;
        for (; wk.valid(); t++) {
            const int bh = wk.bh, b = wk.b, h = wk.h, i = wk.i, j = wk.j;
            const bool last = wk.last_of_tile();
            const int g = wk.g, seg = wk.seg;
            wk.next();
            // ---- the pair's dQ contribution: 64 fp32 of query row rr, slot order [group of 4 columns][row][4 floats].  The second key tile of a unit
            //      is added to what the first left in the slot, nt - j pairs ago, by a copy that reduces in L2.  (All contributions of a head summed
            //      that way, without the fold kernel, took longer: reductions of 32 KB per pair and SM run at 1.4 TB/s.)
            if (threadIdx.x == 384) TRACE(2, 0);
            ok = mbar_wait_relaxed(dq_full, t & 1, abort_flag, a.status, 0x6b1) && ok;
            tc_fence_after();
            if (threadIdx.x == 384) TRACE(2, 1);
            // through the staging buffer and one bulk copy: 16 global stores per thread and pair through the load/store unit held up
            // the shared-memory reads of the softmax warps for about a thousand cycles per pair (measured)
            // WHOLE: one slot per query tile, of the CTA.  What it holds was fetched into the staging buffer behind the pair before; the last key tile's sum is
            // rounded and leaves for good.
            float* slot = a.dq_ws + (WHOLE ? (size_t)blockIdx.x * nt + i : (size_t)bh * nslots + slot_of(i, G) + g) * SLOT_FLOATS;
            const bool more = WHOLE && j > 0, done = WHOLE ? j == min(i, nt >> 1) : nt == 1;
            if (!WHOLE && seg == 1 && issuer) {
                if (nt - j == 1) tma_store_wait<0>(); else if (nt - j == 2) tma_store_wait<1>(); else tma_store_wait<2>();
            }
            {
                uint32_t v[64];
                tmem_ld32(tdQ + lane_off, v);
                tmem_ld32(tdQ + lane_off + 32, v + 32);
                tmem_ld_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(dq_empty);
                if (more) {
                    ok = mbar_wait_relaxed(part_full, parts & 1, abort_flag, a.status, 0x6b3) && ok;
                    parts++;
                    #pragma unroll
                    for (int e = 0; e < 16; e++) {
                        const float4 s4 = *reinterpret_cast<const float4*>(sOut + e * (BT * 16) + rr * 16);
                        v[4 * e] = __float_as_uint(s4.x + __uint_as_float(v[4 * e])); v[4 * e + 1] = __float_as_uint(s4.y + __uint_as_float(v[4 * e + 1]));
                        v[4 * e + 2] = __float_as_uint(s4.z + __uint_as_float(v[4 * e + 2])); v[4 * e + 3] = __float_as_uint(s4.w + __uint_as_float(v[4 * e + 3]));
                    }
                    if (done) asm volatile("bar.sync 1, 128;" ::: "memory");        // all have read what the rounded rows go over
                } else if (staged) {
                    if (issuer) tma_store_wait_read<0>();                           // the previous copy has read the buffer
                    asm volatile("bar.sync 1, 128;" ::: "memory");
                }
                if (!done) {
                    #pragma unroll
                    for (int e = 0; e < 16; e++)
                        *reinterpret_cast<uint4*>(sOut + e * (BT * 16) + rr * 16) = make_uint4(v[4 * e], v[4 * e + 1], v[4 * e + 2], v[4 * e + 3]);
                } else {
                    // dQ is finished
                    #pragma unroll
                    for (int u = 0; u < 8; u++) {
                        uint4 o;
                        o.x = pack_bf16x2(__uint_as_float(v[8 * u]), __uint_as_float(v[8 * u + 1]));
                        o.y = pack_bf16x2(__uint_as_float(v[8 * u + 2]), __uint_as_float(v[8 * u + 3]));
                        o.z = pack_bf16x2(__uint_as_float(v[8 * u + 4]), __uint_as_float(v[8 * u + 5]));
                        o.w = pack_bf16x2(__uint_as_float(v[8 * u + 6]), __uint_as_float(v[8 * u + 7]));
                        *reinterpret_cast<uint4*>(sOut + rr * 128 + ((u ^ (rr & 7)) * 16)) = o;
                    }
                }
            }
            fence_async_smem();
            asm volatile("bar.sync 1, 128;" ::: "memory");
            if (issuer && ok) {
                if (done)
                    tma_store_4d(&tmDQKV, sOut, 0, h, i * BT, b);
                else if (WHOLE || seg == 0)
                    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
                                 ::"l"(slot), "r"(smem_u32(sOut)), "r"(SLOT_FLOATS * 4) : "memory");
                else
                    asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;"
                                 ::"l"(slot), "r"(smem_u32(sOut)), "r"(SLOT_FLOATS * 4) : "memory");
                tma_store_commit();
            }
            staged = true;
            if (threadIdx.x == 384) TRACE(2, 2);
            if (last) {
                // ---- end of a key tile: dV_j and dK_j as bf16 tiles in the layout of a 128-byte-swizzled TMA box, one bulk store
                //      each (rows past T are clipped by TMA); a warp writing rows itself would touch 32 cache lines per instruction
                ok = mbar_wait_relaxed(acc_full, kvt & 1, abort_flag, a.status, 0x6b2) && ok;
                tc_fence_after();
                // (first into registers: the next tile's products wait for the accumulators, not for the staging buffer)
                uint32_t pk[64];
                #pragma unroll
                for (int c = 0; c < 4; c++) {
                    uint32_t v[32];
                    tmem_ld32((c < 2 ? tdV : tdK) + lane_off + (c & 1) * 32, v);
                    tmem_ld_wait();
                    #pragma unroll
                    for (int e = 0; e < 16; e++) pk[c * 16 + e] = pack_bf16x2(__uint_as_float(v[2 * e]), __uint_as_float(v[2 * e + 1]));
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(acc_empty);
                if (staged) { if (issuer) tma_store_wait_read<0>(); asm volatile("bar.sync 1, 128;" ::: "memory"); }
                #pragma unroll
                for (int u = 0; u < 16; u++)
                    *reinterpret_cast<uint4*>(sOut + (u >> 3) * TILE_BYTES + rr * 128 + (((u & 7) ^ (rr & 7)) * 16)) = make_uint4(pk[4 * u], pk[4 * u + 1], pk[4 * u + 2], pk[4 * u + 3]);
                fence_async_smem();
                asm volatile("bar.sync 1, 128;" ::: "memory");
                if (issuer && ok) {
                    tma_store_4d(&tmDQKV, sOut, 0, 2 * a.NH + h, j * BT, b);
                    tma_store_4d(&tmDQKV, sOut + TILE_BYTES, 0, a.NH + h, j * BT, b);
                    tma_store_commit();
                }
                staged = true;
                kvt++;
            }
            if (WHOLE && wk.valid() && wk.j > 0 && issuer && ok) {
                // what the next pair's query tile has so far.  Its last addition left nt - j pairs ago or more.
                if (nt - wk.j == 1) tma_store_wait<0>(); else if (nt - wk.j == 2) tma_store_wait<1>(); else tma_store_wait<2>();
                tma_store_wait_read<0>();
                mbar_expect_tx(part_full, SLOT_FLOATS * 4);
                asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                             ::"r"(smem_u32(sOut)), "l"(a.dq_ws + ((size_t)blockIdx.x * nt + wk.i) * SLOT_FLOATS), "r"(SLOT_FLOATS * 4), "r"(smem_u32(part_full)) : "memory");
            }
        }
        if (issuer) tma_store_wait<0>();
    }
#undef TRACE
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

// dQ[b, t, h, :] = bf16( sum over the units g of slot(i, g)[r, :] ), i = t / 128, r = t % 128, added in the order of g.
// One CTA per (batch, head, query tile), heaviest tiles first.  A slot is read as it was written (order [group of 4 columns][row]
// [4 floats]): a warp reads 512 contiguous bytes per instruction, every thread has 16 loads of 16 bytes in flight (two slots);
// the sums are transposed through shared memory so that the 8 lanes of a row store its 128 bytes together.
__global__ void __launch_bounds__(256)
dq_fold_kernel(bf16* __restrict__ dqkv, const float* __restrict__ ws, int bh0, int T, int NH, int nt) {
    __shared__ __align__(16) bf16 tile[BT][HS + 8];
    const int nbh = gridDim.x / nt;
    const int i = nt - 1 - (int)(blockIdx.x / nbh);
    const int bh = bh0 + (int)(blockIdx.x % nbh);
    const int G = (nt + 1) >> 1, n = min(i, G - 1) + 1;
    const int t = threadIdx.x;
    const float* src = ws + ((size_t)bh * slot_of(nt, G) + slot_of(i, G)) * SLOT_FLOATS + t * 4;
    f32x4 acc[8];
    #pragma unroll
    for (int k = 0; k < 8; k++)
        #pragma unroll
        for (int e = 0; e < 4; e++) acc[k][e] = 0.f;
    for (int j = 0; j < n; j += 2) {
        const bool two = j + 1 < n;
        f32x4 a0[8], a1[8];
        #pragma unroll
        for (int k = 0; k < 8; k++) a0[k] = ld128cs(src + (size_t)j * SLOT_FLOATS + k * 1024);
        if (two) {
            #pragma unroll
            for (int k = 0; k < 8; k++) a1[k] = ld128cs(src + (size_t)(j + 1) * SLOT_FLOATS + k * 1024);
        }
        #pragma unroll
        for (int k = 0; k < 8; k++)
            #pragma unroll
            for (int e = 0; e < 4; e++) acc[k][e] += a0[k][e];
        if (two) {
            #pragma unroll
            for (int k = 0; k < 8; k++)
                #pragma unroll
                for (int e = 0; e < 4; e++) acc[k][e] += a1[k][e];
        }
    }
    // thread t holds row t % 128, column groups 2k + t / 128
    const int row = t & (BT - 1), g0 = t >> 7;
    #pragma unroll
    for (int k = 0; k < 8; k++) {
        __nv_bfloat162 lo = __floats2bfloat162_rn(acc[k][0], acc[k][1]), hi = __floats2bfloat162_rn(acc[k][2], acc[k][3]);
        uint2 w;
        w.x = *reinterpret_cast<uint32_t*>(&lo);
        w.y = *reinterpret_cast<uint32_t*>(&hi);
        *reinterpret_cast<uint2*>(&tile[row][(2 * k + g0) * 4]) = w;
    }
    __syncthreads();
    const int b = bh / NH, h = bh - b * NH;
    #pragma unroll
    for (int q = 0; q < 4; q++) {
        const int c = q * 256 + t, r = c >> 3, c8 = c & 7;
        const int tq = i * BT + r;
        if (tq < T)
            *reinterpret_cast<uint4*>(dqkv + (((size_t)b * T + tq) * 3) * NH * HS + (size_t)h * HS + c8 * 8) = *reinterpret_cast<const uint4*>(&tile[r][c8 * 8]);
    }
}

}  // namespace

// How many heads, the first ones, are dealt to CTAs whole (WHOLE_HEADS); the others are split into units over the CTAs and folded.
// Whole up to 10 tiles.  The CTAs' slots, 32 KB a tile, share L2 with the streams that pass by them: with 296 heads dQ costs 105 MB of memory traffic at 8 tiles
// (39 MB of slots), 423 at 10 (48 MB), 945 at 12 and 2377 at 16 (counted: bytes moved beyond the inputs and gradients), the split heads' slots, written
// and folded, at least 504, 776, 1106 and 1940.  us of all launches, split in brackets, B x T x heads: 64 x 1024 x 12 459 (523), 128 x 384 x 12 177 (278),
// 64 x 256 x 12 63 (85), 40 x 1152 x 12 390 (437), 32 x 1280 x 12 379 (396), 20 x 1536 x 12 345 (336), 16 x 2048 x 12 484 (459).
// Heads that do not fill the CTAs once more are split if that is shorter by more than what it costs: the fold, 4 pairs, or 2 where each CTA has one unit at most and the
// fold is small (12 x 640 x 8 37 whole, 38 split, 1 x 512 x 12 30.3, 25.9, 2 x 300 x 12 18.0, 16.8, 4 x 384 x 12 18.7, 17.9; 8 x 384 x 12, two units, 19.8, 27.0, and with two
// tiles, where nothing gets shorter, 4 x 256 x 12 13.0, 15.8), and next to whole heads a kernel of their own as well, 6 pairs (16 x 512 x 12 56.9 whole, 63.8 split,
// 16 x 300 x 12 31.9, 37.7).  With one full round of heads only, the split slots still fit into L2: 13 x 1024 x 12 127.5 in two kernels, 126.3 all split,
// 13 x 768 x 12 87.1, 85.2.
constexpr int WHOLE_TILES = 10, SPLIT_GAIN = 4, SPLIT_GAIN_ONCE = 2, SPLIT_GAIN_BESIDE = 6;
static int whole_heads(int heads, int nt, int sms) {
    if (nt < 2 || nt > WHOLE_TILES) return 0;
    const int rest = heads % sms, full = heads - rest, G = (nt + 1) / 2;
    const int gain = nt * (nt + 1) / 2 - CEIL_DIV(rest * G, sms) * (nt + 1);
    if (rest == 0 || gain < (full ? SPLIT_GAIN_BESIDE : rest * G <= sms ? SPLIT_GAIN_ONCE : SPLIT_GAIN)) return heads;
    return full >= 2 * sms ? full : 0;
}

// Profiling aid: with a device buffer of 4 * 8 * 64 int64 set here, CTA 0 of every later single-pass launch records clock64()
// stamps of its first 64 tile pairs (role 0 = issuer, 1 = first softmax warp, 2 = first drain warp; events in program
// order).  Null (the default) switches it off.
static long long* g_trace = nullptr;
extern "C" int llmc_attention_bwd_set_trace(long long* buf) { g_trace = buf; return 0; }

// number of fp32 words of workspace that llmc_attention_bwd needs (delta + the dQ contributions of the single-pass kernel)
extern "C" long long llmc_attention_bwd_workspace(int B, int T, int NH, int hs) {
    long long words = (long long)B * NH * T;                       // delta
    words = (words + 63) & ~63ll;
    if (hs == HS) {
        const long long nt = CEIL_DIV(T, BT);
        words += (long long)B * NH * slot_of((int)nt, (int)(nt + 1) / 2) * SLOT_FLOATS;
    }
    return words;
}

// dqkv (B,T,3,NH,HS) = gradient of causal attention; ws: llmc_attention_bwd_workspace(...) floats.  Head sizes: multiples of 8, 64..128.
extern "C" int llmc_attention_bwd(bf16* dqkv, float* ws, const bf16* dout, const bf16* qkv, const bf16* out, const float* lse,
                                  int B, int T, int NH, int hs, cudaStream_t stream) {
    if (hs != HS) return llmc_attention_bwd_two_pass(dqkv, ws, dout, qkv, out, lse, B, T, NH, hs, stream);
    if ((reinterpret_cast<uintptr_t>(ws) & 15u) != 0) return -1;
    float* delta = ws;
    float* dq_ws = ws + ((((long long)B * NH * T) + 63) & ~63ll);
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
    const int nt = CEIL_DIV(T, BT);
    // one tile per sequence: delta and the finished dQ come from the same launch (4 x 64 x 12 heads 19.5 -> 13.4 us)
    if (nt > 1 && (rc = llmc_attention_delta(delta, out, dout, B, T, NH, hs, stream))) return rc;
    Args a;
    a.dqkv = dqkv; a.dq_ws = dq_ws; a.lse = lse; a.delta = nt > 1 ? delta : nullptr; a.out = out; a.dout = dout; a.T = T; a.NH = NH;
    a.scale = 1.0f / sqrtf((float)hs);
    a.scale_log2e = a.scale * 1.4426950408889634f;
    a.status = llmc_status_ptr();
    a.trace = g_trace;
    int sms = llmc_device_sm_count(); if (sms <= 0) sms = 148;
    const int G = (nt + 1) / 2;
    static bool configured[3] = {false, false, false};
    auto launch = [&](auto kernel, int mode, int item0, int items) {
        if (!configured[mode]) { CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM)); configured[mode] = true; }
        const int grid = items - item0 < sms ? items - item0 : sms;
        a.item0 = item0; a.items = items;
        a.early = nt == 1 && grid < sms;       // as in the forward pass; with more tiles the kernels before and after are launched plainly
        if (a.early) { CUDA_CHECK(launch_pdl(kernel, dim3(grid), dim3(THREADS), SMEM, stream, 0, tmQKV, tmDO, tmDQKV, a)); return 0; }
        kernel<<<grid, THREADS, SMEM, stream>>>(tmQKV, tmDO, tmDQKV, a);
        CUDA_CHECK(cudaGetLastError());
        return 0;
    };
    const int whole = whole_heads(B * NH, nt, sms), rest = B * NH - whole;
    if (whole && (rc = launch(attn_bwd1_kernel<WHOLE_HEADS>, WHOLE_HEADS, 0, whole))) return rc;
    if (rest == 0) return 0;
    if (T <= SHORT_T || (T <= SHORT_T_MANY && rest > 2 * sms)) rc = launch(attn_bwd1_kernel<SHORT_SPLIT>, SHORT_SPLIT, whole * G, B * NH * G);
    else rc = launch(attn_bwd1_kernel<SPLIT>, SPLIT, whole * G, B * NH * G);
    if (rc || nt == 1) return rc;
    dq_fold_kernel<<<(unsigned)(rest * nt), 256, 0, stream>>>(dqkv, dq_ws, whole, T, NH, nt);
    CUDA_CHECK(cudaGetLastError());
    return 0;
}

// kernels that llmc_attention_bwd launches
extern "C" int llmc_attention_bwd_launches(int B, int T, int NH, int hs) {
    if (hs != HS) return 3;
    const int nt = CEIL_DIV(T, BT);
    if (nt <= 1) return 1;
    int sms = llmc_device_sm_count(); if (sms <= 0) sms = 148;
    const int whole = whole_heads(B * NH, nt, sms);
    return 1 + (whole > 0) + (whole < B * NH ? 2 : 0);
}
