// Causal flash attention forward for sm_100a, head size 64, on the packed (B, T, 3, NH, HS) QKV layout.
//
// A CTA works on TWO adjacent 128-row query tiles (slots A = 2p, B = 2p + 1) of one (batch, head) at a time and streams key / value tiles of 64 rows
// past both, so every K / V tile is loaded once for 256 queries.  TWO CTAs share an SM.
//
//   warp 0       TMA producer: the Q tiles of an item, each loaded again as soon as its slot's last score product is done, and K_0 V_0 K_1 V_1 ... through
//                a ring of six.
//   warps 1, 2   issuers of S_X = Q_X K_j^T (SS) and O_X += P_X V_j (TS: A = P_X in tensor memory), one warp for each slot X, with one elected lane
//                executing the tcgen05 instructions.
//   warps 4-7    softmax of tile A, warps 8-11 softmax of tile B: ONE THREAD PER QUERY ROW holding the row's 64 scores in
//                registers.  Row maximum and row sum need no exchange between threads; P goes back to tensor memory as bf16
//                (no shared-memory round trip, no proxy fence) over the scores it came from; S_X(j+1) is issued directly behind O_X += P_X(j) V, whose
//                completion it thereby reports.  O accumulates in tensor memory across the key tiles and is
//                rescaled by its own row's thread only when the running maximum grows by more than 2^8 (the stale maximum
//                is a valid reference point for the exponentials in between, the final division by the row sum cancels it).
//
// A slot is bound by its own chain: scores from tensor memory, maxima, exponentials (8 cycles of the special-function unit a warp), conversion, P back, two
// products, about 2000 cycles for 64 keys, of which the unit is busy for 450.  So four slots share an SM, each with an issuer of its own (one issuer for both
// slots took 1200 cycles a step), an item's Q tile arrives under the item before, and its output leaves from its own Q buffer.  Key tiles of 64 and the P-over-S
// overlay are what lets four slots into tensor memory and two CTAs into shared memory; the softmax loop is short enough for the instruction caches (with
// 128-column tiles and every branch unrolled a warp waited for instructions longer than for anything else).  A part of the exponentials runs on the
// FMA pipe (ex2_poly2): one pair of eight in the ordinary kernel (none / one / two: 177 / 171 / 175 us at 64 x 1024 x 12), two in DUO (none / one / two: 16.1 /
// 16.0 / 14.9 us at 1 x 777 x 32).
//
// DUO: where the query tiles are so few that SMs would get one chain only, a CTA works on ONE query tile, its slots on alternate key tiles, and adds the two
// at the end.  us, with the kernel this one replaces (one CTA of two slots per SM, tiles of 128 keys, slots taking turns at the exponentials) in brackets, in turn on one
// GPU, B x T x heads: 64 x 1024 x 12 175 (205), 2 x 4096 x 32 198 (233), 64 x 256 x 12 27.3 (35.9), 8 x 1024 x 12 28.6 (34.5); DUO 4 x 512 x 12 10.3 (11.0),
// 3 x 1000 x 16 19.1 (22.9), 1 x 2048 x 25 27.3 (41.7), 1 x 129 x 32 5.5 (7.0).  Where about half of the SMs get a second CTA, which then decides, DUO gains
// nothing: 1 x 777 x 32 14.7 (14.4), 4 x 512 x 16 11.5 (11.3).
//
// TMEM columns of a CTA: S_A [0,64)  O_A [64,128)  S_B [128,192)  O_B [192,256); P_X: the first 32 columns of S_X (64 bf16 per row)
//
// Statistics are written as natural-log LSE per (b, h, t), the layout cuDNN's SDPA uses in the reference
// (llmc/cudnn_att.cpp:105-113).  Output tiles leave through shared memory and TMA stores (rows past T are clipped).
// Head sizes above 64 use the kernel of attention_fwd.cu.
//
// Capability parity: attention_forward_cudnn (llmc/cudnn_att.cpp:222-254) and attention_forward of llmc/attention.cuh.
#include "common.cuh"
#include "decoder_ops.h"
#include "pdl.cuh"

int llmc_attn_qkv_map(CUtensorMap* tm, const bf16* qkv, int B, int T, int NH, int hs, int rows);   // attention_fwd.cu
int llmc_attention_fwd_general(bf16* out, float* lse, const bf16* qkv, int B, int T, int NH, int hs, cudaStream_t stream);

namespace {

constexpr int BT = 128;                             // query rows of a tile
constexpr int KT = 64;                              // keys of a tile
constexpr int HS = 64;
constexpr int TILE_BYTES = BT * HS * 2;             // 16 KB: one 128-byte-swizzled TMA box
constexpr int KV_BYTES = KT * HS * 2;               // 8 KB
constexpr int PAIRS = 3;                            // K / V tile pairs in flight
constexpr int RING = 2 * PAIRS;
constexpr int THREADS = 384;                        // TMA warp, two issuer warps, an idle one, 2 x 4 softmax warps
constexpr int REGS_LOW = 48, REGS_HIGH = 96;        // of 80 at launch (two CTAs): 4 x 48 + 8 x 96 = 12 x 80
constexpr int REGS_LAUNCH = (4 * REGS_LOW + 8 * REGS_HIGH) / 12;
static_assert(12 * REGS_LAUNCH == 4 * REGS_LOW + 8 * REGS_HIGH, "the shares of the warps add up to what a block is launched with");
constexpr int TMEM_COLS = 256;
constexpr int SMEM = 4 * TILE_BYTES + RING * KV_BYTES + 256;      // two Q / output tiles of each slot, K/V ring
static_assert(2 * (SMEM + 1024) <= 228 * 1024, "two CTAs share an SM");
constexpr float RESCALE_LOG2 = 8.0f;                // the running maximum may lag by this much (in log2 units of the scaled scores)

struct Args {
    float* lse;        // (B, NH, T)
    int T, NH, BH;
    float scale_log2e; // (1/sqrt(HS)) * log2(e)
    float scale;
    int early;           // the next kernel may start while this one runs
    unsigned int* status;
};

// The items of one CTA.  Ordinarily query-tile pair p of a head, late (heavy) pairs first; the slots take the longer tile of a pair in turn.  DUO: one query
// tile (p) for both slots, slot 0 with its even key tiles and slot 1 with the odd ones.
template <bool DUO>
struct Items {
    int w, grid, total, BH, np, NH, nq, nk;
    int p, b, h, flip;
    DEVINL Items(int cta, int grid_, const Args& a) : w(cta), grid(grid_), BH(a.BH), NH(a.NH) {
        nq = CEIL_DIV(a.T, BT); nk = CEIL_DIV(a.T, KT); np = DUO ? nq : (nq + 1) >> 1; total = BH * np;
        p = b = h = flip = 0;
        if (w < total) item();
    }
    DEVINL bool valid() const { return w < total; }
    DEVINL void item() { const int rank = w / BH, bh = w - rank * BH; p = np - 1 - rank; b = bh / NH; h = bh - b * NH; }
    DEVINL void next() { w += grid; flip ^= 1; if (w < total) item(); }
    DEVINL int qtile(int x) const { return DUO ? p : 2 * p + (x ^ flip); }                             // query tile of slot x
    DEVINL int kv_tiles() const { return min(2 * (DUO ? p : min(2 * p + 1, nq - 1)) + 2, nk); }        // key tiles of the item
    DEVINL int tiles(int x) const {                                                                    // and of slot x: STEP * i + (DUO ? x : 0)
        return DUO ? (kv_tiles() + 1 - x) >> 1 : qtile(x) < nq ? min(2 * qtile(x) + 2, nk) : 0;
    }
    static constexpr int STEP = DUO ? 2 : 1;
};

template <bool DUO>
__global__ void __launch_bounds__(THREADS, 2)
attn_fwd1_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmKV, const __grid_constant__ CUtensorMap tmOut, const Args a) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sQ = smem;                                   // [A, B][2]: Q of an item, then its output on the way out; the next item's Q meanwhile in the other
    uint8_t* sKV = sQ + 4 * TILE_BYTES;                   // [RING]
    uint64_t* bars = reinterpret_cast<uint64_t*>(sKV + RING * KV_BYTES);
    uint64_t* q_full = bars + 0;      // [2 slots][2 buffers]
    uint64_t* q_empty = bars + 4;     // [2][2] the output has left the buffer                  (1 arrival)
    uint64_t* s_full = bars + 8;      // [2] S_X(t) complete, and with it every earlier product (1 commit)
    uint64_t* p_ready = bars + 10;    // [2] P_X(t) is in TMEM (and O_X rescaled if needed)     (4 arrivals)
    uint64_t* o_full = bars + 12;     // [2] the item's O_X is complete                         (1 commit)
    uint64_t* o_free = bars + 14;     // [2] the slot's warps have read O_X                     (4 arrivals)
    uint64_t* kv_full = bars + 16;    // [RING] K_0 V_0 K_1 V_1 ...
    uint64_t* kv_empty = kv_full + RING;      // both slots are done with the tile, or have no use for it
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(kv_empty + RING);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = warp_index(), lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        if ((smem_u32(smem) & 1023u) != 0) record_error(a.status, ST_BAD_ARG, 0x18);
        for (int i = 0; i < 4; i++) { mbar_init(&q_full[i], 1); mbar_init(&q_empty[i], 1); }
        for (int i = 0; i < 2; i++) {
            mbar_init(&s_full[i], 1); mbar_init(&p_ready[i], 4); mbar_init(&o_full[i], 1); mbar_init(&o_free[i], 4);
        }
        for (int i = 0; i < RING; i++) { mbar_init(&kv_full[i], 1); mbar_init(&kv_empty[i], 2); }
        *abort_flag = 0;
        mbar_fence_init();
        tma_prefetch_desc(&tmQ); tma_prefetch_desc(&tmKV); tma_prefetch_desc(&tmOut);
    }
    if (warp == 1) { tmem_alloc(tmem_slot, TMEM_COLS); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_wait();
    if (a.early) pdl_trigger();

    Items<DUO> im(blockIdx.x, gridDim.x, a);

    if (warp < 4) {
        regs_shrink<REGS_LOW>();
        if (warp == 0) {
        // ---------------------------------------------------------------- TMA producer, per item: Q_A Q_B K_0 V_0 K_1 V_1 ...
        if (lane == 0) {
            uint32_t st = 0, ph = 1;
            uint32_t nx[2] = {0, 0};           // items of each slot so far
            bool ok = true;
            for (; im.valid() && ok; im.next()) {
                const int nkv = im.kv_tiles();
                #pragma unroll
                for (int x = 0; x < 2; x++) {
                    if (!ok || im.tiles(x) == 0) continue;
                    const uint32_t q = 2 * x + (nx[x] & 1);
                    ok = mbar_wait_relaxed(&q_empty[q], ((nx[x] >> 1) & 1) ^ 1, abort_flag, a.status, 0x502);
                    if (!ok) break;
                    mbar_expect_tx(&q_full[q], TILE_BYTES);
                    tma_load_4d(sQ + q * TILE_BYTES, &tmQ, &q_full[q], 0, im.h, im.qtile(x) * BT, im.b);       // zeros past T
                    nx[x]++;
                }
                for (int j = 0; j < 2 * nkv && ok; j++) {
                    ok = mbar_wait_relaxed(&kv_empty[st], ph, abort_flag, a.status, 0x500);
                    if (!ok) break;
                    mbar_expect_tx(&kv_full[st], KV_BYTES);
                    tma_load_4d(sKV + st * KV_BYTES, &tmKV, &kv_full[st], 0, (1 + (j & 1)) * a.NH + im.h, (j >> 1) * KT, im.b);
                    if (++st == RING) { st = 0; ph ^= 1; }
                }
            }
        }
        } else if (warp < 3) {
        // ---------------------------------------------------------------- issuer of slot x, per item: S(0), then for every key tile j  O += P(j) V_j, S(j+1).
        // A chain of short waits and few instructions; one warp for both slots left each waiting for the other's (1200 cycles a step).
        const int x = warp - 1;
        const bool leader = elect_one();
        constexpr uint32_t idesc_s = umma_idesc_bf16(BT, KT, 0, 0);      // Q (K-major) x K (K-major)
        constexpr uint32_t idesc_o = umma_idesc_bf16(BT, HS, 0, 1);      // P (TMEM) x V (N-major)
        constexpr uint32_t KV_UNITS = KV_BYTES / 16;
        const uint64_t dQ0 = umma_desc_sw128(smem_u32(sQ + 2 * x * TILE_BYTES), 16, 1024);
        const uint64_t dK0 = umma_desc_sw128(smem_u32(sKV), 16, 1024), dV0 = umma_desc_sw128(smem_u32(sKV + KV_BYTES), KV_BYTES, 1024);
        const uint32_t tS = tmem_base + x * 128, tO = tS + 64;
        uint32_t st = 0, ph = 0;          // of the K / V pair j
        uint32_t t = 0, it = 0;           // tiles and items of this slot so far
        bool ok = true;
        auto issue_s = [&](uint64_t q, uint32_t st) {
            const uint64_t k = dK0 + st * (2 * KV_UNITS);
            #pragma unroll
            for (int kk = 0; kk < HS / 16; kk++) umma_ss(tS, q + 2 * kk, k + 2 * kk, idesc_s, kk > 0);
            umma_commit(&s_full[x]);
            umma_commit(&kv_empty[2 * st]);
        };
        for (; im.valid() && ok; im.next()) {
            const int n = im.tiles(x), nkv = im.kv_tiles();
            const uint64_t q = dQ0 + (it & 1) * (TILE_BYTES / 16);
            int i = 0;                    // tiles of this slot in the item so far
            for (int j = 0; j < nkv && ok; j++) {
                if (j == (DUO ? x : 0) && n > 0) {
                    ok = mbar_wait_relaxed(&q_full[2 * x + (it & 1)], (it >> 1) & 1, abort_flag, a.status, 0x510) && mbar_wait_relaxed(&kv_full[2 * st], ph, abort_flag, a.status, 0x511);
                    if (!ok) break;
                    tc_fence_after();
                    if (leader) issue_s(q, st);
                }
                if (DUO ? (j & 1) == x : j < n) {
                    const uint32_t sn = st + Items<DUO>::STEP, st1 = sn >= PAIRS ? sn - PAIRS : sn, ph1 = sn >= PAIRS ? ph ^ 1 : ph;      // of this slot's next tile
                    // the tiles first, P last: what follows its arrival is the chain of the slot
                    ok = mbar_wait_relaxed(&kv_full[2 * st + 1], ph, abort_flag, a.status, 0x515);
                    if (ok && i + 1 < n) ok = mbar_wait_relaxed(&kv_full[2 * st1], ph1, abort_flag, a.status, 0x516);
                    if (ok && i == 0 && it > 0) ok = mbar_wait_relaxed(&o_free[x], (it - 1) & 1, abort_flag, a.status, 0x517);
                    ok = ok && mbar_wait_relaxed(&p_ready[x], t & 1, abort_flag, a.status, 0x514);
                    if (!ok) break;
                    tc_fence_after();
                    const uint64_t v = dV0 + st * (2 * KV_UNITS);
                    if (leader) {
                        // A = P in TMEM (16 keys = 8 columns per step), B = V N-major (16 rows = 2048 bytes per step)
                        #pragma unroll
                        for (int kk = 0; kk < KT / 16; kk++) umma_ts(tO, tS + kk * 8, v + 128 * kk, idesc_o, i > 0 || kk > 0);
                        if (i + 1 < n) issue_s(q, st1); else umma_commit(&o_full[x]);
                        umma_commit(&kv_empty[2 * st + 1]);
                    }
                    t++; i++;
                } else {
                    // a tile that only the other slot reads; its buffer is not given back before it has been filled
                    ok = mbar_wait_relaxed(&kv_full[2 * st], ph, abort_flag, a.status, 0x512);
                    if (ok && leader) mbar_arrive(&kv_empty[2 * st]);
                    ok = ok && mbar_wait_relaxed(&kv_full[2 * st + 1], ph, abort_flag, a.status, 0x513);
                    if (ok && leader) mbar_arrive(&kv_empty[2 * st + 1]);
                }
                if (++st == PAIRS) { st = 0; ph ^= 1; }
            }
            if (n > 0) it++;
        }
        __syncwarp();
        }
    } else {
        regs_grow<REGS_HIGH>();
        // ---------------------------------------------------------------- softmax of slot x: thread = query row r of the slot's tile
        const int x = (warp - 4) >> 2;
        const int q4 = warp & 3;                           // the warp's quarter of the tensor memory lanes
        const int r = q4 * 32 + lane;
        const uint32_t lane_off = (uint32_t)(q4 * 32) << 16;
        const uint32_t tS = tmem_base + x * 128 + lane_off, tO = tS + 64;
        const bool issuer = q4 == 0 && lane == 0;          // the thread of the slot that issues its output store
        const float c = a.scale_log2e;
        bool ok = true;
        uint32_t t = 0;                                    // tiles of this slot so far
        uint32_t it = 0;                                   // items of this slot so far
        for (; im.valid(); im.next()) {
            const int nj = im.tiles(x);
            if (!DUO && nj == 0) continue;                 // (uniform for the slot) no second tile in this item
            const int qi = im.qtile(x);                    // this slot's query tile
            const int jd = 2 * qi + (q4 >> 1);             // the key tile on this warp's diagonal: none of the later ones is seen
            float m = -INFINITY, l = 0.f;                  // reference maximum (raw score units) and row sum relative to it
            // Tiles that move the reference however little their maximum is above it.  The largest probability of a row, which alone is exact in bf16 where it is 1,
            // is more often 1 with a maximum over 128 keys than over 64: error of O against 64 bits at 12 x 700 x 16 0.002010 and 0.002034 (0.002017 in the kernel
            // before, which took tiles of 128 keys).  Two slots on a row have a reference each: 1 x 777 x 32 0.002006 with 64 keys (0.002022).
            constexpr int FIRST_TILES = DUO ? 1 : 2;
            #pragma unroll 1
            for (int i = 0; i < nj; i++, t++) {
                const int j = Items<DUO>::STEP * i + (DUO ? x : 0);
                ok = mbar_wait(&s_full[x], t & 1, abort_flag, a.status, 0x520 + x) && ok;
                tc_fence_after();
                uint32_t pk[32];
                if (j <= jd) {
                    uint32_t sv[64];
                    tmem_ld32(tS, sv);
                    tmem_ld32(tS + 32, sv + 32);
                    tmem_ld_wait();
                    if (j == jd) {
                        // -inf above the diagonal, which crosses the first 32 columns for even quarters and the others for odd ones
                        if (q4 & 1) {
                            #pragma unroll
                            for (int e = 0; e < 32; e++) if (e > lane) sv[32 + e] = 0xff800000u;
                        } else {
                            #pragma unroll
                            for (int e = 0; e < 32; e++) { if (e > lane) sv[e] = 0xff800000u; sv[32 + e] = 0xff800000u; }
                        }
                    }
                    float mx4[4];
                    #pragma unroll
                    for (int e = 0; e < 4; e++) mx4[e] = fmaxf(__uint_as_float(sv[2 * e]), __uint_as_float(sv[2 * e + 1]));
                    #pragma unroll
                    for (int e = 8; e < 64; e += 2) mx4[(e >> 1) & 3] = max3(mx4[(e >> 1) & 3], __uint_as_float(sv[e]), __uint_as_float(sv[e + 1]));
                    const float mx = max3(fmaxf(mx4[0], mx4[1]), mx4[2], mx4[3]);
                    // move the reference maximum only when it lags by more than 2^RESCALE_LOG2 or is that of the first tiles (decided per warp, so that
                    // the TMEM accesses stay warp-wide); a moved maximum rescales the row sum and the row of O_X
                    const bool grow = (mx - m) * c > RESCALE_LOG2 || i < FIRST_TILES;
                    if (__any_sync(0xffffffffu, grow)) {
                        const float m_new = fmaxf(m, mx);
                        const float alpha = m == m_new ? 1.0f : ex2_fast((m - m_new) * c);      // (-inf - -inf while a row has seen no score above -inf)
                        l *= alpha;
                        m = m_new;
                        if (i > 0) {                       // O_X(t-1) is complete: its product was issued ahead of S_X(t)
                            #pragma unroll 1
                            for (int g = 0; g < 64; g += 16) {
                                uint32_t ov[16];
                                tmem_ld16(tO + g, ov);
                                tmem_ld_wait();
                                #pragma unroll
                                for (int e = 0; e < 16; e++) ov[e] = __float_as_uint(__uint_as_float(ov[e]) * alpha);
                                tmem_st16(tO + g, ov);
                            }
                        }
                    }
                    const float moff = m == -INFINITY ? 0.f : m * c;         // probabilities of 0, not of -inf - -inf
                    const uint64_t c2 = f2_both(c), off2 = f2_both(-moff);
                    uint64_t rs0 = 0, rs1 = 0;
                    #pragma unroll
                    for (int e = 0; e < 64; e += 2) {
                        const uint64_t x2 = f2_fma(f2_pack_u(sv[e], sv[e + 1]), c2, off2);
                        float2 p;
                        if (((e >> 1) & 7) < (DUO ? 2 : 1)) {              // one or two of eight pairs on the FMA pipe
                            p = ex2_poly2(x2);
                        } else {
                            p = f2_unpack(x2);
                            p.x = ex2_fast(p.x); p.y = ex2_fast(p.y);
                        }
                        if (e & 2) rs1 = f2_add(rs1, f2_pack(p.x, p.y)); else rs0 = f2_add(rs0, f2_pack(p.x, p.y));
                        pk[e >> 1] = pack_bf16x2(p.x, p.y);
                    }
                    const float2 rs = f2_unpack(f2_add(rs0, rs1));
                    l += rs.x + rs.y;
                } else {
                    #pragma unroll
                    for (int e = 0; e < 32; e++) pk[e] = 0;
                }
                tmem_st32(tS, pk);                          // over this row's own scores
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&p_ready[x]);
                // the output of the item before has left its buffer long ago: the Q tile of the next item may come
                if (!DUO && i == 0 && it > 0 && issuer) { tma_store_wait_read<0>(); mbar_arrive(&q_empty[2 * x + ((it - 1) & 1)]); }
            }
            // ---- item epilogue: O_X / l -> bf16 tile in the layout of a 128-byte-swizzled TMA box -> one bulk store
            if (nj > 0) ok = mbar_wait(&o_full[x], it & 1, abort_flag, a.status, 0x528 + x) && ok;
            tc_fence_after();
            // DUO: slot 1 leaves its sums, its maximum and its row sum in shared memory (over its own Q buffers and slot 0's second one, which a
            // block of one item does not use); slot 0 adds them to its own
            float* other = reinterpret_cast<float*>(sQ + 2 * TILE_BYTES);               // [channel][row]
            float* other_ml = reinterpret_cast<float*>(sQ + TILE_BYTES);                // [max, sum][row]
            float mine = 1.0f, theirs = 0.0f;
            if (DUO) {
                if (x == 1) {
                    #pragma unroll 1
                    for (int g = 0; g < 64; g += 16) {
                        uint32_t ov[16];
                        if (nj > 0) { tmem_ld16(tO + g, ov); tmem_ld_wait(); }
                        #pragma unroll
                        for (int e = 0; e < 16; e++) other[(g + e) * BT + r] = nj > 0 ? __uint_as_float(ov[e]) : 0.f;
                    }
                    other_ml[r] = m;
                    other_ml[BT + r] = l;
                }
                asm volatile("bar.sync 3, 256;" ::: "memory");
                if (x == 1) break;
                const float mo = other_ml[r], m_new = fmaxf(m, mo);      // slot 1 may have seen none of this row's keys
                mine = ex2_fast((m - m_new) * c);
                theirs = ex2_fast((mo - m_new) * c);
                l = l * mine + other_ml[BT + r] * theirs;
                m = m_new;
            }
            if (m == -INFINITY) l = NAN;                   // no score above -inf: no softmax
            const float inv = 1.0f / l;
            uint8_t* otile = sQ + (2 * x + (it & 1)) * TILE_BYTES;     // over the item's Q tile, which its last score product has read
            uint8_t* orow = otile + r * 128;
            #pragma unroll 1
            for (int half = 0; half < 2; half++) {
                uint32_t ov[32];
                tmem_ld32(tO + half * 32, ov);
                tmem_ld_wait();
                if (DUO) {
                    #pragma unroll
                    for (int e = 0; e < 32; e++) ov[e] = __float_as_uint(__uint_as_float(ov[e]) * mine + other[(half * 32 + e) * BT + r] * theirs);
                }
                #pragma unroll
                for (int u = 0; u < 4; u++) {
                    uint4 o;
                    o.x = pack_bf16x2(__uint_as_float(ov[8 * u]) * inv, __uint_as_float(ov[8 * u + 1]) * inv);
                    o.y = pack_bf16x2(__uint_as_float(ov[8 * u + 2]) * inv, __uint_as_float(ov[8 * u + 3]) * inv);
                    o.z = pack_bf16x2(__uint_as_float(ov[8 * u + 4]) * inv, __uint_as_float(ov[8 * u + 5]) * inv);
                    o.w = pack_bf16x2(__uint_as_float(ov[8 * u + 6]) * inv, __uint_as_float(ov[8 * u + 7]) * inv);
                    *reinterpret_cast<uint4*>(orow + (((half * 4 + u) ^ (r & 7)) * 16)) = o;
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&o_free[x]);            // O_X may be overwritten by the next item's first product
            fence_async_smem();
            asm volatile("bar.sync %0, 128;" ::"r"(1 + x) : "memory");
            if (issuer && ok) {
                tma_store_4d(&tmOut, otile, 0, im.h, qi * BT, im.b);
                tma_store_commit();
            }
            it++;
            const int trow = qi * BT + r;
            if (trow < a.T && ok) a.lse[((size_t)im.b * a.NH + im.h) * a.T + trow] = m * a.scale + logf(l);
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

// out (B,T,NH,HS) = causal softmax(Q K^T / sqrt(HS)) V ; lse (B,NH,T) fp32.  Head sizes: multiples of 8 from 64 to 128.
extern "C" int llmc_attention_fwd(bf16* out, float* lse, const bf16* qkv, int B, int T, int NH, int hs, cudaStream_t stream) {
    if (hs != HS) return llmc_attention_fwd_general(out, lse, qkv, B, T, NH, hs, stream);
    CUtensorMap tmQ, tmKV, tmOut;
    int rc = llmc_attn_qkv_map(&tmQ, qkv, B, T, NH, hs, BT);
    if (!rc) rc = llmc_attn_qkv_map(&tmKV, qkv, B, T, NH, hs, KT);
    if (rc) return rc;
    {
        uint64_t dims[4] = {(uint64_t)hs, (uint64_t)NH, (uint64_t)T, (uint64_t)B};
        uint64_t strides[4] = {2, (uint64_t)hs * 2, (uint64_t)NH * hs * 2, (uint64_t)T * NH * hs * 2};
        uint32_t box[4] = {64, 1, 128, 1};
        if ((rc = llmc_get_tensormap(&tmOut, out, 2, 4, dims, strides, box, 3))) return rc;
    }
    Args a;
    a.lse = lse; a.T = T; a.NH = NH; a.BH = B * NH;
    a.scale = 1.0f / sqrtf((float)hs);
    a.scale_log2e = a.scale * 1.4426950408889634f;
    a.status = llmc_status_ptr();
    const int nq = CEIL_DIV(T, BT);
    int sms = llmc_device_sm_count(); if (sms <= 0) sms = 148;
    // us, pairs / DUO, query tiles per SM in brackets: 8 x 300 x 12 (1.9) 10.3 / 9.8, 3 x 1000 x 16 (2.6) 23.0 / 19.6, 1 x 2048 x 25 (2.7) 39.3 / 27.7, but
    // 16 x 256 x 16 (3.5) 11.1 / 17.1, 8 x 1024 x 12 (5.2) 29.4 / 37.1
    const bool duo = (long long)B * NH * nq <= 3 * sms && T > KT;
    const int total = B * NH * (duo ? nq : (nq + 1) / 2);
    const int grid = duo || total < 2 * sms ? total : 2 * sms;
    auto kernel = duo ? attn_fwd1_kernel<true> : attn_fwd1_kernel<false>;
    static bool configured[2] = {false, false};
    if (!configured[duo]) {
        // a block compiled to fewer registers would wait for its larger shares for good
        cudaFuncAttributes attr;
        CUDA_CHECK(cudaFuncGetAttributes(&attr, kernel));
        if (attr.numRegs < REGS_LAUNCH) { fprintf(stderr, "[llmc_b200] attention: compiled to %d registers, %d expected\n", attr.numRegs, REGS_LAUNCH); return -1; }
        CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
        configured[duo] = true;
    }
    // early launch (pdl.cuh) only where SMs have room for another block: a prefill of 777 tokens (224 blocks) 617 -> 607 us; otherwise the blocks of the next
    // kernel sit beside this one's for all of its run (64 x 1024 x 12, forward and backward, in the kernels before this one: 938 -> 986 us)
    a.early = grid < 2 * sms;
    if (a.early) {
        CUDA_CHECK(launch_pdl(kernel, dim3(grid), dim3(THREADS), SMEM, stream, 0, tmQ, tmKV, tmOut, a));
        return 0;
    }
    kernel<<<grid, THREADS, SMEM, stream>>>(tmQ, tmKV, tmOut, a);
    CUDA_CHECK(cudaGetLastError());
    return 0;
}
