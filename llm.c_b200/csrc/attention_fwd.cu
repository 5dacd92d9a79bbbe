// Causal flash attention forward for sm_100a on the packed (B, T, 3, NH, HS) QKV layout, head sizes 72..128 (multiples of 8; a
// narrower head runs as a 128-wide one whose missing channels TMA fills with zeros, with the products cut to whole 16-channel steps).
//
// The scheme of the 64-wide kernel (attention_fwd1.cu): a CTA works on TWO adjacent 128-row query tiles (slots A = 2p, B = 2p + 1) of
// one head and streams the key / value tiles 0..2p+1 past both; one softmax thread owns a whole row of 128 scores in registers; P goes
// back to tensor memory as bf16 and is the A operand of O += P V; O stays in tensor memory and is rescaled when the running maximum of a
// row of the warp has moved.  What 128 channels change:
//   * S and O of both slots take all 512 TMEM columns, so P_X(t) overwrites the scores S_X(t) it came from, and S_X(t+1) is issued
//     directly behind O_X += P_X(t) V (program order keeps it from overwriting P).  A slot therefore alternates between its softmax
//     and its products; the other slot's products fill the tensor pipe meanwhile.
//   * K and V tiles (32 KB each) share one three-stage ring, and the Q tiles are single-buffered, each released by its slot's last
//     score product: the next item's Q tile arrives while that slot finishes its last softmax and its epilogue.
// Bound by the softmax of the two slots (1024 exponential cycles per 128 x 128 tile each) with the tensor pipe right behind (2 x 1024
// cycles per key tile).  Measured, with the kernel this one replaces (16 softmax warps exchanging row statistics, P through shared
// memory) in brackets: B=16 T=2048 NH=8 HS=128 166 us (256), B=2 T=4096 NH=32 HS=128 280 us (422), B=3 T=1000 NH=32 HS=80 39 us (68).
// Letting the maximum lag by up to 2^8, as the 64-wide kernel does, took 167 / 274 / 44 us where this took 178 / 296 / 47, but then the largest probability of a row is not 1
// and is rounded to bf16 like the others: the error against 64 bits grows by 1 % (0.00200 -> 0.00204 on the last case).
// Handing P over in two halves, so that the product starts under the second half's exponentials, was slower than that (174 / 281 us).
//
// Items are dealt to the persistent CTAs heaviest first in alternating direction, which evens out their decreasing lengths.
//
// TMEM columns: S_A [0,128)  S_B [128,256)  O_A [256,384)  O_B [384,512);  P_X: the first 64 columns of S_X (128 bf16 per row)
//
// Statistics are written as natural-log LSE per (b, h, t), the layout cuDNN's SDPA uses in the reference (llmc/cudnn_att.cpp:105-113).
// Capability parity: attention_forward_cudnn (llmc/cudnn_att.cpp:222-254) and attention_forward of llmc/attention.cuh.
#include "common.cuh"

namespace {

constexpr int BT = 128;
constexpr int CHUNK_BYTES = BT * 64 * 2;            // 16 KB: 128 rows x 64 channels, one 128-byte-swizzled TMA box
constexpr int TILE_BYTES = 2 * CHUNK_BYTES;
constexpr int RING = 3;                             // K_0 V_0 K_1 V_1 ... tiles in flight
constexpr int THREADS = 384;                        // TMA warp, issuer warp, two idle warps, 2 x 4 softmax warps
constexpr int TMEM_COLS = 512;
constexpr int SMEM = 2 * TILE_BYTES + RING * TILE_BYTES + 2 * TILE_BYTES + 256;     // Q, K/V ring, two output tiles
static_assert(SMEM <= 232448, "shared memory of one CTA");
constexpr long long SKEW_CYCLES = 1200;

struct Args {
    float* lse;        // (B, NH, T)
    int T, NH, BH;
    int ks;            // 16-channel steps of the head: ceil(hs / 16)
    float scale_log2e; // (1/sqrt(HS)) * log2(e)
    float scale;
    unsigned int* status;
};

// The items of one CTA: query-tile pair p of a head, late (heavy) pairs first.
struct Items {
    int round, cta, grid, total, BH, np, NH, nq;
    int w, p, b, h;
    DEVINL void start(int cta_, int grid_, int BH_, int nq_, int NH_) {
        cta = cta_; grid = grid_; BH = BH_; nq = nq_; np = (nq_ + 1) >> 1; NH = NH_; total = BH * np; round = 0;
        p = b = h = 0;
        w = cta;
        if (w < total) item();
    }
    DEVINL bool valid() const { return w < total; }
    DEVINL void item() { const int rank = w / BH, bh = w - rank * BH; p = np - 1 - rank; b = bh / NH; h = bh - b * NH; }
    DEVINL void next() {
        round++;
        w = round * grid + ((round & 1) ? grid - 1 - cta : cta);
        if (w < total) item();
    }
    DEVINL bool has_b() const { return 2 * p + 1 < nq; }
    DEVINL int tiles(int x) const { return x == 0 ? 2 * p + 1 : (has_b() ? 2 * p + 2 : 0); }      // key tiles of slot x
    DEVINL int kv_tiles() const { return has_b() ? 2 * p + 2 : 2 * p + 1; }
};

__global__ void __launch_bounds__(THREADS, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tmQKV, const __grid_constant__ CUtensorMap tmOut, const Args a) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* sQ = smem;                                   // [A, B]
    uint8_t* sKV = sQ + 2 * TILE_BYTES;                   // [RING]
    uint8_t* sO = sKV + RING * TILE_BYTES;                // [A, B] output tiles on their way out
    uint64_t* bars = reinterpret_cast<uint64_t*>(sO + 2 * TILE_BYTES);
    uint64_t* q_full = bars + 0;      // [2 slots]
    uint64_t* q_empty = bars + 2;     // [2] the slot's last S of the item is complete          (1 commit)
    uint64_t* kv_full = bars + 4;     // [3]
    uint64_t* kv_empty = bars + 7;    // [3]
    uint64_t* s_full = bars + 10;     // [2] S_X(t) complete, and with it every earlier product (1 commit)
    uint64_t* p_ready = bars + 12;    // [2] P_X(t) is in TMEM (and O_X rescaled if needed)     (4 arrivals)
    uint64_t* o_full = bars + 14;     // [2] the item's O_X is complete                         (1 commit)
    uint64_t* o_free = bars + 16;     // [2] the slot's warps have read O_X                     (4 arrivals)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 18);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const int nq = CEIL_DIV(a.T, BT);

    if (threadIdx.x == 0) {
        if ((smem_u32(smem) & 1023u) != 0) record_error(a.status, ST_BAD_ARG, 0x18);
        for (int i = 0; i < 2; i++) {
            mbar_init(&q_full[i], 1); mbar_init(&q_empty[i], 1);
            mbar_init(&s_full[i], 1); mbar_init(&p_ready[i], 4); mbar_init(&o_full[i], 1); mbar_init(&o_free[i], 4);
        }
        for (int i = 0; i < RING; i++) { mbar_init(&kv_full[i], 1); mbar_init(&kv_empty[i], 1); }
        *abort_flag = 0;
        mbar_fence_init();
        tma_prefetch_desc(&tmQKV); tma_prefetch_desc(&tmOut);
    }
    if (warp == 1) { tmem_alloc(tmem_slot, TMEM_COLS); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    Items im;
    im.start(blockIdx.x, gridDim.x, a.BH, nq, a.NH);

    if (warp == 0) {
        // ---------------------------------------------------------------- TMA producer
        if (lane == 0) {
            auto load = [&](uint8_t* dst, uint64_t* bar, int head, int tile, int b) {
                mbar_expect_tx(bar, TILE_BYTES);
                tma_load_4d(dst, &tmQKV, bar, 0, head, tile * BT, b);
                tma_load_4d(dst + CHUNK_BYTES, &tmQKV, bar, 64, head, tile * BT, b);
            };
            uint32_t n = 0;                    // ring tiles so far
            uint32_t nx[2] = {0, 0};           // items of each slot so far
            bool fail = false;
            for (; im.valid() && !fail; im.next()) {
                const int nkv = im.kv_tiles();
                for (int j = 0; j < nkv && !fail; j++) {
                    if (j == 0) {
                        for (int x = 0; x < (im.has_b() ? 2 : 1) && !fail; x++) {
                            if (!mbar_wait_relaxed(&q_empty[x], (nx[x] & 1) ^ 1, abort_flag, a.status, 0x502)) { fail = true; break; }
                            load(sQ + x * TILE_BYTES, &q_full[x], im.h, 2 * im.p + x, im.b);
                            nx[x]++;
                        }
                    }
                    for (int kv = 0; kv < 2 && !fail; kv++, n++) {
                        const uint32_t st = n % RING;
                        if (!mbar_wait_relaxed(&kv_empty[st], ((n / RING) & 1) ^ 1, abort_flag, a.status, 0x500)) { fail = true; break; }
                        load(sKV + st * TILE_BYTES, &kv_full[st], (kv + 1) * a.NH + im.h, j, im.b);
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ---------------------------------------------------------------- issuer: per item  S_A(0) S_B(0), then for every key tile j
        // O_A += P_A(j) V_j, S_A(j+1), O_B += P_B(j) V_j, S_B(j+1); slot B's last two steps have the next item's S_A(0) between them
        const bool leader = elect_one();
#define WAIT_ALL(bar, parity, code) (__all_sync(0xffffffffu, mbar_wait_relaxed(bar, parity, abort_flag, a.status, code)) != 0)
        constexpr uint32_t idesc_s = umma_idesc_bf16(BT, BT, 0, 0);                             // Q (K-major) x K (K-major)
        const uint32_t idesc_o = umma_idesc_bf16(BT, 0, 0, 1) | ((uint32_t)(a.ks * 2) << 17);   // P (TMEM) x V (N-major), N = 16 ks
        constexpr uint32_t TILE_UNITS = TILE_BYTES / 16, CHUNK_UNITS = CHUNK_BYTES / 16;
        const uint64_t dQ0 = umma_desc_sw128(smem_u32(sQ), 16, 1024), dK0 = umma_desc_sw128(smem_u32(sKV), 16, 1024);
        const uint64_t dV0 = umma_desc_sw128(smem_u32(sKV), CHUNK_BYTES, 1024);
        const int ks = a.ks;
        uint32_t tp[2] = {0, 0};          // P V products issued per slot
        uint32_t qn[2] = {0, 0};          // Q tiles (items) whose first S has been issued per slot
        uint32_t on[2] = {0, 0};          // items whose first P V has been issued per slot
        uint32_t kabs = 0;                // key tiles of earlier items: K_j sits at ring position 2 (kabs + j), V_j behind it
        bool ok = true;
        auto kv_wait = [&](uint32_t pos, uint32_t code) { return WAIT_ALL(&kv_full[pos % RING], (pos / RING) & 1, code); };
        // S_x of the key tile at ring position pos; first: the slot's Q tile is new; the slot that reads a K tile last releases it
        auto issue_s = [&](int x, uint32_t pos, bool first, bool release_k, bool last) {
            bool good = true;
            if (first) good = WAIT_ALL(&q_full[x], qn[x]++ & 1, 0x510);
            good = good && kv_wait(pos, 0x511);
            if (!good) return false;
            tc_fence_after();
            const uint64_t q = dQ0 + (uint32_t)x * TILE_UNITS, k = dK0 + (pos % RING) * TILE_UNITS;
            if (leader) {
                #pragma unroll
                for (int kk = 0; kk < 8; kk++)
                    if (kk < ks)
                        umma_ss(tmem_base + x * 128, q + (kk >> 2) * CHUNK_UNITS + (kk & 3) * 2, k + (kk >> 2) * CHUNK_UNITS + (kk & 3) * 2, idesc_s, kk > 0);
                umma_commit(&s_full[x]);
                if (release_k) umma_commit(&kv_empty[pos % RING]);
                if (last) umma_commit(&q_empty[x]);
            }
            return true;
        };
        // O_x += P_x V: A = P_x in TMEM (16 keys = 8 columns per step), B = V N-major (16 rows = 2048 bytes per step)
        auto issue_pv = [&](int x, uint32_t pos, bool first, bool release_v, bool last) {
            bool good = kv_wait(pos, 0x515) && WAIT_ALL(&p_ready[x], tp[x] & 1, 0x514);
            if (good && first && on[x] > 0) good = WAIT_ALL(&o_free[x], (on[x] - 1) & 1, 0x517);
            if (!good) return false;
            tc_fence_after();
            const uint64_t v = dV0 + (pos % RING) * TILE_UNITS;
            if (leader) {
                #pragma unroll
                for (int kk = 0; kk < BT / 16; kk++) umma_ts(tmem_base + 256 + x * 128, tmem_base + x * 128 + kk * 8, v + 128 * kk, idesc_o, !first || kk > 0);
                if (release_v) umma_commit(&kv_empty[pos % RING]);
                if (last) umma_commit(&o_full[x]);
            }
            tp[x]++;
            if (first) on[x]++;
            return true;
        };
        // S_x(0) of an item whose key tiles start at kabs_
        auto issue_first = [&](const Items& it, int x, uint32_t kabs_) {
            const bool reads_last = it.has_b() ? x == 1 : x == 0;
            return issue_s(x, 2 * kabs_, true, reads_last, it.tiles(x) == 1);
        };
        if (im.valid()) {
            ok = issue_first(im, 0, 0);
            if (ok && im.has_b()) ok = issue_first(im, 1, 0);
        }
        while (im.valid() && ok) {
            Items nx = im; nx.next();
            const int nA = im.tiles(0), nB = im.tiles(1), nkv = im.kv_tiles();
            for (int j = 0; j < nkv && ok; j++) {
                const uint32_t kpos = 2 * (kabs + j);
                if (j < nA) {
                    ok = issue_pv(0, kpos + 1, j == 0, nB == 0, j == nA - 1);
                    if (ok && j + 1 < nA) ok = issue_s(0, kpos + 2, false, nB == 0, j + 1 == nA - 1);
                }
                // the next item's first S of slot A: its K tile is behind this item's tiles in the ring
                if (ok && j == nkv - 1 && nx.valid()) ok = issue_first(nx, 0, kabs + nkv);
                if (ok && j < nB) {
                    ok = issue_pv(1, kpos + 1, j == 0, true, j == nB - 1);
                    if (ok && j + 1 < nB) ok = issue_s(1, kpos + 2, false, true, j + 1 == nB - 1);
                }
            }
            kabs += nkv;
            if (ok && nx.valid() && nx.has_b()) ok = issue_first(nx, 1, kabs);
            im = nx;
        }
#undef WAIT_ALL
    }
    else if (warp >= 4) {
        // ---------------------------------------------------------------- softmax of slot x: thread = query row r of the slot's tile
        const int x = (warp - 4) >> 2;
        const int q4 = warp & 3;
        const int r = q4 * 32 + lane;
        const uint32_t lane_off = (uint32_t)(q4 * 32) << 16;
        const uint32_t tS = tmem_base + x * 128 + lane_off, tO = tmem_base + 256 + x * 128 + lane_off;
        const bool issuer = q4 == 0 && lane == 0;          // the thread of the slot that issues its output stores
        const float c = a.scale_log2e;
        bool ok = true;
        bool staged = false;
        uint32_t t = 0;                                    // tiles of this slot so far
        uint32_t it = 0;                                   // items of this slot so far
        for (; im.valid(); im.next()) {
            const int nj = im.tiles(x);
            if (nj == 0) continue;                         // (uniform for the slot) no second tile in this item
            float m = -INFINITY, l = 0.f;                  // reference maximum (raw score units) and row sum relative to it
            for (int j = 0; j < nj; j++, t++) {
                ok = mbar_wait(&s_full[x], t & 1, abort_flag, a.status, 0x520 + x) && ok;
                // The first S products of both slots complete together: the slots would compete for the special-function unit and then leave
                // it idle together.  Slot B starts half a tile late; from then on the order of the products keeps the two apart.
                if (x == 1 && t == 0) { const long long t0 = clock64(); while (clock64() - t0 < SKEW_CYCLES) { } }
                tc_fence_after();
                uint32_t sv[128];
                tmem_ld32(tS, sv);
                tmem_ld32(tS + 32, sv + 32);
                tmem_ld32(tS + 64, sv + 64);
                tmem_ld32(tS + 96, sv + 96);
                tmem_ld_wait();
                if (j == nj - 1) {
                    #pragma unroll
                    for (int e = 0; e < 128; e++) if (e > r) sv[e] = 0xff800000u;      // -inf above the diagonal
                }
                float mx0 = -INFINITY, mx1 = -INFINITY, mx2 = -INFINITY, mx3 = -INFINITY;
                #pragma unroll
                for (int e = 0; e < 128; e += 4) {
                    mx0 = fmaxf(mx0, __uint_as_float(sv[e])); mx1 = fmaxf(mx1, __uint_as_float(sv[e + 1]));
                    mx2 = fmaxf(mx2, __uint_as_float(sv[e + 2])); mx3 = fmaxf(mx3, __uint_as_float(sv[e + 3]));
                }
                const float mx = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3));
                // a moved maximum rescales the row sum now and the row of O_X below (decided per warp, so that the TMEM accesses stay
                // warp-wide)
                const bool moved = __any_sync(0xffffffffu, mx > m || j == 0) != 0;
                float alpha = 1.0f;
                if (moved) {
                    const float m_new = fmaxf(m, mx);
                    alpha = ex2_fast((m - m_new) * c);      // 0 on the first tile (m = -inf)
                    l *= alpha;
                    m = m_new;
                }
                const float moff = m * c;
                float rs[4] = {0.f, 0.f, 0.f, 0.f};
                uint32_t pk[64];
                #pragma unroll
                for (int e = 0; e < 128; e += 2) {
                    const float p0 = ex2_fast(fmaf(__uint_as_float(sv[e]), c, -moff));
                    const float p1 = ex2_fast(fmaf(__uint_as_float(sv[e + 1]), c, -moff));
                    rs[(e >> 1) & 3] += p0 + p1;
                    pk[e >> 1] = pack_bf16x2(p0, p1);
                }
                l += (rs[0] + rs[1]) + (rs[2] + rs[3]);
                tmem_st16(tS, pk);                          // over this row's own scores
                tmem_st16(tS + 16, pk + 16);
                tmem_st16(tS + 32, pk + 32);
                tmem_st16(tS + 48, pk + 48);
                if (moved && j > 0) {                       // O_X(t-1) is complete: its product was issued ahead of S_X(t)
                    #pragma unroll
                    for (int cc = 0; cc < 4; cc++) {
                        if (cc * 2 < a.ks) {
                            uint32_t ov[32];
                            tmem_ld32(tO + cc * 32, ov);
                            tmem_ld_wait();
                            #pragma unroll
                            for (int e = 0; e < 32; e++) ov[e] = __float_as_uint(__uint_as_float(ov[e]) * alpha);
                            tmem_st16(tO + cc * 32, ov);
                            tmem_st16(tO + cc * 32 + 16, ov + 16);
                        }
                    }
                }
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&p_ready[x]);
            }
            // ---- item epilogue: O_X / l -> bf16 tile in the layout of two 128-byte-swizzled TMA boxes -> bulk stores
            ok = mbar_wait(&o_full[x], it & 1, abort_flag, a.status, 0x528 + x) && ok;
            it++;
            tc_fence_after();
            if (staged) { if (issuer) tma_store_wait_read<0>(); asm volatile("bar.sync %0, 128;" ::"r"(1 + x) : "memory"); }
            const float inv = 1.0f / l;
            #pragma unroll
            for (int cc = 0; cc < 4; cc++) {
                if (cc * 2 < a.ks) {
                    uint32_t ov[32];
                    tmem_ld32(tO + cc * 32, ov);
                    tmem_ld_wait();
                    uint8_t* orow = sO + x * TILE_BYTES + (cc >> 1) * CHUNK_BYTES + r * 128;
                    #pragma unroll
                    for (int u = 0; u < 4; u++) {
                        uint4 o;
                        o.x = pack_bf16x2(__uint_as_float(ov[8 * u]) * inv, __uint_as_float(ov[8 * u + 1]) * inv);
                        o.y = pack_bf16x2(__uint_as_float(ov[8 * u + 2]) * inv, __uint_as_float(ov[8 * u + 3]) * inv);
                        o.z = pack_bf16x2(__uint_as_float(ov[8 * u + 4]) * inv, __uint_as_float(ov[8 * u + 5]) * inv);
                        o.w = pack_bf16x2(__uint_as_float(ov[8 * u + 6]) * inv, __uint_as_float(ov[8 * u + 7]) * inv);
                        *reinterpret_cast<uint4*>(orow + ((((cc & 1) * 4 + u) ^ (r & 7)) * 16)) = o;
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&o_free[x]);            // O_X may be overwritten by the next item's first product
            fence_async_smem();
            asm volatile("bar.sync %0, 128;" ::"r"(1 + x) : "memory");
            const int qi = 2 * im.p + x;
            if (issuer && ok) {
                tma_store_4d(&tmOut, sO + x * TILE_BYTES, 0, im.h, qi * BT, im.b);
                tma_store_4d(&tmOut, sO + x * TILE_BYTES + CHUNK_BYTES, 64, im.h, qi * BT, im.b);
                tma_store_commit();
            }
            staged = true;
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

// Tensor map over a packed (B, T, 3, NH, HS) tensor seen as 4-D {HS, 3*NH, T, B} with a box of `rows` rows.
int llmc_attn_qkv_map(CUtensorMap* tm, const bf16* qkv, int B, int T, int NH, int hs, int rows) {
    uint64_t dims[4] = {(uint64_t)hs, (uint64_t)(3 * NH), (uint64_t)T, (uint64_t)B};
    uint64_t strides[4] = {2, (uint64_t)hs * 2, (uint64_t)3 * NH * hs * 2, (uint64_t)T * 3 * NH * hs * 2};
    uint32_t box[4] = {64, 1, (uint32_t)rows, 1};
    return llmc_get_tensormap(tm, qkv, 2, 4, dims, strides, box, 3);
}

// out (B,T,NH,HS) = causal softmax(Q K^T / sqrt(HS)) V ; lse (B,NH,T) fp32.  Head sizes: multiples of 8, 72..128.
// The entry point llmc_attention_fwd (attention_fwd1.cu) sends every head size but 64 here.
int llmc_attention_fwd_general(bf16* out, float* lse, const bf16* qkv, int B, int T, int NH, int hs, cudaStream_t stream) {
    if (hs <= 64 || hs > 128 || (hs % 8)) { fprintf(stderr, "[llmc_b200] attention: head size %d not supported (multiples of 8 from 64 to 128)\n", hs); return -1; }
    CUtensorMap tmQKV, tmOut;
    int rc = llmc_attn_qkv_map(&tmQKV, qkv, B, T, NH, hs, BT);
    if (rc) return rc;
    {
        uint64_t dims[4] = {(uint64_t)hs, (uint64_t)NH, (uint64_t)T, (uint64_t)B};
        uint64_t strides[4] = {2, (uint64_t)hs * 2, (uint64_t)NH * hs * 2, (uint64_t)T * NH * hs * 2};
        uint32_t box[4] = {64, 1, 128, 1};
        if ((rc = llmc_get_tensormap(&tmOut, out, 2, 4, dims, strides, box, 3))) return rc;
    }
    Args a;
    a.lse = lse; a.T = T; a.NH = NH; a.BH = B * NH;
    a.ks = CEIL_DIV(hs, 16);
    a.scale = 1.0f / sqrtf((float)hs);
    a.scale_log2e = a.scale * 1.4426950408889634f;
    a.status = llmc_status_ptr();
    const int total = B * NH * ((CEIL_DIV(T, BT) + 1) / 2);
    int sms = llmc_device_sm_count(); if (sms <= 0) sms = 148;
    const int grid = total < sms ? total : sms;
    static bool configured = false;
    if (!configured) {
        CUDA_CHECK(cudaFuncSetAttribute(attn_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
        configured = true;
    }
    attn_fwd_kernel<<<grid, THREADS, SMEM, stream>>>(tmQKV, tmOut, a);
    CUDA_CHECK(cudaGetLastError());
    return 0;
}
