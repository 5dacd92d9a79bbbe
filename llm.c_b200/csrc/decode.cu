// Incremental decoding with a key / value cache (the inference path of the reference's LLaMA script,
// train_llama3.py:167-190 and :476-556: keys and values of earlier positions are kept, only the new tokens run through
// the network).  The kernels are memory-bound and small; the products of the step are in stream_gemm.cu:
//
//   rope_cache      raw (N, (NH + 2 NKV) * HS), N = B * Tq new tokens at positions start_pos .. start_pos + Tq - 1
//                     -> q (N, NH, HS) rotated queries
//                     -> kcache / vcache (B, Tmax, NKV, HS): rotated keys and the values written at their positions
//   cached_attention  out (N, NH, HS) = softmax(q . K[0 .. pos] / sqrt(HS)) V[0 .. pos] per (batch row, new token, head);
//                     grouped queries read the cache head h / (NH / NKV) directly, nothing is expanded.
//
// llmc_cached_attention_rope does both in one launch where the fast kernel of the second is taken.
//
// start_pos comes from the host or, when `pos_ptr` is given, from device memory: a decoding step captured in a CUDA graph is
// replayed with the position advanced on the device.  A device position that would leave the cache or the rotary table makes
// the kernel record ST_BAD_ARG in the status word and return without touching memory.
#include "common.cuh"
#include "decoder_ops.h"
#include "pdl.cuh"

namespace {

// One rotary pair.  The fused product of each sum is written out: left to the compiler, it differs from one kernel to another, and with it about one bf16 in 10^5.
DEVINL float2 rotate(float re, float im, float c, float s) { return make_float2(fmaf(re, c, -__fmul_rn(im, s)), fmaf(re, s, __fmul_rn(im, c))); }
DEVINL bf16x8 rotate8(const bf16x8& a, const float4& cs0, const float4& cs1) {
    bf16x8 r;
    const float c[4] = {cs0.x, cs0.z, cs1.x, cs1.z};
    const float s[4] = {cs0.y, cs0.w, cs1.y, cs1.w};
    #pragma unroll
    for (int j = 0; j < 4; j++) {
        const float re = __bfloat162float(a[2 * j]), im = __bfloat162float(a[2 * j + 1]);
        const float2 t = rotate(re, im, c[j], s[j]);
        r[2 * j] = __float2bfloat16_rn(t.x);
        r[2 * j + 1] = __float2bfloat16_rn(t.y);
    }
    return r;
}

__global__ void __launch_bounds__(256)
rope_cache_kernel(bf16* __restrict__ q, bf16* __restrict__ kcache, bf16* __restrict__ vcache, const bf16* __restrict__ raw,
                  const float2* __restrict__ freqs, long long N, int Tq, int Tmax, int start_pos, int NH, int NKV, int HS,
                  const int* __restrict__ pos_ptr, int freqs_len, unsigned int* status) {
    pdl_wait();
    pdl_trigger();
    if (pos_ptr) {
        start_pos = *pos_ptr;
        if (start_pos < 0 || start_pos > Tmax - Tq || start_pos > freqs_len - Tq) {
            if (threadIdx.x == 0 && blockIdx.x == 0) record_error(status, ST_BAD_ARG, 0x30);
            return;
        }
    }
    const int hp = HS >> 3;
    const int heads = NH + 2 * NKV;
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= N * heads * hp) return;
    const int p = (int)(idx % hp);
    const int h = (int)((idx / hp) % heads);
    const long long n = idx / ((long long)hp * heads);
    const int pos = start_pos + (int)(n % Tq);
    const long long b = n / Tq;
    bf16x8 a = ld128cs(raw + (n * heads + h) * HS + p * 8);
    if (h < NH + NKV) {
        const float4* f = reinterpret_cast<const float4*>(freqs + (size_t)pos * (HS >> 1) + p * 4);
        a = rotate8(a, f[0], f[1]);
    }
    if (h < NH) {
        st128(q + (n * NH + h) * HS + p * 8, a);
    } else if (h < NH + NKV) {
        st128(kcache + ((b * Tmax + pos) * NKV + (h - NH)) * HS + p * 8, a);
    } else {
        st128(vcache + ((b * Tmax + pos) * NKV + (h - NH - NKV)) * HS + p * 8, a);
    }
}

constexpr int DEC_THREADS = 128;
constexpr int DEC_CHUNK = 512;      // keys whose scores sit in shared memory at a time (running maximum across chunks)
constexpr int DEC_MAX_HS = 128;

// One CTA per (head, new token, batch row).  Scores: a thread per key, the query in shared memory as fp32 (already scaled).
// Weighted sum of the values: a thread per pair of channels, DEC_THREADS / (HS / 2) key groups side by side, folded at the end.
__global__ void __launch_bounds__(DEC_THREADS)
cached_attention_kernel(bf16* __restrict__ out, const bf16* __restrict__ q, const bf16* __restrict__ kcache,
                        const bf16* __restrict__ vcache, int Tq, int Tmax, int start_pos, int NH, int NKV, int HS, float scale,
                        const int* __restrict__ pos_ptr, unsigned int* status) {
    if (pos_ptr) {
        start_pos = *pos_ptr;
        if (start_pos < 0 || start_pos > Tmax - Tq) {
            if (threadIdx.x == 0 && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0) record_error(status, ST_BAD_ARG, 0x31);
            return;
        }
    }
    __shared__ float qs[DEC_MAX_HS];
    __shared__ float sc[DEC_CHUNK];
    __shared__ float red[32];
    __shared__ float part[DEC_THREADS * 2];
    const int tid = threadIdx.x;
    const int h = blockIdx.x, t = blockIdx.y;
    const long long b = blockIdx.z;
    const long long n = b * Tq + t;
    const int g = h / (NH / NKV);
    const int nkeys = start_pos + t + 1;
    if (tid < HS) qs[tid] = __bfloat162float(q[(n * NH + h) * HS + tid]) * scale;
    __syncthreads();
    const int pairs = HS >> 1;
    const int groups = DEC_THREADS / pairs;
    const int my_pair = tid % pairs, my_group = tid / pairs;
    const int hp = HS >> 3;
    float m = -INFINITY, l = 0.f, acc0 = 0.f, acc1 = 0.f;
    for (int base = 0; base < nkeys; base += DEC_CHUNK) {
        const int cnt = min(DEC_CHUNK, nkeys - base);
        float lmax = -INFINITY;
        for (int j = tid; j < cnt; j += DEC_THREADS) {
            const bf16* krow = kcache + ((b * Tmax + base + j) * NKV + g) * HS;
            float s = 0.f;
            #pragma unroll 4
            for (int p = 0; p < hp; p++) {                    // four independent 128-bit loads in flight per thread
                const bf16x8 kk = ld128(krow + p * 8);
                #pragma unroll
                for (int e = 0; e < 8; e++) s += qs[p * 8 + e] * __bfloat162float(kk[e]);
            }
            sc[j] = s;
            lmax = fmaxf(lmax, s);
        }
        const float m_new = fmaxf(m, block_max(lmax, red));
        float lsum = 0.f;
        for (int j = tid; j < cnt; j += DEC_THREADS) {
            const float pj = __expf(sc[j] - m_new);
            sc[j] = pj;
            lsum += pj;
        }
        const float csum = block_sum(lsum, red);
        const float corr = __expf(m - m_new);
        l = l * corr + csum;
        acc0 *= corr;
        acc1 *= corr;
        m = m_new;
        if (my_group < groups) {
            #pragma unroll 8
            for (int j = my_group; j < cnt; j += groups) {
                const bf16* vrow = vcache + ((b * Tmax + base + j) * NKV + g) * HS;
                const float2 vv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(vrow + 2 * my_pair));
                acc0 += sc[j] * vv.x;
                acc1 += sc[j] * vv.y;
            }
        }
        __syncthreads();
    }
    part[tid * 2] = (my_group < groups) ? acc0 : 0.f;
    part[tid * 2 + 1] = (my_group < groups) ? acc1 : 0.f;
    __syncthreads();
    if (tid < pairs) {
        float o0 = 0.f, o1 = 0.f;
        for (int gi = 0; gi < groups; gi++) {
            o0 += part[(gi * pairs + tid) * 2];
            o1 += part[(gi * pairs + tid) * 2 + 1];
        }
        const float inv = 1.0f / l;
        *reinterpret_cast<__nv_bfloat162*>(out + (n * NH + h) * HS + 2 * tid) = __floats2bfloat162_rn(o0 * inv, o1 * inv);
    }
}

// ---------------------------------------------------------------------------------------------------------------
// Decoding attention, fast path (head width 64 or 128, at most 8 query rows per cached head: the decoding step itself).
// Reading the cache once is all the work there is, so
//   * a CTA serves ONE cached head of one batch row for ALL its (NH / NKV) * Tq query rows and a slice of the keys;
//   * each of its 4 warps walks tiles of 16 keys whose K and V rows arrive by cp.async through a ring of its own (16-byte chunks of row j XOR-swizzled
//     by j & 7).  A warp has the next two tiles on their way, or one (ca_stages);
//   * the products run on warp-level MMAs: S = Q K^T with the query rows as the 16-row operand (8 of them used), O += P V with the
//     probabilities taken from the score registers.  fp32 FMAs with one key per lane (the kernel before this one) were bound by the
//     shared-memory reads of the queries and the probabilities (187 us for the case below).
//   * probabilities keep all 24 bits: P = hi + mid + lo, each the next 8 bits as a bf16.  hi in rows 0..7 of the MMA operand and mid in the
//     otherwise idle rows 8..15, lo through a second MMA; the two halves of the accumulator are added at the end.  Queries, keys and values
//     are bf16 as stored.
//   * running (max, sum, accumulator) per warp, merged over the warps through shared memory, then over the key slices in slice
//     order: through distributed shared memory when the slices of a head form one cluster (at most 8), else through a small fp32
//     workspace and a second kernel.
// 32 rows at position 4095, 32 heads on 8 cached heads of 128: 81 us (6.6 TB/s), behind one another; 4 rows at position 160, heads of 64: 4.2 us.
constexpr int CA_WARPS = 4;
constexpr int CA_THREADS = CA_WARPS * 32;
constexpr int CA_MAX_R = 8;
constexpr int CA_TILE = 16;           // keys per tile of a warp
constexpr int CA_MIN_KEYS = 128;      // a slice is at least this long (unless the cache is shorter)
constexpr int CA_MAX_CLUSTER = 8;
constexpr float CA_LOG2E = 1.4426950408889634f;

DEVINL void cp_async16_or_zero(void* smem_dst, const void* gsrc, bool in) {     // gsrc is a readable address either way
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(smem_dst)), "l"(gsrc), "r"(in ? 16 : 0) : "memory");
}
DEVINL void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> DEVINL void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
DEVINL void ldmatrix4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
DEVINL void ldmatrix4_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
DEVINL void mma_16x8x16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// the upper 16 bits of two floats: bf16 without rounding
DEVINL uint32_t top_bf16x2(float lo, float hi) { return __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x7632); }
// a lower bound for the parts of probability p: half of it is still a positive bf16
DEVINL float least_part(float p) { return p > 0.f ? fmaxf(p * 0x1p-32f, 0x1p-132f) : 0.f; }
// float of this CTA's shared memory at byte address `addr`, in CTA `rank` of the cluster
DEVINL float ld_peer(uint32_t addr, uint32_t rank) {
    uint32_t ra; float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(ra) : "memory");
    return v;
}
DEVINL void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int HS_, int STAGES> __host__ __device__ constexpr int ca_ring_bytes() { return STAGES * 2 * CA_TILE * HS_ * 2; }             // of one warp
template <int HS_> __host__ __device__ constexpr int ca_part_floats() { return CA_MAX_R * (HS_ + 2); }                                 // acc, max, sum of 8 rows
template <int HS_, int STAGES> __host__ __device__ constexpr int ca_smem_bytes() { return CA_WARPS * ca_ring_bytes<HS_, STAGES>() + ca_part_floats<HS_>() * 4; }

// Where the queries and the new keys and values come from when they are not in q and the caches yet (ROPE): the output of the QKV projection
struct Fresh {
    const bf16* raw;           // (N, NH + 2 NKV, HS), not rotated
    const float2* freqs;       // (freqs_len, HS / 2) cos, sin
    int freqs_len;
    int early;                 // no kernel directly in front of this one writes the caches or the position: cached keys are read before it has completed
};

// CLUSTER: the gridDim.x slices of a head are one cluster and `out` receives the result; otherwise the slice's partial goes to ws.
// ROPE: the queries are rotated in registers; the warp whose tile a new key falls into rotates it, puts it and its value into the tile and writes both
// to the caches.  A launch of its own for that (rope_cache_kernel) costs a decoding step 3 to 4 us in every layer.
template <int HS_, int STAGES, bool CLUSTER, bool ROPE>
__global__ void __launch_bounds__(CA_THREADS)
cached_attention_split_kernel(bf16* __restrict__ out, float* __restrict__ ws, const bf16* __restrict__ q, const Fresh fresh, bf16* kcache,
                              bf16* vcache, int Tq, int Tmax, int start_pos, int NH, int NKV, float scale,
                              const int* __restrict__ pos_ptr, unsigned int* status, int keys_per_slice, int rows) {
    const bool early = ROPE && fresh.early;
    if (!early) { pdl_wait(); pdl_trigger(); }
    if (pos_ptr) {
        start_pos = *pos_ptr;
        if (start_pos < 0 || start_pos > Tmax - Tq || (ROPE && start_pos > fresh.freqs_len - Tq)) {           // the same for every CTA of a cluster
            if (early) pdl_wait();             // the kernel behind this one relies on what is before it
            if (threadIdx.x == 0 && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0) record_error(status, ST_BAD_ARG, ROPE ? 0x30 : 0x32);
            return;
        }
    }
    constexpr int ROWB = HS_ * 2;              // bytes of a key row
    constexpr int CHUNKS = HS_ / 8;            // 16-byte chunks of a row
    constexpr int KS = HS_ / 16;               // 16-channel steps
    constexpr int STAGE = 2 * CA_TILE * ROWB;  // K tile, V tile
    constexpr int PART = ca_part_floats<HS_>();
    extern __shared__ __align__(16) uint8_t ca_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int gq = lane >> 2, tq4 = lane & 3;                  // MMA fragment coordinates: row gq, column pair tq4
    uint8_t* ring = ca_smem + warp * ca_ring_bytes<HS_, STAGES>();
    float* part = reinterpret_cast<float*>(ca_smem + CA_WARPS * ca_ring_bytes<HS_, STAGES>());      // this CTA's merged partial: [8][HS_], max[8], sum[8]
    const int slice = blockIdx.x, g = blockIdx.y, nslices = gridDim.x;
    const long long b = blockIdx.z;
    const int G = NH / NKV;
    const int nkeys = start_pos + Tq;                          // keys visible to the last new token
    const int k0 = min(nkeys, slice * keys_per_slice), k1 = min(nkeys, k0 + keys_per_slice);

    const long long row_stride = (long long)NKV * HS_;
    bf16* kbase = kcache + ((b * Tmax) * NKV + g) * HS_;
    bf16* vbase = vcache + ((b * Tmax) * NKV + g) * HS_;
    const int cached = ROPE ? min(k1, start_pos) : k1;         // keys below are in the cache
    // K and V rows kt .. kt + 15 -> stage st; rows past the slice are zero, and so are their probabilities
    auto fetch = [&](int kt, int st) {
        if (kt < k1) {
            uint8_t* dst = ring + st * STAGE;
            #pragma unroll
            for (int i = 0; i < CA_TILE * CHUNKS / 32; i++) {
                const int id = i * 32 + lane, row = id / CHUNKS, c = id % CHUNKS;
                const long long src = min(kt + row, k1 - 1) * row_stride + c * 8;
                const int off = row * ROWB + ((c ^ (row & 7)) * 16);
                cp_async16_or_zero(dst + off, kbase + src, kt + row < cached);
                cp_async16_or_zero(dst + CA_TILE * ROWB + off, vbase + src, kt + row < cached);
            }
        }
        cp_async_commit();                                     // possibly empty: the group count per tile stays one
    };
    constexpr int TSTEP = CA_WARPS * CA_TILE;
    const int kt0 = k0 + warp * CA_TILE;
    #pragma unroll
    for (int s = 0; s < STAGES - 1; s++) fetch(kt0 + s * TSTEP, s);
    if (early) { pdl_wait(); pdl_trigger(); }

    // query rows r -> token r / G, head g * G + r % G; the A operand of S: lane holds channels 2 tq4, 2 tq4 + 1 and + 8, + 9 of row gq.
    // Rows past `rows` are zero and dropped at the end.
    uint32_t qa[KS][2];
    {
        const int r = gq < rows ? gq : 0;
        const bf16* qr = ROPE ? fresh.raw + ((b * Tq + r / G) * (NH + 2 * NKV) + g * G + r % G) * HS_ + 2 * tq4
                              : q + ((b * Tq + r / G) * NH + g * G + r % G) * HS_ + 2 * tq4;
        #pragma unroll
        for (int kk = 0; kk < KS; kk++) {
            qa[kk][0] = gq < rows ? *reinterpret_cast<const uint32_t*>(qr + kk * 16) : 0u;
            qa[kk][1] = gq < rows ? *reinterpret_cast<const uint32_t*>(qr + kk * 16 + 8) : 0u;
        }
        if (ROPE) {
            // the two channels of a word are a rotary pair
            const float2* fr = fresh.freqs + (size_t)(start_pos + r / G) * (HS_ / 2) + tq4;
            #pragma unroll
            for (int kk = 0; kk < KS; kk++)
                #pragma unroll
                for (int i = 0; i < 2; i++) {
                    const float2 x = unpack_bf16x2(qa[kk][i]), f = fr[kk * 8 + i * 4], y = rotate(x.x, x.y, f.x, f.y);
                    qa[kk][i] = pack_bf16x2(y.x, y.y);
                }
        }
    }
    const int limit = min(k1, start_pos + (gq < rows ? gq : 0) / G + 1);      // keys [0, limit) are visible to this lane's row
    const float sl2 = scale * CA_LOG2E;
    float m = -INFINITY, l = 0.f;                              // of row gq; l: this lane's keys only
    float acc[HS_ / 8][4];                                     // columns 2 tq4, + 1 of channel group n: [0,1] from P hi and lo, [2,3] from P mid
    #pragma unroll
    for (int n = 0; n < HS_ / 8; n++) { acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f; }
    // ldmatrix: lane supplies the row address of matrix lane / 8, row lane % 8
    const int mrow = lane & 7, mid = lane >> 3;
    int st = 0;
    for (int kt = kt0; kt < k1; kt += TSTEP) {
        fetch(kt + (STAGES - 1) * TSTEP, st == 0 ? STAGES - 1 : st - 1);
        cp_async_wait<STAGES - 1>();
        __syncwarp();
        const uint32_t kb = smem_u32(ring + st * STAGE), vb = kb + CA_TILE * ROWB;
        if (ROPE && kt + CA_TILE > start_pos) {
            // new rows of this tile: 16 bytes of a key or of its value per lane
            const int t0 = max(0, kt - start_pos), t1 = min(min(kt + CA_TILE, k1) - start_pos, Tq);
            for (int id = lane; id < (t1 - t0) * 2 * CHUNKS; id += 32) {
                const int t = t0 + id / (2 * CHUNKS), c = id % CHUNKS, row = start_pos + t - kt;
                const bool value = (id / CHUNKS) & 1;
                bf16x8 x = ld128(fresh.raw + ((b * Tq + t) * (NH + 2 * NKV) + NH + (value ? NKV : 0) + g) * HS_ + c * 8);
                if (!value) {
                    const float4* f = reinterpret_cast<const float4*>(fresh.freqs + (size_t)(start_pos + t) * (HS_ / 2) + c * 4);
                    x = rotate8(x, f[0], f[1]);
                }
                st128((value ? vbase : kbase) + (kt + row) * row_stride + c * 8, x);
                *reinterpret_cast<bf16x8*>(ring + st * STAGE + (value ? CA_TILE * ROWB : 0) + row * ROWB + ((c ^ (row & 7)) * 16)) = x;
            }
            __syncwarp();
        }
        // ---- S (row gq, keys 2 tq4 + {0,1} of each group of 8 keys)
        float s[2][4];
        #pragma unroll
        for (int h = 0; h < 2; h++) { s[h][0] = s[h][1] = s[h][2] = s[h][3] = 0.f; }
        #pragma unroll
        for (int kk = 0; kk < KS; kk++) {
            uint32_t kf[4];     // matrices: keys 0-7 channels 0-7 / 8-15 of the step, keys 8-15 likewise
            const int row = (mid >> 1) * 8 + mrow, c = kk * 2 + (mid & 1);
            ldmatrix4(kf, kb + row * ROWB + ((c ^ (row & 7)) * 16));
            mma_16x8x16(s[0], qa[kk][0], 0u, qa[kk][1], 0u, kf[0], kf[1]);
            mma_16x8x16(s[1], qa[kk][0], 0u, qa[kk][1], 0u, kf[2], kf[3]);
        }
        // ---- running softmax of row gq (base 2); the four lanes of a row hold its 16 keys
        float sv[4];
        #pragma unroll
        for (int e = 0; e < 4; e++) {
            const int key = kt + (e >> 1) * 8 + 2 * tq4 + (e & 1);
            sv[e] = key < limit ? s[e >> 1][e & 1] * sl2 : -INFINITY;
        }
        float mn = fmaxf(fmaxf(sv[0], sv[1]), fmaxf(sv[2], sv[3]));
        mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, 1));
        mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, 2));
        mn = fmaxf(mn, m);
        const float mref = mn == -INFINITY ? 0.f : mn;         // no key seen yet: every probability below is 2^-inf = 0
        const float corr = ex2_fast(m - mref);
        float p[4];
        #pragma unroll
        for (int e = 0; e < 4; e++) p[e] = ex2_fast(sv[e] - mref);
        l = l * corr + ((p[0] + p[1]) + (p[2] + p[3]));
        m = mn;
        if (__any_sync(0xffffffffu, corr != 1.0f)) {
            #pragma unroll
            for (int n = 0; n < HS_ / 8; n++) { acc[n][0] *= corr; acc[n][1] *= corr; acc[n][2] *= corr; acc[n][3] *= corr; }
        }
        // 8 bits each, cut off: the differences are exact and not negative.  No part of a positive probability is zero (which changes it by at
        // most 2^-31 of its value, or of the smallest normal number), so that its product with an infinite value is that infinity in
        // all three parts; lo goes through both halves of the operand for the same reason.
        uint32_t hi[2], md[2], lo[2];
        #pragma unroll
        for (int h = 0; h < 2; h++) {
            hi[h] = top_bf16x2(p[2 * h], p[2 * h + 1]);
            const float2 hf = unpack_bf16x2(hi[h]);
            const float e0 = least_part(p[2 * h]), e1 = least_part(p[2 * h + 1]);
            const float r0 = fmaxf(p[2 * h] - hf.x, e0), r1 = fmaxf(p[2 * h + 1] - hf.y, e1);
            md[h] = top_bf16x2(r0, r1);
            const float2 mf = unpack_bf16x2(md[h]);
            lo[h] = top_bf16x2(0.5f * fmaxf(r0 - mf.x, e0), 0.5f * fmaxf(r1 - mf.y, e1));
        }
        // ---- O += P V: 16 keys, 16 channels per ldmatrix
        #pragma unroll
        for (int n2 = 0; n2 < HS_ / 16; n2++) {
            uint32_t vf[4];     // matrices: keys 0-7 / 8-15 of channels 0-7 of the pair of groups, then of channels 8-15
            const int row = (mid & 1) * 8 + mrow, c = n2 * 2 + (mid >> 1);
            ldmatrix4_trans(vf, vb + row * ROWB + ((c ^ (row & 7)) * 16));
            mma_16x8x16(acc[2 * n2], hi[0], md[0], hi[1], md[1], vf[0], vf[1]);
            mma_16x8x16(acc[2 * n2 + 1], hi[0], md[0], hi[1], md[1], vf[2], vf[3]);
            mma_16x8x16(acc[2 * n2], lo[0], lo[0], lo[1], lo[1], vf[0], vf[1]);
            mma_16x8x16(acc[2 * n2 + 1], lo[0], lo[0], lo[1], lo[1], vf[2], vf[3]);
        }
        __syncwarp();                                          // the stage may be refilled
        st = st + 1 == STAGES ? 0 : st + 1;
    }
    cp_async_wait<0>();
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);
    // ---- merge the warps in warp order (the rings are free now)
    __syncthreads();
    float* wp = reinterpret_cast<float*>(ca_smem) + warp * PART;
    #pragma unroll
    for (int n = 0; n < HS_ / 8; n++) {
        wp[gq * HS_ + n * 8 + 2 * tq4] = acc[n][0] + acc[n][2];
        wp[gq * HS_ + n * 8 + 2 * tq4 + 1] = acc[n][1] + acc[n][3];
    }
    if (tq4 == 0) { wp[CA_MAX_R * HS_ + gq] = m; wp[CA_MAX_R * HS_ + CA_MAX_R + gq] = l; }
    __syncthreads();
    const float* w0 = reinterpret_cast<const float*>(ca_smem);
    float* dst = CLUSTER ? part : ws + ((size_t)(b * NKV + g) * nslices + slice) * PART;
    for (int i = threadIdx.x; i < rows * HS_; i += CA_THREADS) {
        const int r = i / HS_;
        float mn = -INFINITY;
        #pragma unroll
        for (int w = 0; w < CA_WARPS; w++) mn = fmaxf(mn, w0[w * PART + CA_MAX_R * HS_ + r]);
        float a = 0.f, ls = 0.f;
        #pragma unroll
        for (int w = 0; w < CA_WARPS; w++) {
            const float mw = w0[w * PART + CA_MAX_R * HS_ + r];
            const float cw = (mw == -INFINITY) ? 0.f : ex2_fast(mw - mn);
            a += w0[w * PART + i] * cw;
            ls += w0[w * PART + CA_MAX_R * HS_ + CA_MAX_R + r] * cw;
        }
        dst[i] = a;
        if (i - r * HS_ == 0) { dst[CA_MAX_R * HS_ + r] = mn; dst[CA_MAX_R * HS_ + CA_MAX_R + r] = ls; }
    }
    if (CLUSTER) {
        __syncwarp();
        cluster_sync();                                        // the partials of all slices are in place
        const uint32_t base = smem_u32(part);
        for (int i = slice * CA_THREADS + threadIdx.x; i < rows * HS_; i += nslices * CA_THREADS) {
            const int r = i / HS_, c = i - r * HS_;
            float mn = -INFINITY;
            for (int s2 = 0; s2 < nslices; s2++) mn = fmaxf(mn, ld_peer(base + (CA_MAX_R * HS_ + r) * 4, s2));
            float a = 0.f, ls = 0.f;
            for (int s2 = 0; s2 < nslices; s2++) {
                const float ms = ld_peer(base + (CA_MAX_R * HS_ + r) * 4, s2);
                const float cw = (ms == -INFINITY) ? 0.f : ex2_fast(ms - mn);
                a += ld_peer(base + i * 4, s2) * cw;
                ls += ld_peer(base + (CA_MAX_R * HS_ + CA_MAX_R + r) * 4, s2) * cw;
            }
            out[((b * Tq + r / G) * NH + g * G + r % G) * HS_ + c] = __float2bfloat16_rn(a / ls);
        }
        __syncwarp();
        cluster_sync();                                        // no CTA leaves while a peer may still read its shared memory
    }
}

// out[row r of (b, g)] = sum over slices of acc_s * 2^(m_s - M) / sum over slices of l_s * 2^(m_s - M), slices in order
template <int HS_>
__global__ void cached_attention_combine_kernel(bf16* __restrict__ out, const float* __restrict__ ws, int Tq, int NH, int NKV, int nslices) {
    pdl_wait();
    pdl_trigger();
    constexpr int PART = ca_part_floats<HS_>();
    const int r = blockIdx.x, g = blockIdx.y;
    const long long b = blockIdx.z;
    const int c = threadIdx.x;
    const float* src = ws + (size_t)(b * NKV + g) * nslices * PART;
    float mn = -INFINITY;
    for (int s = 0; s < nslices; s++) mn = fmaxf(mn, src[(size_t)s * PART + CA_MAX_R * HS_ + r]);
    float a = 0.f, ls = 0.f;
    for (int s = 0; s < nslices; s++) {
        const float ms = src[(size_t)s * PART + CA_MAX_R * HS_ + r];
        const float cw = (ms == -INFINITY) ? 0.f : ex2_fast(ms - mn);        // the maxima are in base-2 units
        a += src[(size_t)s * PART + r * HS_ + c] * cw;
        ls += src[(size_t)s * PART + CA_MAX_R * HS_ + CA_MAX_R + r] * cw;
    }
    const int G = NH / NKV;
    const int t = r / G, hq = g * G + r % G;
    out[((b * Tq + t) * NH + hq) * HS_ + c] = __float2bfloat16_rn(a / ls);
}

// ---------------------------------------------------------------------------------------------------------------
// Skinny product, launched by itself: out (M, N) = x (M, K) . w (N, K)^T with M <= 8 rows.  It is bound by streaming the weights once.
// stream_gemm.cu does the same product faster inside a replayed step, where it starts and prefetches under its predecessor, but slower
// alone (us, this kernel first): 4 x 28672 x 4096 50 / 59, 4 x 49152 x 4096 76 / 90, 4 x 6144 x 4096 16 / 20, 1 x 768 x 768 8 / 10; 4 x 2048 x 7168
// is the exception at 18 / 16.  Here a CTA owns 16 output columns and its 8 warps split K; a warp feeds warp-level
// m16n8k16 MMAs with the weights as the 16-row operand and the (at most 8) activation rows as the 8-column operand, so that
// the arithmetic costs two instructions per KB of weights and the loop is nothing but 128-bit streaming loads.  A lane
// loads 8 consecutive K elements of weight rows g and g + 8 and of activation row g (g = lane / 4) and uses them as the
// K slots of two MMAs; the dot product does not care that this permutes K, as long as both operands agree.
constexpr int SK_WARPS = 8;
constexpr int SK_THREADS = SK_WARPS * 32;
constexpr int SK_COLS = 16;
constexpr int SK_UNROLL = 4;
constexpr int SK_MAX_M = 8;

__global__ void __launch_bounds__(SK_THREADS)
skinny_gemm_kernel(bf16* __restrict__ out, const bf16* __restrict__ x, const bf16* __restrict__ w, int M, int N, int K,
                   int ldx, int ldw, int ldo) {
    __shared__ float red[SK_WARPS][4][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int n0 = blockIdx.x * SK_COLS;
    const bf16* w0 = w + (size_t)min(n0 + g, N - 1) * ldw;          // a clamped row is computed, not stored
    const bf16* w1 = w + (size_t)min(n0 + g + 8, N - 1) * ldw;
    const bool xvalid = g < M;
    const bf16* xr = x + (size_t)min(g, M - 1) * ldx;
    const int nchunks = (K + 31) >> 5;                               // 32 K elements per chunk: 8 per lane of a quad
    const int per_warp = (nchunks + SK_WARPS - 1) / SK_WARPS;
    const int c_begin = warp * per_warp, c_end = min(c_begin + per_warp, nchunks);
    float c[4] = {0.f, 0.f, 0.f, 0.f};
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    // whole groups of SK_UNROLL full chunks: every load is issued before the first MMA, nothing is predicated
    const int full_end = min(c_end, K >> 5);
    int ch = c_begin;
    for (; ch + SK_UNROLL <= full_end; ch += SK_UNROLL) {
        uint4 a0[SK_UNROLL], a1[SK_UNROLL], b[SK_UNROLL];
        #pragma unroll
        for (int u = 0; u < SK_UNROLL; u++) {
            const int k = ((ch + u) << 5) + t * 8;
            a0[u] = __ldcs(reinterpret_cast<const uint4*>(w0 + k));
            a1[u] = __ldcs(reinterpret_cast<const uint4*>(w1 + k));
            b[u] = *reinterpret_cast<const uint4*>(xr + k);
        }
        #pragma unroll
        for (int u = 0; u < SK_UNROLL; u++) {
            if (!xvalid) b[u] = zero;
            mma_16x8x16(c, a0[u].x, a1[u].x, a0[u].y, a1[u].y, b[u].x, b[u].y);
            mma_16x8x16(c, a0[u].z, a1[u].z, a0[u].w, a1[u].w, b[u].z, b[u].w);
        }
    }
    // the rest, one chunk at a time; the last chunk of K may be partial
    for (; ch < c_end; ch++) {
        const int k = (ch << 5) + t * 8;
        const bool ok = k < K;
        const uint4 a0 = ok ? __ldcs(reinterpret_cast<const uint4*>(w0 + k)) : zero;
        const uint4 a1 = ok ? __ldcs(reinterpret_cast<const uint4*>(w1 + k)) : zero;
        const uint4 b = (ok && xvalid) ? *reinterpret_cast<const uint4*>(xr + k) : zero;
        mma_16x8x16(c, a0.x, a1.x, a0.y, a1.y, b.x, b.y);
        mma_16x8x16(c, a0.z, a1.z, a0.w, a1.w, b.z, b.w);
    }
    #pragma unroll
    for (int i = 0; i < 4; i++) red[warp][i][lane] = c[i];
    __syncthreads();
    if (warp == 0) {
        // accumulator layout: c[2 i + j] = out[row 2 t + j][column n0 + g + 8 i]
        #pragma unroll
        for (int i = 0; i < 4; i++) {
            float v = 0.f;
            #pragma unroll
            for (int ww = 0; ww < SK_WARPS; ww++) v += red[ww][i][lane];
            const int m = 2 * t + (i & 1), n = n0 + g + 8 * (i >> 1);
            if (m < M && n < N) out[(size_t)m * ldo + n] = __float2bfloat16_rn(v);
        }
    }
}

int decode_check(int B, int Tq, int Tmax, int start_pos, int NH, int NKV, int HS, bool device_pos) {
    if (HS % 8 || HS > DEC_MAX_HS || HS < 16 || NKV <= 0 || NH % NKV) return -1;
    if (B <= 0 || Tq <= 0 || Tq > Tmax) return -2;
    if (!device_pos && (start_pos < 0 || start_pos > Tmax - Tq)) return -2;      // (their sum may not fit an int)
    if (B > 65535 || Tq > 65535) return -3;
    return 0;
}

}  // namespace

// freqs holds (cos, sin) for freqs_len positions; every position written must lie inside it and inside the cache.
// pos_ptr: null, or a device int that replaces start_pos when the kernel runs.
extern "C" int llmc_rope_cache(bf16* q, bf16* kcache, bf16* vcache, const bf16* raw, const float* freqs, int freqs_len, int B, int Tq,
                               int Tmax, int start_pos, int NH, int NKV, int HS, const int* pos_ptr, cudaStream_t stream) {
    const int rc = decode_check(B, Tq, Tmax, start_pos, NH, NKV, HS, pos_ptr != nullptr);
    if (rc) return rc;
    if (!pos_ptr && start_pos > freqs_len - Tq) return -4;
    const long long N = (long long)B * Tq;
    const long long total = N * (NH + 2 * NKV) * (HS / 8);
    CUDA_CHECK(launch_pdl(rope_cache_kernel, dim3((unsigned)CEIL_DIV(total, 256)), dim3(256), 0, stream, 0, q, kcache, vcache, raw,
                          reinterpret_cast<const float2*>(freqs), N, Tq, Tmax, start_pos, NH, NKV, HS, pos_ptr, freqs_len, llmc_status_ptr()));
    return 0;
}

namespace {
// Key slices of the fast path: whole multiples of the 64 keys a CTA covers per trip, at least CA_MIN_KEYS, and about as many CTAs as
// are resident at once (two per SM); one cluster per head as long as eight slices do, since a second launch costs more than the SMs
// it leaves idle, except where a slice would get longer than 1024 keys.  The cache's capacity decides, not the current length,
// because the position may live on the device.
int ca_keys_per_slice(int B, int Tmax, int NKV) {
    int sms = llmc_device_sm_count(); if (sms <= 0) sms = 148;
    int want = (2 * sms) / (B * NKV);
    if (want < 1) want = 1;
    if (want > CA_MAX_CLUSTER && CEIL_DIV(Tmax, CA_MAX_CLUSTER) <= 1024) want = CA_MAX_CLUSTER;
    const int trip = CA_WARPS * CA_TILE;
    const int kps = CEIL_DIV(CEIL_DIV(Tmax, want), trip) * trip;
    return kps < CA_MIN_KEYS ? CA_MIN_KEYS : kps;
}
int ca_slices(int B, int Tmax, int NKV) { return CEIL_DIV(Tmax, ca_keys_per_slice(B, Tmax, NKV)); }
bool ca_fast(int Tq, int NH, int NKV, int HS) { return (HS == 64 || HS == 128) && (NH / NKV) * Tq <= CA_MAX_R; }

// Stages of a warp's ring.  With two (one tile in flight behind the one that is worked on) a 128-wide CTA asks for 32 KB at a time instead of 64, and two CTAs on an SM
// stream long slices of keys faster; everywhere else the deeper ring is the better or an equal one.  Whole steps of four layers of 4096 channels, us, three /
// two stages (rows x position, CTAs): 32 x 2000 (256) 754 / 743, 37 x 3000 (296) 889 / 870, 32 x 4000 (256) 928 / 893, 8 x 8000 (256) 712 / 706; shorter slices
// 32 x 700 (256) 644 / 644, 8 x 2000 (256) 598 / 602; fewer CTAs 24 x 2000 (192) 709 / 713, 20 x 2000 (160) 696 / 702; more 40 x 1000 (320) 751 / 757,
// 64 x 2000 (512) 965 / 976; slices without a cluster 1 x 16000 (296) 617 / 643, 4 x 16000 (288) 724 / 752.  Without the rotary embedding the kernel is small
// enough for three CTAs on an SM and two stages are slower in long slices too: 32 x 2000 46 / 53, 32 x 4000 83 / 111.
int ca_stages(int B, int Tmax, int NKV, int HS, bool rope) {
    int sms = llmc_device_sm_count(); if (sms <= 0) sms = 148;
    const int slices = ca_slices(B, Tmax, NKV), ctas = B * NKV * slices;
    return rope && HS == 128 && slices <= CA_MAX_CLUSTER && 2 * ctas > 3 * sms && ctas <= 2 * sms && ca_keys_per_slice(B, Tmax, NKV) >= 1024 ? 2 : 3;
}

template <int HS_, int STAGES, bool CLUSTER, bool ROPE>
int ca_launch(bf16* out, float* ws, const bf16* q, const Fresh& fresh, bf16* kcache, bf16* vcache, int B, int Tq, int Tmax, int start_pos, int NH,
              int NKV, const int* pos_ptr, cudaStream_t stream) {
    const int rows = (NH / NKV) * Tq, slices = ca_slices(B, Tmax, NKV);
    constexpr int smem = ca_smem_bytes<HS_, STAGES>();
    static bool configured = false;
    if (!configured) {
        CUDA_CHECK(cudaFuncSetAttribute(cached_attention_split_kernel<HS_, STAGES, CLUSTER, ROPE>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        configured = true;
    }
    CUDA_CHECK(launch_pdl(cached_attention_split_kernel<HS_, STAGES, CLUSTER, ROPE>, dim3(slices, NKV, B), dim3(CA_THREADS), smem, stream, CLUSTER ? slices : 0,
                          out, ws, q, fresh, kcache, vcache, Tq, Tmax, start_pos, NH, NKV, rsqrtf((float)HS_), pos_ptr, llmc_status_ptr(),
                          ca_keys_per_slice(B, Tmax, NKV), rows));
    if (!CLUSTER)
        CUDA_CHECK(launch_pdl(cached_attention_combine_kernel<HS_>, dim3(rows, NKV, B), dim3(HS_), 0, stream, 0, out, (const float*)ws, Tq, NH, NKV, slices));
    return 0;
}

template <bool ROPE>
int ca_dispatch(bf16* out, float* ws, const bf16* q, const Fresh& fresh, bf16* kcache, bf16* vcache, int B, int Tq, int Tmax, int start_pos, int NH,
                int NKV, int HS, const int* pos_ptr, cudaStream_t stream) {
    const bool cluster = ca_slices(B, Tmax, NKV) <= CA_MAX_CLUSTER;
#define CA_GO(H, ST, CL) return ca_launch<H, ST, CL, ROPE>(out, ws, q, fresh, kcache, vcache, B, Tq, Tmax, start_pos, NH, NKV, pos_ptr, stream)
    if (HS == 64) { if (cluster) CA_GO(64, 3, true); CA_GO(64, 3, false); }
    if constexpr (ROPE) if (ca_stages(B, Tmax, NKV, HS, true) == 2) CA_GO(128, 2, true);
    if (cluster) CA_GO(128, 3, true);
    CA_GO(128, 3, false);
#undef CA_GO
}
}  // namespace

// How many tiles of keys a warp of llmc_cached_attention (rope: llmc_cached_attention_rope) has room for, where it takes the fast path
extern "C" int llmc_cached_attention_stages(int B, int Tmax, int NKV, int HS, int rope) { return ca_stages(B, Tmax, NKV, HS, rope != 0); }

// fp32 words of workspace llmc_cached_attention needs for this problem (0: it runs without one)
extern "C" long long llmc_cached_attention_workspace(int B, int Tq, int Tmax, int NH, int NKV, int HS) {
    if (NKV <= 0 || NH % NKV || !ca_fast(Tq, NH, NKV, HS)) return 0;
    const int slices = ca_slices(B, Tmax, NKV);
    return slices <= CA_MAX_CLUSTER ? 0 : (long long)B * NKV * slices * CA_MAX_R * (HS + 2);
}

extern "C" int llmc_cached_attention(bf16* out, const bf16* q, const bf16* kcache, const bf16* vcache, int B, int Tq, int Tmax,
                                     int start_pos, int NH, int NKV, int HS, const int* pos_ptr, float* ws, cudaStream_t stream) {
    const int rc = decode_check(B, Tq, Tmax, start_pos, NH, NKV, HS, pos_ptr != nullptr);
    if (rc) return rc;
    const bool cluster = ca_fast(Tq, NH, NKV, HS) && ca_slices(B, Tmax, NKV) <= CA_MAX_CLUSTER;
    if (ca_fast(Tq, NH, NKV, HS) && (cluster || ws != nullptr)) {
        if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(kcache) | reinterpret_cast<uintptr_t>(vcache)) & 15) return -5;
        return ca_dispatch<false>(out, ws, q, Fresh{}, const_cast<bf16*>(kcache), const_cast<bf16*>(vcache), B, Tq, Tmax, start_pos, NH, NKV, HS, pos_ptr, stream);
    }
    const dim3 grid(NH, Tq, B);
    cached_attention_kernel<<<grid, DEC_THREADS, 0, stream>>>(out, q, kcache, vcache, Tq, Tmax, start_pos, NH, NKV, HS, rsqrtf((float)HS),
                                                              pos_ptr, llmc_status_ptr());
    CUDA_CHECK(cudaGetLastError());
    return 0;
}

// llmc_rope_cache and llmc_cached_attention in one launch, from the output of the QKV projection; the same bits.  For what the fast path of the
// second takes (head width 64 or 128, at most 8 query rows per cached head, a workspace where it needs one); otherwise -6, and nothing is done.
// early: the kernel in front writes neither the caches nor the position (csrc/decoder.cu); what others before it wrote is complete (pdl.cuh).
extern "C" int llmc_cached_attention_rope(bf16* out, const bf16* raw, const float* freqs, int freqs_len, bf16* kcache, bf16* vcache, int B, int Tq, int Tmax,
                                          int start_pos, int NH, int NKV, int HS, const int* pos_ptr, float* ws, int early, cudaStream_t stream) {
    const int rc = decode_check(B, Tq, Tmax, start_pos, NH, NKV, HS, pos_ptr != nullptr);
    if (rc) return rc;
    if (!pos_ptr && start_pos > freqs_len - Tq) return -4;
    if (!ca_fast(Tq, NH, NKV, HS) || (ca_slices(B, Tmax, NKV) > CA_MAX_CLUSTER && ws == nullptr)) return -6;
    if ((reinterpret_cast<uintptr_t>(raw) | reinterpret_cast<uintptr_t>(kcache) | reinterpret_cast<uintptr_t>(vcache) | reinterpret_cast<uintptr_t>(freqs)) & 15) return -6;
    const Fresh fresh = {raw, reinterpret_cast<const float2*>(freqs), freqs_len, early};
    return ca_dispatch<true>(out, ws, nullptr, fresh, kcache, vcache, B, Tq, Tmax, start_pos, NH, NKV, HS, pos_ptr, stream);
}

// out (M, N) = x (M, K) . w (N, K)^T for M <= 8; K and the row strides of x and w are multiples of 8 elements.
extern "C" int llmc_skinny_gemm(bf16* out, const bf16* x, const bf16* w, int M, int N, int K, int ldx, int ldw, int ldo, cudaStream_t stream) {
    if (M <= 0 || M > SK_MAX_M || N <= 0 || K <= 0 || (K % 8) || (ldx % 8) || (ldw % 8)) return -1;
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) return -1;
    skinny_gemm_kernel<<<(unsigned)CEIL_DIV(N, SK_COLS), SK_THREADS, 0, stream>>>(out, x, w, M, N, K, ldx, ldw, ldo);
    CUDA_CHECK(cudaGetLastError());
    return 0;
}
