// Optimizer-side kernels on flat parameter / gradient buffers: squared global gradient norm,
// AdamW with fp32 master weights and stochastic rounding to bf16, re-rounding of parameters from the
// master copy (resume), master initialisation from bf16 parameters.
//
// All kernels take a table of up to 16 "tensor views".  A view describes the part of one parameter
// tensor this rank owns: `L` layer slices of `n` elements each, slice l starting at
// p_base + l * p_stride in the parameter/gradient buffers and at o_base + l * o_stride in the
// optimizer-state buffers (m, v, master).  With one rank the views cover whole tensors; with ZeRO-1
// they cover this rank's 1/N of every layer slice, which is the layout the reference stores in its
// state files (train_gpt2.cu:1035-1124 of the reference).
//
// The clipping coefficient is computed on the device from the squared norm, so a training step
// needs no host synchronisation between backward and the parameter update.
//
// Capability parity: llmc/adamw.cuh, llmc/global_norm.cuh, init_from_master, copy_and_cast.
#include "common.cuh"

struct TensorView {
    long long p_base, p_stride, o_base, o_stride, n;
    int L;
    float wd;              // weight decay applied to this tensor
    unsigned int seed;     // stochastic rounding seed of this tensor for this step
    int pad;
};
struct TensorTable {
    TensorView t[16];
    int count;
};

namespace {

struct alignas(8) Pack64 { bf16 v[4]; };

// The elements of a table's views as one list of chunks of at most `per` elements, none across a slice: view by view, slice by slice.  Blocks take chunks,
// not views: most views of a transformer are small, and a block for every view and place in it came to thousands that found nothing to do.
struct Chunks {
    TensorTable tab;
    int first[17];         // number of chunks in front of view i
    int per;
    Chunks(const TensorTable& t, int per_) : tab(t), per(per_) {
        first[0] = 0;
        for (int i = 0; i < 16; i++) first[i + 1] = first[i] + (i < t.count ? (int)CEIL_DIV(t.t[i].n, (long long)per_) * t.t[i].L : 0);
    }
    int total() const { return first[16]; }
};
// Walks from chunk to chunk in increasing order.
struct ChunkAt {
    int view = 0, per_slice = 0, l = 0, c = 0;
    DEVINL void seek(const Chunks& k, int i) {
        while (i >= k.first[view + 1]) { view++; per_slice = 0; }
        if (per_slice == 0) per_slice = (int)CEIL_DIV(k.tab.t[view].n, (long long)k.per);
        const int j = i - k.first[view];
        l = j / per_slice; c = j - l * per_slice;
    }
};

constexpr int OPT_THREADS = 512;

// Bound by reading the gradients once; 124 million elements, with its sum of the partials, 46 us, 30 million 33 us (59 and 34 with a grid of every SM times every view; alone
// between other passes: the time the host takes for the two launches is about 30 us).
constexpr int NORM_THREADS = 256;
constexpr int NORM_PACKS = 4;            // 128-bit loads of a thread in flight
constexpr int NORM_BLOCKS = 16;          // per SM

__global__ void __launch_bounds__(NORM_THREADS)
norm_sq_kernel(float* __restrict__ partials, const bf16* __restrict__ grads, const __grid_constant__ Chunks k) {
    __shared__ float red[32];
    // the order of the additions is fixed by the launch geometry, which the host derives from the device alone: the same sum on every run
    float a[NORM_PACKS];
    #pragma unroll
    for (int u = 0; u < NORM_PACKS; u++) a[u] = 0.f;
    ChunkAt at;
    for (int i = blockIdx.x; i < k.first[16]; i += gridDim.x) {
        at.seek(k, i);
        const TensorView& tv = k.tab.t[at.view];
        const bf16* base = grads + tv.p_base + (long long)at.l * tv.p_stride;
        const long long packs = tv.n >> 3, p0 = (long long)at.c * (NORM_PACKS * NORM_THREADS) + threadIdx.x;
        bf16x8 g[NORM_PACKS];
        #pragma unroll
        for (int u = 0; u < NORM_PACKS; u++) g[u] = p0 + u * NORM_THREADS < packs ? ld128(base + (p0 + u * NORM_THREADS) * 8) : bf16x8::zeros();
        #pragma unroll
        for (int u = 0; u < NORM_PACKS; u++)
            #pragma unroll
            for (int e = 0; e < 8; e++) { const float f = __bfloat162float(g[u][e]); a[u] = fmaf(f, f, a[u]); }
    }
    float acc = 0.f;
    #pragma unroll
    for (int u = 0; u < NORM_PACKS; u++) acc += a[u];
    acc = block_sum(acc, red);
    if (threadIdx.x == 0) partials[blockIdx.x] = acc;
}

// out[0] = scale * sum(partials[0..n)) in index order with a fixed tree: deterministic
__global__ void __launch_bounds__(1024) final_sum_kernel(float* __restrict__ out, const float* __restrict__ partials, int n, float scale = 1.0f) {
    __shared__ float red[32];
    float acc = 0.f;
    for (int i = threadIdx.x; i < n; i += 1024) acc += partials[i];
    acc = block_sum(acc, red);
    if (threadIdx.x == 0) out[0] = acc * scale;
}

DEVINL unsigned int sr_position(long long idx, int layer) {
    // noise index of element `idx` of layer slice `layer`; a pure function of the element, so the
    // result does not depend on launch geometry (needed for bit-exact resume from a state file)
    return (unsigned int)(idx & 511) + 198491317u * ((unsigned int)(idx & ~511ll) + (unsigned int)layer);
}

template <bool HAS_MASTER>
__global__ void __launch_bounds__(OPT_THREADS)
adamw_kernel(bf16* __restrict__ params, float* __restrict__ master, const bf16* __restrict__ grads,
             float* __restrict__ m_buf, float* __restrict__ v_buf, const TensorTable tab,
             float lr, float beta1, float beta2, float bc1, float bc2, float eps,
             float grad_scale, const float* __restrict__ norm_sq, float grad_clip) {
    float scale = grad_scale;
    if (norm_sq != nullptr) {
        const float nsq = norm_sq[0];
        if (!(nsq >= 0.f) || isinf(nsq)) return;          // non-finite gradient: skip the whole update
        const float nrm = sqrtf(nsq);
        scale = (nrm > grad_clip) ? grad_scale * grad_clip / nrm : grad_scale;
    }
    const TensorView tv = tab.t[blockIdx.y];
    const long long total = tv.n * tv.L;
    for (long long i = (long long)blockIdx.x * OPT_THREADS + threadIdx.x; i < total; i += (long long)gridDim.x * OPT_THREADS) {
        const long long l = i / tv.n, idx = i - l * tv.n;
        const long long pi = tv.p_base + l * tv.p_stride + idx;
        const long long oi = tv.o_base + l * tv.o_stride + idx;
        const float g = scale * __bfloat162float(grads[pi]);
        float m = m_buf[oi], v = v_buf[oi];
        m = fmaf(beta1, m, (1.0f - beta1) * g);          // lerp(g, m, beta1)
        v = fmaf(beta2, v, (1.0f - beta2) * g * g);
        m_buf[oi] = m; v_buf[oi] = v;
        const float mh = m / bc1, vh = v / bc2;
        const float old = HAS_MASTER ? master[oi] : __bfloat162float(params[pi]);
        const float p = old - lr * (mh / (sqrtf(vh) + eps) + tv.wd * old);
        params[pi] = stochastic_round_bf16(p, squirrel_noise5(sr_position(idx, (int)l + tv.pad), tv.seed));
        if (HAS_MASTER) master[oi] = p;
    }
}

// The same update on packs (every tensor slice of a transformer is a multiple of 8 elements, and so
// are its ZeRO shards: the sharding rule demands it); the element-wise kernel above stays as the fallback for odd layouts.
// Bound by memory: 14 bytes read and 14 written per element.  A thread has groups of four elements whose neighbours belong to its neighbours in the warp, so that each
// instruction covers whole sectors (with 8 elements, two 16-byte accesses side by side, every sector of the fp32 streams was asked for and written in two
// halves); blocks are small, and there are many times more of them than fit at once, so that at any time a narrow range of each stream is read
// and written.  Norm and update of 124 / 30 / 355 million parameters 576 / 154 / 1636 us (713 / 210 / 1942 before; 571 is the copy rate's time for the first), with as many
// blocks as fit 650 / 170 / 1870, groups of eight elements 690 / - / 1890, one group per thread 639 / 178 / 1761.
constexpr int PACK_THREADS = 128;
constexpr int PACK_BLOCKS = 8;           // per SM
constexpr int PACK_WAVES = 64;           // times as many blocks at most
constexpr int PACK_QUADS = 2;            // groups of four elements of a thread
DEVINL uint2 ld64cs(const bf16* p) { return __ldcs(reinterpret_cast<const uint2*>(p)); }

template <bool HAS_MASTER>
__global__ void __launch_bounds__(PACK_THREADS, PACK_BLOCKS)
adamw_pack_kernel(bf16* __restrict__ params, float* __restrict__ master, const bf16* __restrict__ grads,
                  float* __restrict__ m_buf, float* __restrict__ v_buf, const __grid_constant__ Chunks k,
                  float lr, float beta1, float beta2, float bc1, float bc2, float eps,
                  float grad_scale, const float* __restrict__ norm_sq, float grad_clip) {
    float scale = grad_scale;
    if (norm_sq != nullptr) {
        const float nsq = norm_sq[0];
        if (!(nsq >= 0.f) || isinf(nsq)) return;          // non-finite gradient: skip the whole update
        const float nrm = sqrtf(nsq);
        scale = (nrm > grad_clip) ? grad_scale * grad_clip / nrm : grad_scale;
    }
    constexpr int U = PACK_QUADS;
    ChunkAt at;
    for (int i = blockIdx.x; i < k.first[16]; i += gridDim.x) {
        at.seek(k, i);
        const TensorView& tv = k.tab.t[at.view];
        const int l = at.l, c = at.c;
        const long long quads = tv.n >> 2;
        const long long pb = tv.p_base + l * tv.p_stride, ob = tv.o_base + l * tv.o_stride;
        const float wd = tv.wd;
        const unsigned int seed = tv.seed;
        const int layer = l + tv.pad;
        uint2 g[U];
        f32x4 m[U], v[U], w[U];
        #pragma unroll
        for (int u = 0; u < U; u++) {
            const long long q = (long long)(c * U + u) * PACK_THREADS + threadIdx.x;
            if (q >= quads) continue;
            g[u] = ld64cs(grads + pb + q * 4);
            m[u] = ld128(m_buf + ob + q * 4); v[u] = ld128(v_buf + ob + q * 4);
            if (HAS_MASTER) w[u] = ld128(master + ob + q * 4);
            else {
                const uint2 pw = *reinterpret_cast<const uint2*>(params + pb + q * 4);
                const float2 a = unpack_bf16x2(pw.x), b = unpack_bf16x2(pw.y);
                w[u][0] = a.x; w[u][1] = a.y; w[u][2] = b.x; w[u][3] = b.y;
            }
        }
        #pragma unroll
        for (int u = 0; u < U; u++) {
            const long long q = (long long)(c * U + u) * PACK_THREADS + threadIdx.x;
            if (q >= quads) continue;
            const float2 ga = unpack_bf16x2(g[u].x), gb = unpack_bf16x2(g[u].y);
            const float gf[4] = {ga.x, ga.y, gb.x, gb.y};
            Pack64 out;
            #pragma unroll
            for (int e = 0; e < 4; e++) {
                const float gg = scale * gf[e];
                m[u][e] = fmaf(beta1, m[u][e], (1.0f - beta1) * gg);
                v[u][e] = fmaf(beta2, v[u][e], (1.0f - beta2) * gg * gg);
                // the same expressions as the element-wise kernel (division by the bias corrections included), so both give the same bits
                const float mh = m[u][e] / bc1, vh = v[u][e] / bc2;
                w[u][e] = w[u][e] - lr * (mh / (sqrtf(vh) + eps) + wd * w[u][e]);
                out.v[e] = stochastic_round_bf16(w[u][e], squirrel_noise5(sr_position(q * 4 + e, layer), seed));
            }
            st128(m_buf + ob + q * 4, m[u]); st128(v_buf + ob + q * 4, v[u]);
            if (HAS_MASTER) st128(master + ob + q * 4, w[u]);
            *reinterpret_cast<uint2*>(params + pb + q * 4) = *reinterpret_cast<const uint2*>(&out);
        }
    }
}

// params <- stochastic_round(master) with the given seeds (resume path)
__global__ void __launch_bounds__(OPT_THREADS)
from_master_kernel(bf16* __restrict__ params, const float* __restrict__ master, const TensorTable tab) {
    const TensorView tv = tab.t[blockIdx.y];
    const long long total = tv.n * tv.L;
    for (long long i = (long long)blockIdx.x * OPT_THREADS + threadIdx.x; i < total; i += (long long)gridDim.x * OPT_THREADS) {
        const long long l = i / tv.n, idx = i - l * tv.n;
        params[tv.p_base + l * tv.p_stride + idx] =
            stochastic_round_bf16(master[tv.o_base + l * tv.o_stride + idx], squirrel_noise5(sr_position(idx, (int)l + tv.pad), tv.seed));
    }
}

// master <- float(params)
__global__ void __launch_bounds__(OPT_THREADS)
to_master_kernel(float* __restrict__ master, const bf16* __restrict__ params, const TensorTable tab) {
    const TensorView tv = tab.t[blockIdx.y];
    const long long total = tv.n * tv.L;
    for (long long i = (long long)blockIdx.x * OPT_THREADS + threadIdx.x; i < total; i += (long long)gridDim.x * OPT_THREADS) {
        const long long l = i / tv.n, idx = i - l * tv.n;
        master[tv.o_base + l * tv.o_stride + idx] = __bfloat162float(params[tv.p_base + l * tv.p_stride + idx]);
    }
}

int opt_grid_x() { int sms = llmc_device_sm_count(); if (sms <= 0) sms = 148; return sms; }

}  // namespace

// out[0] = scale * sum of n floats, one block, fixed summation tree (the mean loss of a step; reference:
// global_sum_deterministic, llmc/cuda_utils.cuh:188-206)
extern "C" int llmc_sum_f32(float* out, const float* in, int n, float scale, cudaStream_t stream) {
    final_sum_kernel<<<1, 1024, 0, stream>>>(out, in, n, scale);
    CUDA_CHECK(cudaGetLastError());
    return 0;
}

extern "C" int llmc_norm_sq_scratch() { return NORM_BLOCKS * opt_grid_x(); }

// out[0] = sum of squares of the gradient elements covered by the table. `partials`: llmc_norm_sq_scratch floats.
extern "C" int llmc_global_norm_sq(float* out, float* partials, const bf16* grads, const TensorTable* tab, cudaStream_t stream) {
    if (tab->count < 1 || tab->count > 16) return -1;
    for (int i = 0; i < tab->count; i++) if (tab->t[i].n % 8 || tab->t[i].p_base % 8 || tab->t[i].p_stride % 8) return -1;
    const Chunks k(*tab, NORM_PACKS * NORM_THREADS * 8);
    const int grid = llmc_norm_sq_scratch();
    norm_sq_kernel<<<grid, NORM_THREADS, 0, stream>>>(partials, grads, k);
    CUDA_CHECK(cudaGetLastError());
    final_sum_kernel<<<1, 1024, 0, stream>>>(out, partials, grid);
    CUDA_CHECK(cudaGetLastError());
    return 0;
}

// One AdamW step over the views of the table. t = step number starting at 1.
// If norm_sq (device pointer) is given, the gradient is additionally scaled by
// min(1, grad_clip / sqrt(norm_sq[0])) and the update is skipped if norm_sq is not finite.
extern "C" int llmc_adamw(bf16* params, float* master, const bf16* grads, float* m, float* v, const TensorTable* tab,
                          float lr, float beta1, float beta2, float eps, int t, float grad_scale,
                          const float* norm_sq, float grad_clip, cudaStream_t stream) {
    if (tab->count < 1 || tab->count > 16) return -1;
    const float bc1 = 1.0f - powf(beta1, (float)t), bc2 = 1.0f - powf(beta2, (float)t);
    dim3 grid(opt_grid_x() * 2, tab->count);
    bool packs = true;
    for (int i = 0; i < tab->count; i++) {
        const TensorView& tv = tab->t[i];
        if (tv.n % 8 || tv.p_base % 8 || tv.p_stride % 8 || tv.o_base % 8 || tv.o_stride % 8) packs = false;
    }
    if (packs) {
        const Chunks k(*tab, PACK_QUADS * PACK_THREADS * 4);
        const int most = opt_grid_x() * PACK_BLOCKS * PACK_WAVES;
        grid = dim3(k.total() < most ? k.total() : most);
        if (k.total() == 0) return 0;
        if (master) adamw_pack_kernel<true><<<grid, PACK_THREADS, 0, stream>>>(params, master, grads, m, v, k, lr, beta1, beta2, bc1, bc2, eps, grad_scale, norm_sq, grad_clip);
        else adamw_pack_kernel<false><<<grid, PACK_THREADS, 0, stream>>>(params, master, grads, m, v, k, lr, beta1, beta2, bc1, bc2, eps, grad_scale, norm_sq, grad_clip);
    } else if (master) adamw_kernel<true><<<grid, OPT_THREADS, 0, stream>>>(params, master, grads, m, v, *tab, lr, beta1, beta2, bc1, bc2, eps, grad_scale, norm_sq, grad_clip);
    else adamw_kernel<false><<<grid, OPT_THREADS, 0, stream>>>(params, master, grads, m, v, *tab, lr, beta1, beta2, bc1, bc2, eps, grad_scale, norm_sq, grad_clip);
    CUDA_CHECK(cudaGetLastError());
    return 0;
}

extern "C" int llmc_params_from_master(bf16* params, const float* master, const TensorTable* tab, cudaStream_t stream) {
    from_master_kernel<<<dim3(opt_grid_x() * 2, tab->count), OPT_THREADS, 0, stream>>>(params, master, *tab);
    CUDA_CHECK(cudaGetLastError());
    return 0;
}

extern "C" int llmc_master_from_params(float* master, const bf16* params, const TensorTable* tab, cudaStream_t stream) {
    to_master_kernel<<<dim3(opt_grid_x() * 2, tab->count), OPT_THREADS, 0, stream>>>(master, params, *tab);
    CUDA_CHECK(cudaGetLastError());
    return 0;
}
