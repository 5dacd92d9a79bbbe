// Stand-alone element-wise and column-reduction kernels: tanh-GELU forward (used when the GELU
// output is recomputed in the backward pass), GELU backward in place, and the bias gradient
// (column sums of a [rows, OC] gradient).  In the normal training path GELU and its derivative
// run inside the GEMM epilogues (gemm.cu); these kernels serve the recompute / unfused modes.
//
// The bias gradient is deterministic: every CTA folds a strip of rows for 256 columns in a fixed
// order and writes one fp32 partial row; a second kernel folds the strips in strip order.
//
// Capability parity: llmc/gelu.cuh and matmul_backward_bias_kernel9 / reduce_add_sum_kernel of
// llmc/matmul.cuh in the reference.
#include "common.cuh"
#include "pdl.cuh"

namespace {

__global__ void gelu_fwd_kernel(bf16* __restrict__ out, const bf16* __restrict__ inp, long long npack) {
    pdl_wait();
    pdl_trigger();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= npack) return;
    bf16x8 a = ld128cs(inp + i * 8), o;
    #pragma unroll
    for (int e = 0; e < 8; e++) o[e] = __float2bfloat16_rn(gelu_fast(__bfloat162float(a[e])));
    st128(out + i * 8, o);
}

__global__ void gelu_bwd_kernel(bf16* __restrict__ d_inout, const bf16* __restrict__ inp, long long npack) {
    pdl_wait();
    pdl_trigger();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= npack) return;
    bf16x8 a = ld128cs(inp + i * 8), d = ld128(d_inout + i * 8), o;
    #pragma unroll
    for (int e = 0; e < 8; e++) o[e] = __float2bfloat16_rn(gelu_grad_fast(__bfloat162float(a[e])) * __bfloat162float(d[e]));
    st128(d_inout + i * 8, o);
}

__global__ void residual_add_kernel(bf16* __restrict__ out, const bf16* __restrict__ a, const bf16* __restrict__ b, long long npack) {
    pdl_wait();
    pdl_trigger();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= npack) return;
    bf16x8 x = ld128cs(a + i * 8), y = ld128cs(b + i * 8), o;
    #pragma unroll
    for (int e = 0; e < 8; e++) o[e] = __float2bfloat16_rn(__bfloat162float(x[e]) + __bfloat162float(y[e]));
    st128(out + i * 8, o);
}

constexpr int BG_WARPS = 8;
constexpr int BG_ROWS = 16;               // rows of a warp in flight: 65536 x 3072 62 us (6.5 TB/s) with 16, 63 with 8, 68 with 4
// grid (ceil(OC/256), strips). partials[strip][OC]
__global__ void __launch_bounds__(BG_WARPS * 32)
bias_grad_kernel(float* __restrict__ partials, const bf16* __restrict__ dout, int rows, int OC, int rows_per_strip) {
    pdl_wait();
    pdl_trigger();
    __shared__ float sh[BG_WARPS][256];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int col = blockIdx.x * 256 + lane * 8;
    const int r0 = blockIdx.y * rows_per_strip, r1 = min(rows, r0 + rows_per_strip);
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (col < OC) {
        int r = r0 + warp;
        for (; r + (BG_ROWS - 1) * BG_WARPS < r1; r += BG_ROWS * BG_WARPS) {
            bf16x8 d[BG_ROWS];
            #pragma unroll
            for (int k = 0; k < BG_ROWS; k++) d[k] = ld128cs(dout + (size_t)(r + k * BG_WARPS) * OC + col);
            #pragma unroll
            for (int k = 0; k < BG_ROWS; k++)
                #pragma unroll
                for (int e = 0; e < 8; e++) acc[e] += __bfloat162float(d[k][e]);
        }
        for (; r < r1; r += BG_WARPS) {
            const bf16x8 d = ld128cs(dout + (size_t)r * OC + col);
            #pragma unroll
            for (int e = 0; e < 8; e++) acc[e] += __bfloat162float(d[e]);
        }
    }
    #pragma unroll
    for (int e = 0; e < 8; e++) sh[warp][lane * 8 + e] = acc[e];
    __syncthreads();
    const int c = threadIdx.x;
    if (blockIdx.x * 256 + c < OC) {
        float s = 0.f;
        #pragma unroll
        for (int w = 0; w < BG_WARPS; w++) s += sh[w][c];
        partials[(size_t)blockIdx.y * OC + blockIdx.x * 256 + c] = s;
    }
}

// A block adds the strips of 16 columns: 64 slices of strips side by side (4 threads x 4 floats each), then the slices in order, a fixed tree.
constexpr int BG_SLICES = 64;
__global__ void __launch_bounds__(4 * BG_SLICES)
bias_grad_fold_kernel(bf16* __restrict__ dbias, const float* __restrict__ partials, int strips, int OC, int accumulate) {
    pdl_wait();
    pdl_trigger();
    __shared__ float sh[BG_SLICES][16];
    const int x = threadIdx.x & 3, y = threadIdx.x >> 2;
    const int c = blockIdx.x * 16 + x * 4;
    f32x4 a = f32x4::zeros();
    if (c < OC) {                                     // OC is a multiple of 8
        #pragma unroll 4
        for (int i = y; i < strips; i += BG_SLICES) {
            const f32x4 p = ld128(partials + (size_t)i * OC + c);
            #pragma unroll
            for (int e = 0; e < 4; e++) a[e] += p[e];
        }
    }
    #pragma unroll
    for (int e = 0; e < 4; e++) sh[y][x * 4 + e] = a[e];
    __syncthreads();
    const int oc = blockIdx.x * 16 + threadIdx.x;
    if (threadIdx.x < 16 && oc < OC) {
        float s = 0.f;
        #pragma unroll 16
        for (int k = 0; k < BG_SLICES; k++) s += sh[k][threadIdx.x];
        if (accumulate) s += __bfloat162float(dbias[oc]);
        dbias[oc] = __float2bfloat16_rn(s);
    }
}

// Few rows: one launch, a CTA sums all rows of 32 columns (4 lanes of 16 bytes per row, 64 rows at a time, then the 64 sums of a column).
constexpr int BGF_SLOTS = 64;
__global__ void __launch_bounds__(4 * BGF_SLOTS)
bias_grad_few_kernel(bf16* __restrict__ dbias, const bf16* __restrict__ dout, int rows, int OC, int accumulate) {
    pdl_wait();
    pdl_trigger();
    __shared__ float sh[BGF_SLOTS][33];
    const int x = threadIdx.x & 3, y = threadIdx.x >> 2;
    const int col = blockIdx.x * 32 + x * 8;
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (col < OC) {
        #pragma unroll 8
        for (int r = y; r < rows; r += BGF_SLOTS) {
            bf16x8 d = ld128(dout + (size_t)r * OC + col);
            #pragma unroll
            for (int e = 0; e < 8; e++) acc[e] += __bfloat162float(d[e]);
        }
    }
    #pragma unroll
    for (int e = 0; e < 8; e++) sh[y][x * 8 + e] = acc[e];
    __syncthreads();
    // column c = warp * 4 + lane / 8: 8 lanes add 8 slots each, then one another's sums in a fixed tree
    const int lane = threadIdx.x & 31, c = (threadIdx.x >> 5) * 4 + (lane >> 3), part = lane & 7;
    float s = 0.f;
    #pragma unroll
    for (int i = 0; i < BGF_SLOTS / 8; i++) s += sh[part * (BGF_SLOTS / 8) + i][c];
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    s += __shfl_xor_sync(0xffffffffu, s, 4);
    const int oc = blockIdx.x * 32 + c;
    if (part == 0 && oc < OC) dbias[oc] = __float2bfloat16_rn(accumulate ? s + __bfloat162float(dbias[oc]) : s);
}
// Its lines: the sums of 1024 rows still take less than a second launch; its CTAs read 64 bytes of a row at a time, which beyond about 80 MB no longer come
// from L2 (us, two launches in brackets: 1024 x 2304 4.6 (5.6), 1024 x 28672 7.7 (13.8), 777 x 50304 14.1 (15.2), 1024 x 50304 24.8 (18.7), 384 x 128256
// 22.9 (18.3)); and of a few thousand CTAs each has little to do (1 x 128256 5.5 (3.1)).
constexpr int BG_FEW_ROWS = 1024, BG_FEW_COLS = 65536;
constexpr long long BG_FEW_VALUES = 40ll << 20;
bool bg_few(int rows, int OC) { return rows <= BG_FEW_ROWS && OC <= BG_FEW_COLS && (long long)rows * OC <= BG_FEW_VALUES; }

int bg_strips(int rows, int OC) {
    int sms = llmc_device_sm_count(); if (sms <= 0) sms = 148;
    int colgroups = CEIL_DIV(OC, 256);
    int strips = CEIL_DIV(4 * sms, colgroups);
    if (strips > CEIL_DIV(rows, BG_WARPS)) strips = CEIL_DIV(rows, BG_WARPS);
    if (strips < 1) strips = 1;
    return strips;
}

}  // namespace

extern "C" int llmc_gelu_fwd(bf16* out, const bf16* inp, long long n, cudaStream_t stream) {
    if (n % 8) return -1;
    CUDA_CHECK(launch_pdl(gelu_fwd_kernel, dim3((unsigned)CEIL_DIV(n / 8, 256)), dim3(256), 0, stream, 0, out, inp, n / 8));
    return 0;
}
extern "C" int llmc_gelu_bwd_inplace(bf16* d_inout, const bf16* inp, long long n, cudaStream_t stream) {
    if (n % 8) return -1;
    CUDA_CHECK(launch_pdl(gelu_bwd_kernel, dim3((unsigned)CEIL_DIV(n / 8, 256)), dim3(256), 0, stream, 0, d_inout, inp, n / 8));
    return 0;
}
extern "C" int llmc_residual_add(bf16* out, const bf16* a, const bf16* b, long long n, cudaStream_t stream) {
    if (n % 8) return -1;
    CUDA_CHECK(launch_pdl(residual_add_kernel, dim3((unsigned)CEIL_DIV(n / 8, 256)), dim3(256), 0, stream, 0, out, a, b, n / 8));
    return 0;
}
extern "C" long long llmc_bias_grad_scratch(int rows, int OC) { return bg_few(rows, OC) ? 0 : (long long)bg_strips(rows, OC) * OC; }
// dbias[c] (+)= sum_r dout[r, c]; scratch: llmc_bias_grad_scratch floats (none for few rows)
extern "C" int llmc_bias_grad(bf16* dbias, float* scratch, const bf16* dout, int rows, int OC, int accumulate, cudaStream_t stream) {
    if (OC % 8) return -1;
    if (bg_few(rows, OC)) {
        CUDA_CHECK(launch_pdl(bias_grad_few_kernel, dim3(CEIL_DIV(OC, 32)), dim3(4 * BGF_SLOTS), 0, stream, 0, dbias, dout, rows, OC, accumulate));
        return 0;
    }
    const int strips = bg_strips(rows, OC);
    const int rps = CEIL_DIV(rows, strips);
    CUDA_CHECK(launch_pdl(bias_grad_kernel, dim3(CEIL_DIV(OC, 256), strips), dim3(BG_WARPS * 32), 0, stream, 0, scratch, dout, rows, OC, rps));
    CUDA_CHECK(launch_pdl(bias_grad_fold_kernel, dim3(CEIL_DIV(OC, 16)), dim3(4 * BG_SLICES), 0, stream, 0, dbias, scratch, strips, OC, accumulate));
    return 0;
}
