// The launches of one pass of a LLaMA decoder with a key / value cache (models/generate.py, CachedDecoder.forward), issued from native code: embedding,
// per layer RMSNorm, QKV projection, rotary embedding into the cache, attention, projection, RMSNorm with residual, the SwiGLU MLP, at the end
// the LM head of the last positions.  No kernel of its own.  Issued from Python, a launch took the host 15 to 20 us: a prompt of 777 tokens in four layers
// was bound by the host (740 us against about 600 on the GPU).
#include "decoder_ops.h"

// Kernel of a forward product, chosen by the caller (ops/kernels.py, forward_kernel)
enum Product : int { GEMM = 0, GEMM2 = 1, STREAM = 2, GEMM2T = 3, SLICED = 4 };
// MLP: up-projections and activation in two launches, or one of the two fused forms
enum Mlp : int { MLP_TWO = 0, MLP_STREAM = 1, MLP_GEMM2T = 2 };

// Mirrored field by field by DecoderCall in _lib.py, which compares the sizes when it loads the library.
struct DecoderCall {
    // model: weights of layer l follow those of layer l - 1
    const bf16 *wte, *ln1w, *qkvw, *attprojw, *ln2w, *fc12w, *fcprojw, *lnfw, *lmhead;
    const float* freqs;
    // caches (L, max_batch, cache_len, NKV, HS)
    bf16 *kcache, *vcache;
    // activations, at least B * Tq rows (last, logits: B)
    bf16 *x, *ln, *raw, *q, *atty, *proj, *res, *fc12, *h, *last, *logits;
    float* logits32;                      // (B, vocab) logits as the caller wants them, for the streamed head (null: bf16 in logits)
    int* advance;                         // position to add 1 to, with logits32 (null: none)
    float* rstd;
    bf16* packed; float* lse;             // dense prompts only (null: attention over the cache)
    float* attention_ws;                  // of llmc_cached_attention, null where it needs none
    const int* tokens; const int* pos;    // pos: position on the device (null: start)
    int L, C, H, NH, NKV, HS, vocab_rows, logit_cols, vocab, freqs_len, max_batch, cache_len;
    int B, Tq, start;
    int how_qkv, how_attproj, how_fc12, how_fcproj, how_head, mlp;
    float eps;
};

namespace {
// In this chain the kernel in front of a product never writes weights, so that those that can do it read them while it drains.
int product(int how, bf16* out, const bf16* x, const bf16* w, int M, int N, int K, cudaStream_t s) {
    switch (how) {
        case GEMM2T: return llmc_gemm2t_chained(out, x, w, M, N, K, K, K, N, s);
        case STREAM: case SLICED: return llmc_stream_gemm_chained(out, x, w, M, N, K, K, K, N, how == SLICED ? 2 : 0, s);
        case GEMM2: return llmc_gemm2(x, w, out, nullptr, nullptr, M, N, K, K, K, N, 0, 0, 0, 0, 1, nullptr, nullptr, s);
        case GEMM: return llmc_gemm(x, w, out, nullptr, nullptr, M, N, K, K, K, N, 0, 0, 0, 0, 1, nullptr, nullptr, 0, s);
    }
    return -1;
}
}  // namespace

// Bytes of the argument, for a caller that declares it in another language
extern "C" int llmc_decoder_call_size() { return (int)sizeof(DecoderCall); }

// launches: number of kernels issued
extern "C" int llmc_decoder_forward(const DecoderCall* c, int* launches, cudaStream_t s) {
    const int N = c->B * c->Tq, C = c->C, H = c->H, QR = (c->NH + 2 * c->NKV) * c->HS;
    const size_t cache = (size_t)c->max_batch * c->cache_len * c->NKV * c->HS;
    const bool dense = c->packed != nullptr;
    int rc, n = 0;
#define GO(call) do { if ((rc = (call))) return rc; n++; } while (0)
    GO(llmc_encoder_fwd(c->x, c->tokens, c->wte, nullptr, c->B, c->Tq, C, c->vocab_rows, s));
    GO(llmc_rmsnorm_fwd(c->ln, c->rstd, c->x, c->ln1w, N, C, c->eps, s));
    for (int l = 0; l < c->L; l++) {
        bf16 *kc = c->kcache + l * cache, *vc = c->vcache + l * cache;
        GO(product(c->how_qkv, c->raw, c->ln, c->qkvw + (size_t)l * QR * C, N, QR, C, s));
        if (dense) {
            GO(llmc_rope_fwd_cache(c->packed, c->raw, c->freqs, kc, vc, c->cache_len, N, c->Tq, c->NH, c->NKV, c->HS, s));
            GO(llmc_attention_fwd(c->atty, c->lse, c->packed, c->B, c->Tq, c->NH, c->HS, s));
        } else if ((rc = llmc_cached_attention_rope(c->atty, c->raw, c->freqs, c->freqs_len, kc, vc, c->B, c->Tq, c->cache_len, c->start, c->NH, c->NKV, c->HS,
                                                    c->pos, c->attention_ws, 1, s)) != -6) {
            if (rc) return rc;
            n += c->attention_ws ? 2 : 1;
        } else {
            GO(llmc_rope_cache(c->q, kc, vc, c->raw, c->freqs, c->freqs_len, c->B, c->Tq, c->cache_len, c->start, c->NH, c->NKV, c->HS, c->pos, s));
            GO(llmc_cached_attention(c->atty, c->q, kc, vc, c->B, c->Tq, c->cache_len, c->start, c->NH, c->NKV, c->HS, c->pos, c->attention_ws, s));
            if (c->attention_ws) n++;
        }
        GO(product(c->how_attproj, c->proj, c->atty, c->attprojw + (size_t)l * C * C, N, C, C, s));
        GO(llmc_rmsnorm_fused_residual_fwd(c->res, c->ln, c->rstd, c->x, c->proj, c->ln2w + (size_t)l * C, N, C, c->eps, s));
        const bf16* w12 = c->fc12w + (size_t)l * 2 * H * C;
        if (c->mlp == MLP_STREAM) {
            GO(llmc_stream_gemm_swiglu_chained(c->h, c->ln, w12, N, H, C, C, C, H, s));
        } else if (c->mlp == MLP_GEMM2T) {
            GO(llmc_gemm2t_swiglu_chained(c->h, c->ln, w12, N, H, C, C, C, H, s));
        } else {
            GO(product(c->how_fc12, c->fc12, c->ln, w12, N, 2 * H, C, s));
            GO(llmc_swiglu_fwd(c->h, c->fc12, N, H, s));
        }
        GO(product(c->how_fcproj, c->proj, c->h, c->fcprojw + (size_t)l * C * H, N, C, H, s));
        GO(llmc_rmsnorm_fused_residual_fwd(c->x, c->ln, c->rstd, c->res, c->proj, l + 1 < c->L ? c->ln1w + (size_t)(l + 1) * C : c->lnfw, N, C, c->eps, s));
    }
    const bf16* last = c->ln;                           // one token per row: the last positions are the rows themselves
    if (c->Tq > 1) {
        CUDA_CHECK(cudaMemcpy2DAsync(c->last, (size_t)C * 2, c->ln + (size_t)(c->Tq - 1) * C, (size_t)c->Tq * C * 2, (size_t)C * 2, c->B,
                                     cudaMemcpyDeviceToDevice, s));
        last = c->last;
    }
    if (c->logits32) GO(llmc_stream_gemm_logits(c->logits32, c->vocab, last, c->lmhead, c->B, c->logit_cols, C, C, C, c->advance, s));
    else GO(product(c->how_head, c->logits, last, c->lmhead, c->B, c->logit_cols, C, s));
#undef GO
    *launches = n;
    return 0;
}
