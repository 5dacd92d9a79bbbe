"""Thin launchers of the sm_100a kernels: tensors in, C entry points out (see csrc/*.cu)."""
import contextlib
import ctypes
import os
import threading

import torch

from .. import _lib
from .._lib import TensorTable, check

MODE_STORE, MODE_GELU, MODE_DGELU, MODE_ACCUM = 0, 1, 2, 3

_launches = 0   # number of kernel-library launches issued (bench.py reports it)
# forward / dgrad GEMMs with at least this many 256 x 256 tiles run on the two-SM kernel (gemm2.cu); 0 disables it
TWO_SM_MIN_TILES = int(os.environ.get("LLMC_GEMM_2SM_MIN_TILES", "74"))

# products of at most this many rows may stream the weights through split-K clusters whatever their depth (_few_rows)
STREAM_MAX_ROWS = 128


def launch_count():
    return _launches


def count_launches(n):
    """Adds launches issued without a launcher call (a replayed graph)."""
    global _launches
    _launches += n


def _stream():
    return ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)


def _p(t):
    return ctypes.c_void_p(t.data_ptr()) if t is not None else ctypes.c_void_p(0)


class _Taken(threading.local):
    by = None                                # list that collects what this thread's calls take (scratch_taken)


class _Scratch:
    """Per-device scratch buffers that grow to the largest request and are then reused."""

    def __init__(self):
        self.bufs = {}
        self.taken = _Taken()

    def get(self, key, numel, dtype, device, zero=False):
        k = (key, device.index, dtype)
        t = self.bufs.get(k)
        if t is None or t.numel() < numel:
            t = (torch.zeros if zero else torch.empty)(max(int(numel), 1), dtype=dtype, device=device)
            self.bufs[k] = t
        if self.taken.by is not None:
            self.taken.by.append(t)
        return t


_scratch = _Scratch()


@contextlib.contextmanager
def scratch_taken():
    """A list of the scratch buffers that this thread's calls take inside the block.  A later call that needs a larger one replaces a buffer, so
    a CUDA graph captured in the block has to keep the list."""
    outer = _scratch.taken.by
    _scratch.taken.by = by = []
    try:
        yield by
    finally:
        _scratch.taken.by = outer
        if outer is not None:
            outer += by


_sm_count = {}


def sm_count(device):
    idx = device.index if device.index is not None else torch.cuda.current_device()
    if idx not in _sm_count:
        _sm_count[idx] = torch.cuda.get_device_properties(idx).multi_processor_count
    return _sm_count[idx]


def _few_rows(M, N, K, mode, b_mn, device):
    """Whether a plain product goes to the split-K kernel with 128 x 256 tiles of csrc/stream_gemm.cu.  The lines are where it overtakes the other
    two kernels (M from 100 to 2048, fourteen pairs of N and K, us): deep products whose tiles leave at least half of the SMs idle
    (K = 3072: 24 tiles 21 against 27, 36 tiles 33 against 27; K = 7168: 64 tiles 37 to 43 against 53, 96 tiles 61 against 55), and
    at most 128 rows, unless there are more weight tiles than resident CTAs (64 rows and more, _wide) or the product is a shallow input gradient
    (100 x 768 x 768: 16 against 14).  Input gradients of more than 128 rows go there as long as four slices of K of row tiles of at most 128
    rows are resident at once and K pays for the reduction, which grows with the number of tiles (in a chain, theirs in brackets: 130 x 512 x 768
    4.4 (6.3), 256 x 768 x 768 4.9 (6.3), x 2304 7.0 (13.0), x 3072 7.9 (16.3), 512 x 768 x 768 6.1 (6.4), 1024 x 768 x 1600 9.8 (10.4),
    1024 x 1024 x 2304 11.7 (13.9); 384 x 2048 x 1024 8.3 (7.8), 1024 x 768 x 1024 8.5 (7.8), 512 x 1600 x 1600 10.7 (10.4)).  Forward products of more than 128 rows
    that are cut into small row tiles too have a rule of their own (``_sliced``).  At most 128 rows are summed in slices from K = 512 on, in fp32 and in slice order."""
    if mode != MODE_STORE:
        return False
    wtiles = (N + 127) // 128
    tiles = (M + 255) // 256 * wtiles
    if (K >= 6144 and tiles <= 64) or (b_mn and K >= 3072 and tiles <= 32):
        return True
    if b_mn and M > STREAM_MAX_ROWS:
        return _slices_pay(M, wtiles, K, device)
    if b_mn:
        return K >= 2048 and wtiles <= 2 * sm_count(device)
    return M <= 64 or (M <= STREAM_MAX_ROWS and wtiles <= 2 * sm_count(device))


def _slices_pay(M, wtiles, K, device):
    narrow = (M + 127) // 128 * wtiles
    return K >= max(768, 32 * narrow) and narrow * 4 <= 2 * (sm_count(device) * 7 // 8)


def _sliced(M, N, K, device):
    """Whether a forward product of more than 128 rows goes to the split-K kernel with row tiles and slices like an input gradient's.  The line is the input
    gradients' one: below it (fewer tiles, deeper) the slices win over the swapped kernel's one sum over K, above it they lose.  us in a chain, the swapped
    kernel in brackets: 129 x 768 x 768 4.7 (6.0), 256 x 768 x 768 5.1 (6.2), 512 x 768 x 768 6.3 (6.3), 256 x 768 x 3072 7.9 (14.1), 1024 x 768 x 3072 12.1
    (15.1), 256 x 384 x 1536 5.9 (8.8), 512 x 1024 x 1024 7.0 (7.3), 1024 x 1024 x 4096 14.7 (18.7), 512 x 2048 x 2048 11.2 (11.7); from K = 6144 on,
    where products of few tiles went to the split-K kernel in large row tiles before, in brackets, 220 x 192 x 13312 12.0 (16.1), 554 x 704 x 6400 14.9 (16.4); beyond the line
    256 x 2304 x 768 7.6 (6.4), 777 x 1024 x 1024 8.7 (8.0), 2048 x 768 x 3072 21 (15).  The sums are fp32 and added in slice order."""
    return M > STREAM_MAX_ROWS and K % 8 == 0 and _slices_pay(M, (N + 127) // 128, K, device)


def _wide(M, N, device):
    """Whether a plain forward product goes to the CTAs of csrc/stream_gemm.cu that stay for several weight tiles: at most 128 rows and more tiles
    than resident CTAs (100 x 50304 x 768 16 us against 22 in 256-column tiles, 128 x 128256 x 2048 96 against 108)."""
    return M <= STREAM_MAX_ROWS and (N + 127) // 128 > 2 * sm_count(device)


def _swapped(M, N, K, device):
    """Whether a plain forward product goes to the two-SM kernel with swapped operand roles (csrc/gemm2t.cu), whose row tiles fit the rows: as long as
    the tiles fill few rounds of the CTA pairs and K is deep enough to hide its epilogue in pieces of 16 rows.  Same bits as the other two kernels.
    us, theirs in brackets: 777 x 3072 x 2048 12.7 (18.5), 777 x 14336 x 2048 40 (49), 500 x 6144 x 4096 23 (30),
    256 x 2304 x 768 6.5 (6.8), 256 x 50304 x 768 25.5 (28.0); 512 x 1152 x 384 5.5 (5.1), 3001 x 28672 x 4096 522 (491).  Above 2048 rows, where a chain
    of products runs at the power limit, the larger loads count: the MLP of 3001 rows of 4096 channels takes 2683 instead of 2663 us with its
    down-projection here, although that alone is faster (267 against 294).
    Deep products with few tiles are left to the split-K kernel: 300 x 2048 x 7168 33 against 20, 300 x 4096 x 14336 51 against 47.  At the line the two
    are level: 500 x 4096 x 14336 57 to 78 against 60 to 75, 777 x 2048 x 7168 29 to 37 against 32 to 35, whole prompts of 500 to 1024 tokens within 1 %."""
    mt = (M + 255) // 256
    if not (128 < M <= 2048 and K >= 768 and K % 8 == 0 and mt * ((N + 255) // 256) <= 5 * sm_count(device)):
        return False
    split = mt * ((N + 127) // 128)
    return K < 6144 or split > 64 or (split > 32 and M > 384)


def _wgrad_two_sm(tiles256, K, accumulate, device):
    """Whether a weight gradient over K rows goes to the two-SM kernel.  Over few rows it is mostly its output: where 256 x 256 tiles leave half of the
    CTA pairs idle, narrower tiles of single SMs keep more of them busy (us on pairs, single SMs in brackets: 2304 x 768 x 256 7.4 (6.2), x 1024 13.3
    (10.0), 3072 x 768 x 256 7.5 (6.4); with more tiles 1600 x 1600 x 256 7.6 (9.0), 3072 x 1024 x 1024 11.4 (12.8), 4096 x 1024 x 64 7.1 (7.3)).  Where it
    adds to what is there the pairs fetch that by TMA before the sum is ready, single SMs a row per thread in the epilogue (2304 x 768 x 256 8.0
    (10.6), 1600 x 1600 x 256 8.3 (15.8))."""
    if tiles256 < 8:
        return False
    return K > 1024 or bool(accumulate) or tiles256 * 4 > sm_count(device)


FORWARD_GEMM, FORWARD_GEMM2, FORWARD_STREAM, FORWARD_SWAPPED, FORWARD_SLICED = range(5)        # csrc/decoder.cu, Product


def forward_kernel(M, N, K, device, aligned=True):
    """The kernel of a plain forward product without flags to wait for.  ``aligned``: the output starts on a 16-byte boundary.  The swapped kernel stores
    with TMA, which needs that and rows of whole 16 bytes; the split-K kernel takes any number of columns and any alignment."""
    if TWO_SM_MIN_TILES > 0 and _sliced(M, N, K, device):
        return FORWARD_SLICED
    if TWO_SM_MIN_TILES > 0 and N % 8 == 0 and aligned and _swapped(M, N, K, device):
        return FORWARD_SWAPPED
    if _few_rows(M, N, K, MODE_STORE, False, device) or _wide(M, N, device):
        return FORWARD_STREAM
    tiles256 = ((M + 255) // 256) * ((N + 255) // 256)
    return FORWARD_GEMM2 if TWO_SM_MIN_TILES > 0 and tiles256 >= TWO_SM_MIN_TILES else FORWARD_GEMM


def gemm(a, b, d, M, N, K, lda, ldb, ldd, a_mn, b_mn, mode, bias=None, aux=None, accumulate=False, splits=1, max_ctas=0, ready=None):
    """Dispatches to the split-K kernel for plain products with few tiles (``_few_rows``, ``_wide``), to one of the two-SM kernels (``_swapped``; 256 x 256 tiles on
    CTA pairs) for problems with enough tiles, else to the single-CTA one.
    ``ready`` (an object with flags_ptr, n, seq and wait()) marks the B operand as the target of an all-gather in flight: the
    two-SM kernel polls the peers' flags itself before its first load; the single-CTA kernel runs after ``ready.wait()``."""
    global _launches
    lib = _lib.cuda()
    _launches += 1
    plain = forward_kernel(M, N, K, d.device, d.data_ptr() % 16 == 0) if mode == MODE_STORE and not a_mn and not b_mn else None
    if plain == FORWARD_SWAPPED and ready is None:
        check(lib.llmc_gemm2t(_p(d), _p(a), _p(b), _p(bias), M, N, K, lda, ldb, ldd, 0, _stream()), "llmc_gemm2t")
        return
    if plain == FORWARD_SLICED and ready is None:
        check(lib.llmc_stream_gemm(_p(d), _p(a), _p(b), _p(bias), M, N, K, lda, ldb, ldd, 2, _stream()), "llmc_stream_gemm")
        return
    if plain == FORWARD_STREAM or (not a_mn and _few_rows(M, N, K, mode, b_mn, d.device)):
        if ready is not None:
            ready.wait()
        check(lib.llmc_stream_gemm(_p(d), _p(a), _p(b), _p(bias), M, N, K, lda, ldb, ldd, int(b_mn), _stream()), "llmc_stream_gemm")
        return
    tiles256 = ((M + 255) // 256) * ((N + 255) // 256)
    if mode == MODE_ACCUM:
        two_sm = TWO_SM_MIN_TILES > 0 and a_mn and b_mn and _wgrad_two_sm(tiles256, K, accumulate, d.device)
        if not two_sm and K <= 1024:
            splits = 1
    else:
        two_sm = TWO_SM_MIN_TILES > 0 and not a_mn and tiles256 >= TWO_SM_MIN_TILES
    ws = cnt = None
    if two_sm:
        if mode == MODE_ACCUM:
            splits = lib.llmc_gemm2_pick_splits(M, N, K, sm_count(d.device))
            wsf, nc = ctypes.c_longlong(0), ctypes.c_int(0)
            lib.llmc_gemm2_workspace(M, N, splits, ctypes.byref(wsf), ctypes.byref(nc))
            if splits > 1:
                ws = _scratch.get("gemm_ws", wsf.value, torch.float32, d.device)
            cnt = _scratch.get("gemm2_cnt", nc.value, torch.int32, d.device, zero=True)
        if ready is not None:
            check(lib.llmc_gemm2_after_flags(_p(a), _p(b), _p(d), _p(bias), _p(aux), M, N, K, lda, ldb, ldd, int(a_mn), int(b_mn), mode,
                                             int(accumulate), splits, _p(ws), _p(cnt), ctypes.c_void_p(ready.flags_ptr), ready.n, ready.seq,
                                             _stream()), "llmc_gemm2_after_flags")
            return
        check(lib.llmc_gemm2(_p(a), _p(b), _p(d), _p(bias), _p(aux), M, N, K, lda, ldb, ldd, int(a_mn), int(b_mn), mode, int(accumulate), splits,
                             _p(ws), _p(cnt), _stream()), "llmc_gemm2")
        return
    if ready is not None:
        ready.wait()
    if mode == MODE_ACCUM and splits > 1:
        wsf, nc = ctypes.c_longlong(0), ctypes.c_int(0)
        lib.llmc_gemm_workspace(M, N, splits, ctypes.byref(wsf), ctypes.byref(nc))
        ws = _scratch.get("gemm_ws", wsf.value, torch.float32, d.device)
        cnt = _scratch.get("gemm_cnt", nc.value, torch.int32, d.device, zero=True)
    check(lib.llmc_gemm(_p(a), _p(b), _p(d), _p(bias), _p(aux), M, N, K, lda, ldb, ldd, int(a_mn), int(b_mn), mode,
                        int(accumulate), splits, _p(ws), _p(cnt), max_ctas, _stream()), "llmc_gemm")


def _too_small(op, **tensors):
    """The launchers take the sizes of a product from two of its operands; the others have to be at least that large."""
    return ValueError("%s: operands of shapes %s do not fit one product" % (op, {n: tuple(t.shape) for n, t in tensors.items() if t is not None}))


def matmul_forward(out, inp, weight, bias=None, pre_gelu=None, ready=None):
    """out[M,OC] = inp[M,C] @ weight[OC,C]^T (+ bias).  With ``pre_gelu`` the pre-activation is stored there and
    ``out`` receives its tanh-GELU (reference: matmul_forward_cublaslt, llmc/matmul.cuh:230-242)."""
    M, C = inp.shape
    OC = weight.shape[0]
    n = M * OC
    if out.numel() < n or weight.numel() < OC * C or (bias is not None and bias.numel() < OC) or (pre_gelu is not None and pre_gelu.numel() < n):
        raise _too_small("matmul_forward", out=out, inp=inp, weight=weight, bias=bias, pre_gelu=pre_gelu)
    mode = MODE_GELU if pre_gelu is not None else MODE_STORE
    gemm(inp, weight, out, M, OC, C, C, C, OC, 0, 0, mode, bias=bias, aux=pre_gelu, ready=ready)


def matmul_dgrad(dinp, dout, weight, pre_gelu=None):
    """dinp[M,C] = dout[M,OC] @ weight[OC,C]; multiplied by GELU'(pre_gelu[M,C]) if given
    (reference: matmul_backward dgrad with the DGELU epilogue, llmc/matmul.cuh:279-285)."""
    M, OC = dout.shape
    C = weight.shape[1]
    n = M * C
    if dinp.numel() < n or weight.shape[0] < OC or (pre_gelu is not None and pre_gelu.numel() < n):
        raise _too_small("matmul_dgrad", dinp=dinp, dout=dout, weight=weight, pre_gelu=pre_gelu)
    mode = MODE_DGELU if pre_gelu is not None else MODE_STORE
    gemm(dout, weight, dinp, M, C, OC, OC, C, C, 0, 1, mode, aux=pre_gelu)


def matmul_wgrad(dweight, dout, inp, accumulate=True):
    """dweight[OC,C] (+)= dout[M,OC]^T @ inp[M,C] with split-K sized to fill the SMs."""
    M, OC = dout.shape
    C = inp.shape[1]
    if dweight.numel() < OC * C or inp.shape[0] < M:
        raise _too_small("matmul_wgrad", dweight=dweight, dout=dout, inp=inp)
    splits = _lib.cuda().llmc_gemm_pick_splits(OC, C, M, sm_count(dout.device))
    gemm(dout, inp, dweight, OC, C, M, OC, C, C, 1, 1, MODE_ACCUM, accumulate=accumulate, splits=splits)


def gemm_tf32(d, a, b, bias=None, accumulate=False):
    """d[M,N] (+)= a[M,K] @ b[N,K]^T (+ bias): fp32 tensors, tcgen05 kind::tf32 with fp32 accumulation (the matmul of the
    full-precision mode; the reference runs cuBLAS in TF32 there when -f 1, train_gpt2_fp32.cu / PRECISION=FP32)."""
    global _launches
    M, K = a.shape
    N = b.shape[0]
    assert a.dtype == b.dtype == d.dtype == torch.float32 and b.shape[1] == K and tuple(d.shape) == (M, N)
    assert a.stride(1) == 1 and b.stride(1) == 1 and d.stride(1) == 1
    _launches += 1
    check(_lib.cuda().llmc_gemm_tf32(_p(a), _p(b), _p(d), _p(bias), M, N, K, a.stride(0), b.stride(0), d.stride(0), int(accumulate), _stream()),
          "llmc_gemm_tf32")


def tf32_shapes_ok(*dims):
    return all(int(x) % 4 == 0 for x in dims)


def bias_grad(dbias, dout, accumulate=True):
    """dbias[OC] (+)= column sums of dout[M,OC]."""
    global _launches
    lib = _lib.cuda()
    M, OC = dout.shape
    words = lib.llmc_bias_grad_scratch(M, OC)
    s = _scratch.get("bias_grad", words, torch.float32, dout.device)
    _launches += 2 if words else 1
    check(lib.llmc_bias_grad(_p(dbias), _p(s), _p(dout), M, OC, int(accumulate), _stream()), "llmc_bias_grad")


def encoder_forward(out, tokens, wte, wpe):
    """out[B,T,C] = wte[tokens] + wpe[:T]."""
    global _launches
    B, T = tokens.shape
    C = wte.shape[1]
    _launches += 1
    check(_lib.cuda().llmc_encoder_fwd(_p(out), _p(tokens), _p(wte), _p(wpe), B, T, C, wte.shape[0], _stream()), "llmc_encoder_fwd")


def encoder_backward(dwte, dwpe, dout, tokens, accumulate_wte=True, accumulate_wpe=True, seed=0):
    """Deterministic scatter-add of dout[B,T,C] into the embedding gradients."""
    global _launches
    B, T = tokens.shape
    C = dwte.shape[1]
    V = dwte.shape[0]
    _launches += 2
    check(_lib.cuda().llmc_encoder_bwd(_p(dwte), _p(dwpe), _p(dout), _p(tokens), B, T, C, V, int(accumulate_wte),
                                       int(accumulate_wpe), seed & 0xFFFFFFFF, _stream()), "llmc_encoder_bwd")


def layernorm_forward(out, mean, rstd, inp, weight, bias):
    global _launches
    N, C = inp.shape
    _launches += 1
    check(_lib.cuda().llmc_layernorm_fwd(_p(out), _p(mean), _p(rstd), _p(inp), _p(weight), _p(bias), N, C, _stream()),
          "llmc_layernorm_fwd")


def fused_residual_forward(residual, normed, mean, rstd, inp1, inp2, weight, bias):
    """residual = inp1 + inp2; normed = LayerNorm(residual)."""
    global _launches
    N, C = inp1.shape
    _launches += 1
    check(_lib.cuda().llmc_fused_residual_fwd(_p(residual), _p(normed), _p(mean), _p(rstd), _p(inp1), _p(inp2), _p(weight),
                                              _p(bias), N, C, _stream()), "llmc_fused_residual_fwd")


def layernorm_backward(dinp, dweight, dbias, dout, inp, weight, mean, rstd, accumulate_dinp=True, accumulate_dwdb=True,
                       dcolsum=None, accumulate_dcol=True, sums_in=None, dinp_old=None):
    """dinp (+)= dLN(dout), added to ``dinp_old`` if that is given; dweight/dbias (+)= their gradients.  ``dcolsum`` (+)= column sums of the final dinp: the bias
    gradient of the projection that wrote into the residual stream, at no extra pass over memory.  ``sums_in()`` may give a
    context (another stream) in which the three column sums are finished; the next call has to follow them."""
    global _launches
    lib = _lib.cuda()
    N, C = inp.shape
    s = _scratch.get("ln_bwd", lib.llmc_layernorm_bwd_scratch(N, C), torch.float32, inp.device)
    _launches += 2
    args = (_p(dinp), _p(dweight), _p(dbias), _p(s), _p(dout), _p(inp), _p(weight), _p(mean), _p(rstd),
            N, C, int(accumulate_dinp), int(accumulate_dwdb), _p(dcolsum), int(accumulate_dcol))
    if sums_in is None:
        check(lib.llmc_layernorm_bwd_parts(*args, _p(dinp_old), 3, _stream()), "llmc_layernorm_bwd_parts")
        return
    check(lib.llmc_layernorm_bwd_parts(*args, _p(dinp_old), 1, _stream()), "llmc_layernorm_bwd_parts")
    with sums_in():
        check(lib.llmc_layernorm_bwd_parts(*args, _p(dinp_old), 2, _stream()), "llmc_layernorm_bwd_parts")


def attention_forward(out, lse, qkv, B, T, NH):
    """out (B,T,NH,HS), lse (B,NH,T) from packed qkv (B,T,3,NH,HS); causal."""
    global _launches
    hs = qkv.numel() // (B * T * 3 * NH)
    _launches += 1
    check(_lib.cuda().llmc_attention_fwd(_p(out), _p(lse), _p(qkv), B, T, NH, hs, _stream()), "llmc_attention_fwd")


def attention_backward(dqkv, dout, qkv, out, lse, B, T, NH):
    """dqkv (B,T,3,NH,HS) from dout, the forward inputs and statistics; deterministic."""
    global _launches
    hs = qkv.numel() // (B * T * 3 * NH)
    lib = _lib.cuda()
    # row statistics and, for 64-wide heads, the dQ contributions of the single-pass kernel's units (csrc/attention_bwd1.cu)
    ws = _scratch.get("attn_bwd", lib.llmc_attention_bwd_workspace(B, T, NH, hs), torch.float32, qkv.device)
    _launches += lib.llmc_attention_bwd_launches(B, T, NH, hs)
    check(lib.llmc_attention_bwd(_p(dqkv), _p(ws), _p(dout), _p(qkv), _p(out), _p(lse), B, T, NH, hs, _stream()),
          "llmc_attention_bwd")


def fused_classifier(logits, losses, targets, dloss, V, write_dlogits=True, accumulate_loss=False):
    """losses[n] (+)= CE(logits[n], targets[n]); logits <- dlogits * dloss in place."""
    global _launches
    N, Vp = logits.shape
    _launches += 1
    check(_lib.cuda().llmc_fused_classifier(_p(logits), _p(losses), _p(targets), float(dloss), N, V, Vp, int(write_dlogits),
                                            int(accumulate_loss), _stream()), "llmc_fused_classifier")


def gelu_forward(out, inp):
    global _launches
    _launches += 1
    check(_lib.cuda().llmc_gelu_fwd(_p(out), _p(inp), inp.numel(), _stream()), "llmc_gelu_fwd")


def gelu_backward_inplace(d_inout, inp):
    global _launches
    _launches += 1
    check(_lib.cuda().llmc_gelu_bwd_inplace(_p(d_inout), _p(inp), inp.numel(), _stream()), "llmc_gelu_bwd_inplace")


def residual_add(out, a, b):
    global _launches
    _launches += 1
    check(_lib.cuda().llmc_residual_add(_p(out), _p(a), _p(b), a.numel(), _stream()), "llmc_residual_add")


def rmsnorm_forward(out, rstd, inp, weight, eps=1e-5):
    """out = inp * rsqrt(mean(inp^2) + eps) * weight, statistics in fp32 (reference module: train_llama3.py:133-146)."""
    global _launches
    N, C = inp.shape
    _launches += 1
    check(_lib.cuda().llmc_rmsnorm_fwd(_p(out), _p(rstd), _p(inp), _p(weight), N, C, float(eps), _stream()), "llmc_rmsnorm_fwd")


def rmsnorm_fused_residual_forward(residual, normed, rstd, inp1, inp2, weight, eps=1e-5):
    """residual = inp1 + inp2; normed = RMSNorm(residual)."""
    global _launches
    N, C = inp1.shape
    _launches += 1
    check(_lib.cuda().llmc_rmsnorm_fused_residual_fwd(_p(residual), _p(normed), _p(rstd), _p(inp1), _p(inp2), _p(weight), N, C,
                                                      float(eps), _stream()), "llmc_rmsnorm_fused_residual_fwd")


def rmsnorm_backward(dinp, dweight, dout, inp, weight, rstd, accumulate_dinp=True, accumulate_dw=True):
    """dinp (+)= dRMSNorm(dout); dweight (+)= its gradient."""
    global _launches
    lib = _lib.cuda()
    N, C = inp.shape
    s = _scratch.get("rms_bwd", lib.llmc_rmsnorm_bwd_scratch(N, C), torch.float32, inp.device)
    _launches += 2
    check(lib.llmc_rmsnorm_bwd(_p(dinp), _p(dweight), _p(s), _p(dout), _p(inp), _p(weight), _p(rstd), N, C, int(accumulate_dinp),
                               int(accumulate_dw), _stream()), "llmc_rmsnorm_bwd")


def rope_forward(packed, raw, freqs, T, NH, NKV, kcache=None, vcache=None):
    """raw (N, (NH + 2 NKV) * HS) -> packed (N, 3, NH, HS): rotary embedding on queries and keys, key / value heads repeated
    NH / NKV times (reference: apply_rotary_emb + repeat_kv, train_llama3.py:107-117 and :59-68).  freqs: (maxT, HS/2, 2) fp32.
    kcache, vcache (B, >= T, NKV, HS), contiguous: the rotated keys and the values of the B = N / T sequences also go to their first T entries."""
    global _launches
    N = raw.shape[0]
    HS = raw.shape[1] // (NH + 2 * NKV)
    _launches += 1
    if kcache is not None:
        B = N // T
        if B * T != N or kcache.shape != vcache.shape or tuple(kcache.shape[2:]) != (NKV, HS) or kcache.shape[0] < B or kcache.shape[1] < T \
                or not (kcache.is_contiguous() and vcache.is_contiguous()):
            raise ValueError("rope_forward: caches of shape %s do not hold %d tokens of sequences of %d" % (tuple(kcache.shape), N, T))
        check(_lib.cuda().llmc_rope_fwd_cache(_p(packed), _p(raw), _p(freqs), _p(kcache), _p(vcache), kcache.shape[1], N, T, NH, NKV, HS, _stream()),
              "llmc_rope_fwd_cache")
        return
    check(_lib.cuda().llmc_rope_fwd(_p(packed), _p(raw), _p(freqs), N, T, NH, NKV, HS, _stream()), "llmc_rope_fwd")


def rope_backward(draw, dpacked, freqs, T, NH, NKV):
    """Gradient of ``rope_forward``: inverse rotation, gradients of repeated heads summed over their group."""
    global _launches
    N = draw.shape[0]
    HS = draw.shape[1] // (NH + 2 * NKV)
    _launches += 1
    check(_lib.cuda().llmc_rope_bwd(_p(draw), _p(dpacked), _p(freqs), N, T, NH, NKV, HS, _stream()), "llmc_rope_bwd")


def swiglu_forward(h, x12):
    """h = x12[:, :H] * silu(x12[:, H:])."""
    global _launches
    N, H = h.shape
    _launches += 1
    check(_lib.cuda().llmc_swiglu_fwd(_p(h), _p(x12), N, H, _stream()), "llmc_swiglu_fwd")


def swiglu_backward(dx12, dh, x12):
    """dx12 = gradient of ``swiglu_forward`` with respect to both halves of x12."""
    global _launches
    N, H = dh.shape
    _launches += 1
    check(_lib.cuda().llmc_swiglu_bwd(_p(dx12), _p(dh), _p(x12), N, H, _stream()), "llmc_swiglu_bwd")


def rope_cache(q, kcache, vcache, raw, freqs, Tq, start_pos, NH, NKV, pos=None):
    """Rotary embedding of the Tq new tokens per batch row at positions start_pos.., queries to ``q`` (N, NH, HS), rotated keys
    and the values into their slots of the caches (B, Tmax, NKV, HS) (reference: CausalSelfAttention.forward with
    ``use_kv``, train_llama3.py:167-180).  ``pos`` (a one-element int32 device tensor) replaces start_pos at run time, for
    steps that are replayed from a CUDA graph."""
    global _launches
    N = raw.shape[0]
    HS = raw.shape[1] // (NH + 2 * NKV)
    _launches += 1
    check(_lib.cuda().llmc_rope_cache(_p(q), _p(kcache), _p(vcache), _p(raw), _p(freqs), freqs.shape[0], N // Tq, Tq, kcache.shape[1],
                                      start_pos, NH, NKV, HS, _p(pos), _stream()), "llmc_rope_cache")


def cached_attention(out, q, kcache, vcache, Tq, start_pos, NH, NKV, pos=None):
    """out (N, NH, HS): causal attention of the Tq new queries per batch row over cache positions 0 .. start_pos + t."""
    global _launches
    lib = _lib.cuda()
    N = q.shape[0]
    HS = kcache.shape[-1]
    B, Tmax = N // Tq, kcache.shape[1]
    # decoding steps (few query rows per cached head, head width 64 or 128) take the split-key kernel; a workspace only for more key
    # slices than a cluster holds
    words = lib.llmc_cached_attention_workspace(B, Tq, Tmax, NH, NKV, HS)
    ws = _scratch.get("cached_attention", words, torch.float32, q.device) if words > 0 else None
    _launches += 2 if words > 0 else 1
    check(lib.llmc_cached_attention(_p(out), _p(q), _p(kcache), _p(vcache), B, Tq, Tmax, start_pos, NH, NKV, HS, _p(pos), _p(ws), _stream()),
          "llmc_cached_attention")


def rope_cached_attention(out, q, kcache, vcache, raw, freqs, Tq, start_pos, NH, NKV, pos=None):
    """``rope_cache`` and ``cached_attention`` on its results; ``q`` is scratch.  Decoding steps run in one launch, with the same bits (a step of 4 rows, 4 layers of 2048
    channels: 266 us, in two launches per layer 271; of 32 rows, 4 layers of 4096 channels: 763, 773)."""
    global _launches
    lib = _lib.cuda()
    N, HS = raw.shape[0], kcache.shape[-1]
    B, Tmax = N // Tq, kcache.shape[1]
    words = lib.llmc_cached_attention_workspace(B, Tq, Tmax, NH, NKV, HS)
    ws = _scratch.get("cached_attention", words, torch.float32, raw.device) if words > 0 else None
    rc = lib.llmc_cached_attention_rope(_p(out), _p(raw), _p(freqs), freqs.shape[0], _p(kcache), _p(vcache), B, Tq, Tmax, start_pos, NH, NKV, HS, _p(pos), _p(ws), 0, _stream())
    if rc != -6:
        check(rc, "llmc_cached_attention_rope")
        _launches += 2 if words > 0 else 1
        return
    rope_cache(q, kcache, vcache, raw, freqs, Tq, start_pos, NH, NKV, pos)
    cached_attention(out, q, kcache, vcache, Tq, start_pos, NH, NKV, pos)


def matmul_skinny(out, inp, weight):
    """out[M,OC] = inp[M,C] @ weight[OC,C]^T for at most 8 rows on warp-level MMAs (csrc/decode.cu); ``matmul_forward`` takes such products too, faster
    behind another kernel of this library and slower alone."""
    global _launches
    M, C = inp.shape
    OC = weight.shape[0]
    if out.shape[0] < M or out.shape[-1] < OC or weight.shape[1] < C:
        raise _too_small("matmul_skinny", out=out, inp=inp, weight=weight)
    _launches += 1
    check(_lib.cuda().llmc_skinny_gemm(_p(out), _p(inp), _p(weight), M, OC, C, inp.stride(0), weight.stride(0), out.stride(0), _stream()),
          "llmc_skinny_gemm")


def matmul_swiglu(h, inp, weight12):
    """h[M,H] = (inp @ w1^T) * silu(inp @ w2^T) with weight12 = [w1; w2] (2H, C), at most 128 rows, H a multiple of 64: the
    up-projections of a decoding step and their activation in one launch (csrc/stream_gemm.cu)."""
    global _launches
    M, C = inp.shape
    H = weight12.shape[0] // 2
    if h.shape[0] < M or h.shape[-1] < H or weight12.shape[1] < C:
        raise _too_small("matmul_swiglu", h=h, inp=inp, weight12=weight12)
    _launches += 1
    check(_lib.cuda().llmc_stream_gemm_swiglu(_p(h), _p(inp), _p(weight12), M, H, C, inp.stride(0), weight12.stride(0), h.stride(0), _stream()),
          "llmc_stream_gemm_swiglu")


def matmul_swiglu_prompt(h, inp, weight12):
    """``matmul_swiglu`` for any number of rows, H a multiple of 128: two-SM tiles (csrc/gemm2t.cu).  us, the product and its activation in launches of their
    own in brackets: 2048 channels and 7168 hidden units, 129 rows 16.4 (14.7), 777 43.7 (43.6), 2048 85 (95), 8192 312 (420)."""
    global _launches
    M, C = inp.shape
    H = weight12.shape[0] // 2
    if h.shape[0] < M or h.shape[-1] < H or weight12.shape[1] < C:
        raise _too_small("matmul_swiglu_prompt", h=h, inp=inp, weight12=weight12)
    _launches += 1
    check(_lib.cuda().llmc_gemm2t_swiglu(_p(h), _p(inp), _p(weight12), M, H, C, inp.stride(0), weight12.stride(0), h.stride(0), 0, _stream()),
          "llmc_gemm2t_swiglu")


def decoder_layout_ok(decoder):
    """Whether ``decoder_forward`` can take this decoder's tensors: it finds a layer's weights and cache by their distance from the first layer's and
    none of the operators' size checks stands between it and the kernels.  Called operator by operator every layer may lie anywhere."""
    cfg, p = decoder.model.cfg, decoder.model.params
    L, C, H, QR = cfg.num_layers, cfg.channels, cfg.hidden_dim, (cfg.num_heads + 2 * cfg.num_kv_heads) * cfg.head_size
    k, v = decoder.kcache, decoder.vcache
    shapes = (("ln1w", (L, C)), ("qkvw", (L, QR, C)), ("attprojw", (L, C, C)), ("ln2w", (L, C)), ("fc12w", (L, 2 * H, C)), ("fcprojw", (L, C, H)),
              ("lnfw", (C,)), ("lmhead", (cfg.padded_vocab_size, C)))
    return all(p[n].shape == s and p[n].is_contiguous() for n, s in shapes) and p["wte"].shape[1] == C and p["wte"].is_contiguous() \
        and k.dim() == 5 and k.shape == v.shape and k.shape[0] == L and k.shape[3:] == (cfg.num_kv_heads, cfg.head_size) \
        and k.is_contiguous() and v.is_contiguous()


def decoder_forward(decoder, bufs, dense, tokens, start_pos, pos, advance=False):
    """The launches of ``models.generate.CachedDecoder.forward`` for a bf16 model, from native code (csrc/decoder.cu).  ``bufs``: the decoder's activation
    buffers; ``dense``: (packed QKV, LSE) buffers for a prompt from position 0, or None.  Returns the fp32 logits (B, vocab_size) where the head's kernel writes
    them, after adding 1 to ``pos`` if ``advance`` asks for it, else None: bf16 logits are in ``bufs``."""
    m = decoder.model
    cfg, p, dev = m.cfg, m.params, m.device
    B, Tq = tokens.shape
    N, C, H, NH, NKV, HS = B * Tq, cfg.channels, cfg.hidden_dim, cfg.num_heads, cfg.num_kv_heads, cfg.head_size
    cache_len, heads = decoder.kcache.shape[2], NH + 2 * NKV
    logit_cols = p["lmhead"].shape[0]
    if N <= 128 and H % 64 == 0:
        mlp = 1
    else:
        # whole passes, us, with the activation in a launch of its own in brackets: four layers of 2048 channels, 129 rows 356 (359), 777 555 (559),
        # 2048 979 (1050), 8192 3431 (3717), 16000 9163 (9797); two of 4096 channels, 129 rows 346 (344), 16000 13691 (14265); four of 768, 777 rows 305 (304)
        mlp = 2 if N > 128 and H % 128 == 0 else 0
    lib = _lib.cuda()
    words = 0 if dense else lib.llmc_cached_attention_workspace(B, Tq, cache_len, NH, NKV, HS)
    ws = _scratch.get("cached_attention", words, torch.float32, dev) if words > 0 else None
    a = lambda t: None if t is None else t.data_ptr()
    # the streamed head writes the logits as they are returned; other heads (more than 128 rows) bf16
    how_head = forward_kernel(B, logit_cols, C, dev)
    logits32 = torch.empty(B, cfg.vocab_size, dtype=torch.float32, device=dev) if how_head == FORWARD_STREAM else None
    call = _lib.DecoderCall(
        **{n: p[n].data_ptr() for n in ("wte", "ln1w", "qkvw", "attprojw", "ln2w", "fc12w", "fcprojw", "lnfw", "lmhead")},
        **{n: bufs[n].data_ptr() for n in ("x", "ln", "raw", "q", "atty", "proj", "res", "fc12", "h", "last", "logits", "rstd")},
        freqs=m.freqs.data_ptr(), kcache=decoder.kcache.data_ptr(), vcache=decoder.vcache.data_ptr(), packed=a(dense and dense[0]), lse=a(dense and dense[1]),
        attention_ws=a(ws), tokens=tokens.data_ptr(), pos=a(pos),
        logits32=a(logits32), advance=a(pos) if advance and logits32 is not None else None,
        L=cfg.num_layers, C=C, H=H, NH=NH, NKV=NKV, HS=HS, vocab_rows=p["wte"].shape[0], logit_cols=logit_cols, vocab=cfg.vocab_size, freqs_len=m.freqs.shape[0],
        max_batch=decoder.kcache.shape[1], cache_len=cache_len, B=B, Tq=Tq, start=0 if pos is not None else start_pos,
        how_qkv=forward_kernel(N, heads * HS, C, dev), how_attproj=forward_kernel(N, C, C, dev), how_fc12=forward_kernel(N, 2 * H, C, dev),
        how_fcproj=forward_kernel(N, C, H, dev), how_head=how_head, mlp=mlp, eps=cfg.norm_eps)
    launches = ctypes.c_int(0)
    check(lib.llmc_decoder_forward(ctypes.byref(call), ctypes.byref(launches), _stream()), "llmc_decoder_forward")
    count_launches(launches.value)
    return logits32


def make_table(views):
    """views: list of dicts(p_base, p_stride, o_base, o_stride, n, L, wd, seed[, l_base])."""
    tab = TensorTable()
    assert len(views) <= 16
    for i, v in enumerate(views):
        t = tab.t[i]
        t.p_base, t.p_stride, t.o_base, t.o_stride = v["p_base"], v["p_stride"], v["o_base"], v["o_stride"]
        t.n, t.L, t.wd, t.seed = v["n"], v["L"], float(v.get("wd", 0.0)), int(v.get("seed", 0)) & 0xFFFFFFFF
        t.pad = int(v.get("l_base", 0))        # layer index of the view's first slice (enters the stochastic-rounding noise index)
    tab.count = len(views)
    return tab


def global_norm_sq(out, grads, views):
    """out[0] = sum of squares of the gradient elements described by ``views`` (deterministic)."""
    global _launches
    lib = _lib.cuda()
    part = _scratch.get("norm_sq", lib.llmc_norm_sq_scratch(), torch.float32, grads.device)
    tab = make_table(views)
    _launches += 2
    check(lib.llmc_global_norm_sq(_p(out), _p(part), _p(grads), ctypes.byref(tab), _stream()), "llmc_global_norm_sq")


def sum_scaled(out, terms, scale=1.0):
    """out[0] = scale * sum(terms) over fp32 device tensors, one block, fixed summation tree (the mean loss of a step)."""
    global _launches
    _launches += 1
    check(_lib.cuda().llmc_sum_f32(_p(out), _p(terms), terms.numel(), float(scale), _stream()), "llmc_sum_f32")


def adamw_update(params, master, grads, m, v, views, lr, beta1, beta2, eps, t, grad_scale=1.0, norm_sq=None, grad_clip=1.0):
    """AdamW on the views; bf16 params are stochastically rounded from the fp32 result."""
    global _launches
    tab = make_table(views)
    _launches += 1
    check(_lib.cuda().llmc_adamw(_p(params), _p(master), _p(grads), _p(m), _p(v), ctypes.byref(tab), lr, beta1, beta2, eps,
                                 int(t), grad_scale, _p(norm_sq), grad_clip, _stream()), "llmc_adamw")


def params_from_master(params, master, views):
    global _launches
    tab = make_table(views)
    _launches += 1
    check(_lib.cuda().llmc_params_from_master(_p(params), _p(master), ctypes.byref(tab), _stream()), "llmc_params_from_master")


def master_from_params(master, params, views):
    global _launches
    tab = make_table(views)
    _launches += 1
    check(_lib.cuda().llmc_master_from_params(_p(master), _p(params), ctypes.byref(tab), _stream()), "llmc_master_from_params")
