// Programmatic dependent launch: a kernel launched through launch_pdl may start while the kernel before it in its stream is still
// running, as soon as every CTA of that one has called pdl_trigger() or exited.  Such a kernel calls pdl_wait() before it touches
// anything another kernel may have written or may still read; pdl_wait() returns when the preceding kernel has completed and its
// writes are visible.  A kernel calls pdl_trigger() only after its own pdl_wait(), so "the preceding kernel has completed" covers all
// kernels before it too.  Behind a kernel that never triggers (or a copy) the launch is an ordinary one.  Works the same inside a
// captured graph.  The kernels of the GPT-2 and LLaMA paths are launched this way: their setup (barriers, tensor memory, tensor maps) and the
// launch itself run under the tail of the kernel before.  The same kernels launched without the attribute in brackets: forward + backward of 4 x 64
// tokens of GPT-2 124M 2.39 ms (2.58), a decoding step of 4 rows 280 us (312), a prefill of 777 tokens 740 us (819), residual + LayerNorm forward
// and backward at 65536 x 768 153 us (157).  The classifier, the attention kernels of wide heads and those of
// 64-wide heads with a block on every SM (the forward: two) are launched plainly and trigger nothing: attention at 64 x 1024 x 12 x 64 forward and backward took
// 986 us with the attribute and 938 without, on one GPU in turn, with the trigger right behind the wait (at the end of a CTA, where gemm2_kernel has
// its own, it was not tried there); the classifier's figures stand with it.  Where 64-wide heads leave SMs free
// the attribute pays: forward + backward of 4 x 64 tokens 1566 us without and 1513 with it.  (The bracketed comparisons were made when the plain launch
// was the only other thing that differed; those passes take 1284, 260 and 628 us now, 3 % more or less from one GPU to another.)
#pragma once
#include "common.cuh"

DEVINL void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
DEVINL void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... P, typename... A>
cudaError_t launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, int cluster_x, A... args) {
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster_x; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream;
    cfg.attrs = attr; cfg.numAttrs = cluster_x > 0 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}
