// Asynchronous copies into shared memory, and chained launches.
//
// Chained launches: a product's kernels follow one another on a stream with programmatic dependent
// launch, so that a kernel's blocks are placed, and its prologue runs, while the kernel before it
// finishes.
//
// Rules that keep this equal to plain stream order:
//  * every block of every kernel of the chain calls chain_wait(), in each thread that touches memory
//    that another kernel writes, or synchronises with one that called it, before it does. chain_wait()
//    returns once the kernel before has completed and its writes are visible; since that kernel waited
//    likewise, everything earlier on the stream has completed too;
//  * chain_release(), which lets the next kernel's blocks be placed, comes after chain_wait(), so at
//    most two kernels of a stream are resident, and two CTA-pair GEMMs never are: another kernel
//    stands between them;
//  * memory that an earlier kernel of the stream writes (operands, residues, CRT inputs) is not read
//    through a const __restrict__ pointer or __ldg: those promise data that is constant for the whole
//    kernel, and a kernel may start before that data is there. A plan's tables may be.
#pragma once
#include <cuda_runtime.h>

namespace negacyclic {

#ifdef __CUDACC__
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_enter() {
    chain_wait();
    chain_release();
}

__device__ __forceinline__ void cp_async_16(uint32_t smem, const void* global) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem), "l"(global) : "memory");
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

template <int kPending>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(kPending) : "memory");
}

template <class... Params, class... Args>
void launch_chained(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                    Args&&... args) {
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = grid;
    config.blockDim = block;
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    config.attrs = &attribute;
    config.numAttrs = 1;
    cudaLaunchKernelEx(&config, kernel, static_cast<Params>(args)...);  // errors: cudaGetLastError()
}
#endif

}  // namespace negacyclic
