// Launches that begin while the previous kernel of the stream ends (programmatic dependent launch). A kernel started
// this way runs its prologue at once and waits in await_previous() until the kernels before it have completed and
// their writes are visible; the kernel behind it may be set up from then on. Of a kernel boundary of a short step
// (five to six microseconds a kernel on a few thousand cells) the launch and the block start-up are then hidden.
#pragma once
#include <cuda_runtime.h>

#include "dg_status.cuh"

namespace fvedg {

// Every warp calls it before its first access to memory that an earlier kernel writes or reads. The result is 0 and not
// known to the compiler: added to an index, it keeps loads behind the wait. What earlier kernels wrote is loaded with
// ld_earlier(), plain loads or through L2, not through the read-only path, whose contents the wait need not renew.
__device__ __forceinline__ int await_previous() {
    int zero;
    asm volatile("griddepcontrol.wait;\n\tmov.b32 %0, 0;" : "=r"(zero)::"memory");
    return zero;
}

// The next kernel's blocks may come as soon as every block has got here (or is done). Where is measured, on steps: at
// the start, waiting blocks' shared memory took L1 from the running ones (mixed P4, 24,576 cells: 439 -> 493 us), and
// blocks of which an SM holds several gathered on the few SMs that had room (FP64 P2, 1,296 cells: 54 -> 94 us).
// So kernels with one block per SM call it as a warp begins its last item (FP64 P2, 7,986 cells: 74 -> 68 us), the
// others at a warp's end (FP64 P1, 3,072 cells: 35.7 -> 34.1 us).
__device__ __forceinline__ void release_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// A load of what an earlier kernel wrote and this one has not: free to move like one of constant memory, up to its
// index. Unconditional (a condition would become a branch): the caller picks an address that is valid.
__device__ __forceinline__ double ld_earlier(const double* p) {
    double v;
    asm("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}

// Opt a kernel into `smem` bytes of dynamic shared memory once per device.
template <class Kernel>
inline int ensure_smem(Kernel k, size_t smem, unsigned long long& done_mask) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return DG_E_CUDA;
    const unsigned long long bit = 1ull << (dev & 63);
    if (done_mask & bit) return DG_OK;
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return DG_E_CUDA;
    done_mask |= bit;
    return DG_OK;
}

// Only for kernels that call await_previous() in every warp.
template <class... P, class... A>
inline int launch_early(void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t s, const A&... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cuda_status(cudaLaunchKernelEx(&cfg, kernel, P(args)...));
}
template <bool EARLY, class... P, class... A>
inline int launch_as(void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t s, const A&... args) {
    if constexpr (EARLY) return launch_early(kernel, grid, block, smem, s, args...);
    kernel<<<grid, block, smem, s>>>(P(args)...);
    return cuda_status(cudaGetLastError());
}

}  // namespace fvedg
