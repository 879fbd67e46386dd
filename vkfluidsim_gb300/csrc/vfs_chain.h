// Kernels of one stream, each the next one's input, launched so that a kernel's blocks are already
// resident when the one before it ends (programmatic dependent launch).
//
// A chained kernel begins with VFS_CHAINED(): it waits until the kernels before it have completed
// and their writes are visible, then lets its successor's blocks in as soon as all of its own have
// started. Every thread of every chained kernel does so before it touches memory, so a kernel waits,
// through its predecessor's wait, for the whole chain; what runs after the chain unchained (a copy,
// another kernel) waits for its last kernel as always. Only the launch latency and the ramp of the
// blocks overlap with the predecessor's tail. us per substep, launched plainly and chained: 1,000
// particles 31.6 / 30.8, 4,913 34.9 / 33.0, 46,656 54.2 / 50.8, 97,336 69.5 / 66.1, 262,144
// 103.2 / 99.9.
//
// VFS_CHAINED_LATE() lets no successor in early, for the kernels of a small model whose successor
// has about a block per SM: let in while the SMs are unevenly full, those blocks crowd a few SMs
// (17,576 particles: 51.8 us a substep instead of 41.1). Letting blocks in before the wait piles up
// several kernels and does the same (64,000 particles: 67.6).
//
// The branch keeps the loads of the kernel's body in a block of their own: loads of read-only data
// (__ldg) are free to move across the wait within a block. (%ntid.x is never 0.)
#pragma once

#include <cuda_runtime.h>

#include <utility>

#ifdef __CUDACC__
#define VFS_CHAINED_WAIT(after)                                                  \
    do {                                                                         \
        unsigned vfs_threads;                                                    \
        asm volatile("griddepcontrol.wait;\n\t" after "mov.u32 %0, %%ntid.x;"    \
                     : "=r"(vfs_threads)                                         \
                     :                                                           \
                     : "memory");                                                \
        if (vfs_threads == 0u) return;                                           \
    } while (0)
#define VFS_CHAINED() VFS_CHAINED_WAIT("griddepcontrol.launch_dependents;\n\t")
#define VFS_CHAINED_LATE() VFS_CHAINED_WAIT("")

namespace vfs {

// Lets the successor's blocks in (VFS_CHAINED_LATE() kernels that turn out to have nothing to do).
__device__ __forceinline__ void chained_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// kernel<<<grid, block, smem, s>>>(args...) for a kernel that begins with VFS_CHAINED().
template <class... P, class... A>
cudaError_t launch_chained(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t s,
                           A&&... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace vfs
#endif
