// chain.cuh -- launches that start while the kernel before them drains. The colour classes of an
// iteration follow one another on one stream; with an ordinary launch each waits for the last
// block of the class before it, then for its own launch and its first loads of the topology. A
// chained launch may start as soon as every block of the kernel before it has called
// chain_wait(); it reads what never changes (topology) and then waits itself. Every block
// of a chained kernel calls chain_wait() before its first access to anything an earlier kernel
// reads or writes, early returns included, so a kernel that has finished implies that all before it
// have. Measured per iteration, plain against chained: flat triangles 64^2 (seven classes of 600 vertices) 36.2 /
// 32.2 us, tets 10^3 1.108 / 1.035 ms for ten iterations, tets 48^3 0.4035 / 0.400 ms, icosphere level 7 0.3914 /
// 0.3910 ms. k_dmo_hex stays plain: 0.551 / 0.561 ms (its blocks hold the shared memory of the class before it).
#pragma once
#include <cuda_runtime.h>

namespace vsdmo {

// Waits until the kernels before this one have finished and their writes are visible; p comes back as a pointer
// that no load can be moved above the wait through (for the loads only: stores go through the parameter,
// which costs no registers while the kernel runs).
template <class T>
static __device__ __forceinline__ T* chain_wait(T* p) {
    asm volatile("griddepcontrol.wait;" : "+l"(p) : : "memory");
    asm volatile("griddepcontrol.launch_dependents;" : : : "memory");
    return p;
}

// chained: the operation before this one on the stream is a kernel that the launch may overlap
template <class... P, class... A>
static inline cudaError_t launch_chained(void (*kernel)(P...), unsigned blocks, unsigned threads, size_t smem, cudaStream_t s,
                                         bool chained, A... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = chained ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

}  // namespace vsdmo
