// Kernel launch with its own status.
//
// A <<<>>> launch reports through cudaGetLastError, which also returns (and
// clears) an error left pending by an earlier, unrelated launch of the
// caller.  cudaLaunchKernel returns the status of this launch alone.
#pragma once
#include <cuda_runtime.h>

#include <tuple>
#include <type_traits>
#include <utility>

namespace gmpm {

template <typename... P, typename... A>
inline cudaError_t launch_kernel(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                 A&&... args) {
    static_assert(sizeof...(P) == sizeof...(A), "launch_kernel: argument count differs from the kernel's");
    std::tuple<std::decay_t<P>...> params(std::forward<A>(args)...);
    return std::apply(
        [&](auto&... p) {
            void* ptrs[] = {static_cast<void*>(&p)...};
            return cudaLaunchKernel(reinterpret_cast<const void*>(kernel), grid, block, ptrs, smem, stream);
        },
        params);
}

// Launch of a substep's kernel that may be set up while its predecessor in the
// stream still runs (programmatic dependent launch).  The kernel starts with
// depend_on_previous(), so it touches memory only after the predecessor has
// completed: the order of the work is that of plain launches, and only the
// launch latency overlaps.  A substep of a small scene is ten kernels of 3 to
// 40 us.
template <typename... P, typename... A>
inline cudaError_t launch_dependent(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                    A&&... args) {
    static_assert(sizeof...(P) == sizeof...(A), "launch_dependent: argument count differs from the kernel's");
    std::tuple<std::decay_t<P>...> params(std::forward<A>(args)...);
    return std::apply(
        [&](auto&... p) {
            void* ptrs[] = {static_cast<void*>(&p)...};
            cudaLaunchAttribute attr{};
            attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr.val.programmaticStreamSerializationAllowed = 1;
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = grid;
            cfg.blockDim = block;
            cfg.dynamicSmemBytes = smem;
            cfg.stream = stream;
            cfg.attrs = &attr;
            cfg.numAttrs = 1;
            return cudaLaunchKernelExC(&cfg, reinterpret_cast<const void*>(kernel), ptrs);
        },
        params);
}

// First statement of a kernel launched by launch_dependent (no effect in any
// other launch): its successor may be set up, and it waits for its predecessor.
// Before that the kernel is already resident while the kernels before it (a
// chain of them, if they are short) write its inputs, so its parameters are
// plain pointers: const with __restrict__ would promise the compiler data that
// is read-only for the kernel's whole life, and allow it loads that are neither
// coherent nor held back by the wait.  G2P alone promises it of the scene block,
// which only copies write (they and the kernels wait for each other) but for its
// time step (scene_dt): its loads of the materials come after stores that they
// would otherwise wait for (G2P 81 -> 88 us at 1M particles).
__device__ __forceinline__ void depend_on_previous() {
    asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
}

}  // namespace gmpm
