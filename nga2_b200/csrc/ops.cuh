// ops.cuh -- arithmetic, launch and memory helpers shared by the solve-phase kernels.
#pragma once
#include "setup.cuh"

namespace bbmg {

// Programmatic dependent launch: every solve-phase kernel lets the next kernel
// in the stream start launching as soon as all of its own blocks are running,
// then waits for its predecessor to finish (and its writes to be visible)
// before touching memory.  Semantics stay those of plain stream order; only
// the launch latency overlaps the previous kernel's tail.
__device__ __forceinline__ void pdl_entry() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
// The two halves, for kernels that first read data no kernel of the solve
// writes (the operator planes, written only by the setup, which ends with a
// stream synchronisation): those loads may start before the wait, while the
// predecessor (or the one before it, still running its own tail) finishes.
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// L2 prefetch of the line holding p (a hint; L2 is coherent, so it is safe
// for any operand, also one the predecessor is still writing)
__device__ __forceinline__ void pf_l2(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

template <typename... KArgs, typename... Args>
static cudaError_t launch_k(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t shm, cudaStream_t s,
                            Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = shm;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, args...);
}

#define BB_CHECK_LAUNCH(call)                \
    do {                                     \
        cudaError_t e0_ = (call);            \
        if (e0_ != cudaSuccess) return e0_;  \
        cudaError_t e_ = cudaGetLastError(); \
        if (e_ != cudaSuccess) return e_;    \
    } while (0)

template <typename T, bool EXACT> struct Ops;
template <> struct Ops<double, true> {
    __device__ static __forceinline__ double mac(double s, double a, double b) { return __dadd_rn(s, __dmul_rn(a, b)); }
    __device__ static __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
    __device__ static __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
    __device__ static __forceinline__ double div(double a, double b) { return __ddiv_rn(a, b); }
};
template <typename T> struct Ops<T, false> {
    __device__ static __forceinline__ T mac(T s, T a, T b) { return fma(a, b, s); }
    __device__ static __forceinline__ T add(T a, T b) { return a + b; }
    __device__ static __forceinline__ T sub(T a, T b) { return a - b; }
    __device__ static __forceinline__ T div(T a, T b) { return a / b; }
};
template <typename T> struct ExactOf { static constexpr bool value = sizeof(T) == 8; };

}  // namespace bbmg
