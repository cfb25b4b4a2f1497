// Shared helpers of the pq3d library: error recording, CUDA checks, the
// device-side bounded grid barrier and small math helpers.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include "pq3d.h"

namespace pq3d {

// Records `msg` as the calling host thread's last error and returns `code`.
int set_error(int code, const char *fmt, ...);
void clear_error();

#define PQ3D_CUDA_TRY(call)                                                              \
    do {                                                                                 \
        cudaError_t e_ = (call);                                                         \
        if (e_ != cudaSuccess)                                                           \
            return ::pq3d::set_error(PQ3D_ERR_CUDA, "%s:%d %s: %s", __FILE__, __LINE__,  \
                                     #call, cudaGetErrorString(e_));                      \
    } while (0)

#define PQ3D_REQUIRE(cond, ...)                                                          \
    do {                                                                                 \
        if (!(cond)) return ::pq3d::set_error(PQ3D_ERR_ARG, __VA_ARGS__);                \
    } while (0)

inline bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Dynamic shared memory beyond 48 KB for the next launch of `kernel`.  Set on every
// call (well below a microsecond) and not once per device: the attribute is one of
// the loaded code, and nothing in CUDA's documents says that it outlives a reset of
// the device between calls (with runtime 13.0 it does).
template <typename... P>
inline cudaError_t allow_smem(void (*kernel)(P...), size_t bytes)
{
    return cudaFuncSetAttribute((const void *)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

// Launch that may start before the stream's previous kernel has ended: when all
// that kernel's blocks have called chain_release or ended.  A kernel launched
// so calls chain_wait, which returns once the previous kernel is complete and its
// writes are visible: in every block that touches what that kernel writes, and in
// one at least, since the next kernel on the stream waits for this one only.
// Before it, a kernel may read only what no kernel since the last one known to be
// complete writes, and writes nothing.  Known to be complete, with its writes
// visible: everything before the previous kernel, where that one (the product,
// ahead of an attempt or a cluster step: both launched by one call) releases
// after its own chain_wait, or never.  So an attempt may read the state that the
// last update left while the product still runs; a product, whose previous kernel
// is the caller's (perhaps the writer of the operator), reads nothing early.  A
// small batched iteration is four kernels of 5-10 us, so launch latency and
// prologues are a visible part of it.
template <typename... P, typename... A>
inline cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args)
{
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
#ifdef __CUDACC__
__device__ __forceinline__ void chain_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
#endif

// Iteration cap of every device-side spin wait (each iteration sleeps ~1 us,
// so a wait gives up after roughly two seconds).
constexpr unsigned kSpinLimit = 1u << 21;

// Grid-wide barrier for a cooperative launch.  Every block calls it with the
// same sequence; `count` and `gen` live in device memory and start at 0.
// Returns false when the wait hit `limit` iterations (kSpinLimit unless a
// self-test lowers it; the caller then records PQ3D_ERR_TIMEOUT and leaves).
__device__ __forceinline__ bool grid_barrier(unsigned *count, unsigned *gen, unsigned nblocks,
                                             unsigned limit = kSpinLimit)
{
    __shared__ bool ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        ok = true;
        unsigned my_gen = *((volatile unsigned *)gen);
        __threadfence();
        unsigned arrived = atomicAdd(count, 1u) + 1u;
        if (arrived == nblocks) {
            *((volatile unsigned *)count) = 0u;
            __threadfence();
            atomicAdd(gen, 1u);
        } else {
            // short looks first (a barrier of resident blocks takes a few
            // microseconds), then ~1 us each up to the limit
            unsigned it = 0, looks = 0;
            while (*((volatile unsigned *)gen) == my_gen) {
                if (looks < 256) { ++looks; __nanosleep(32); continue; }
                if (++it > limit) { ok = false; break; }
                __nanosleep(1000);
            }
        }
        __threadfence();
    }
    __syncthreads();
    return ok;
}

}  // namespace pq3d
