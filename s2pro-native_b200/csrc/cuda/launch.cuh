/* Kernels of a chain that start before the one in front of them has finished.
 *
 * A tick is several hundred short kernels in one stream, and each pays for its launch, its set-up and its predecessor's last
 * CTAs.  A kernel launched by launch_after may begin as soon as every CTA of its predecessor has begun (grid_release)
 * or ended, and calls grid_wait before it reads or writes anything that an earlier kernel of the stream reads or writes;
 * what comes before that call is index arithmetic, barrier set-up and the first loads of weights, which nothing in a stream writes.
 * grid_wait returns when the predecessor has completed and its writes are visible; as every kernel so launched calls it in
 * every CTA that does not leave at once, a completed predecessor implies the completion of all before it.
 * grid_release follows grid_wait, so that what comes before a kernel's grid_wait overlaps its predecessor alone and may rely on
 * everything older (positions, cached keys).  The exception are the short kernels in front of a wide linear: they release at
 * once, and the linear, which reads nothing but weights before it waits, fills its stages while the linear before last drains
 * (batch of 128: 13.43 -> 13.20 ms; the same everywhere costs the small batches 1 to 3 %).
 *
 * Measured, tick of the full model, before and now: batch of 3 5.88 -> 5.60 ms, 16 (INT8) 13.4 -> 12.9, 128 14.2 -> 13.2; request
 * start on a cached voice 10.4 -> 9.3 ms.
 *
 * A kernel in front that never calls grid_release, or one behind that is launched the ordinary way, behaves as usual. */
#pragma once
#include <cuda_runtime.h>

__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
/* A load through const __restrict__ (or __ldg) counts as constant over the whole kernel, and the kernel begins before the one in front of it has
 * ended: the compiler may move such a load in front of the wait, and take it from a cache that nobody keeps coherent.  So what an
 * earlier kernel may have written is read behind the wait, through a pointer that is not restricted; or through one that comes out of the wait, where what
 * it points at is settled in some calls and not in others: */
template <class P> __device__ __forceinline__ void grid_wait_for(P& a, P& b) { asm volatile("griddepcontrol.wait;" : "+l"(a), "+l"(b)::"memory"); }
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <class... P, class... A>
static inline cudaError_t launch_after(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchAttribute early = {};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = grid;
    c.blockDim = dim3(threads);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = &early;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}

/* For kernels that read before grid_wait what the kernel in front does not write inside a tick (weights, settled cache), but
 * what a caller of the public entry points may have written just before: early only inside a tick. */
template <class... P, class... A>
static inline cudaError_t launch_early(int early, void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, A... args) {
    if (early) return launch_after(kernel, grid, threads, smem, st, args...);
    kernel<<<grid, threads, smem, st>>>(static_cast<P>(args)...);
    return cudaGetLastError();
}
