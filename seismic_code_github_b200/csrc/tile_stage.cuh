// Staging of a tile's fields by TMA for kernels that load each tile once: one mbarrier, one phase, a
// bounded wait; and the launch of consecutive kernels as programmatic dependents.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "sfd_internal.h"

namespace sfd {
namespace tile {

__device__ __forceinline__ unsigned sptr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

// One thread announces the bytes and requests the boxes.  The z coordinate of a box is a multiple of
// four floats and no coordinate is negative (the slabs have ghost margins).
__device__ __forceinline__ void expect(uint64_t* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(sptr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void box(float* dst, const CUtensorMap* map, int z, int x, int shot, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];" ::"r"(sptr(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(z), "r"(x), "r"(shot), "r"(sptr(bar))
        : "memory");
}
__device__ __forceinline__ void bar_init(uint64_t* bar) {
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sptr(bar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
}
__device__ __forceinline__ bool bar_try(uint64_t* bar) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], 0;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(sptr(bar))
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool bar_wait_1s(uint64_t* bar) {
    bool done = bar_try(bar);
    if (!done) {
        uint64_t t0, t1;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
        do {
            done = bar_try(bar);
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
        } while (!done && t1 - t0 < 1000000000ull);
    }
    return done;
}
// every thread waits for the boxes; after a second without them it reports the timeout, gives the
// copies another second to land before the CTA's shared memory is released, and gives up
__device__ __forceinline__ bool staged(uint64_t* bar, int* err_flag) {
    if (bar_wait_1s(bar)) return true;
    atomicExch(err_flag, 1);
    bar_wait_1s(bar);
    return false;
}
// Programmatic dependent launch: release() lets the next kernel's CTAs start on what does not depend on
// this one (indexes, model values, tables), acquire() waits for the previous kernel before the first
// access to its fields.  What a kernel reads before acquire() must have been written before the chain of
// programmatic dependents began: by a kernel that a plain launch followed, or a copy that was waited for.
// The same goes for __ldg, whose data must not change while the kernel runs, and which the compiler may move
// above acquire(): model, tables and receiver lists only, never what a kernel of the chain writes.
__device__ __forceinline__ void release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void acquire() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// launch whose release() and acquire() make the edge to the kernel before it a programmatic one; chained =
// false: a plain launch, which starts when everything before it is done and visible
inline cudaError_t launch(const void* fn, dim3 grid, int threads, size_t smem, cudaStream_t st, void** args,
                          bool chained = true) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = chained && pdl_enabled() ? 1 : 0;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelExC(&cfg, fn, args);
}
template <class Args>
inline cudaError_t launch(const void* fn, dim3 grid, int threads, size_t smem, cudaStream_t st, const Args& a) {
    void* args[] = {const_cast<Args*>(&a)};
    return launch(fn, grid, threads, smem, st, args);
}
// Launch over columns of tiles (grid: 64-row tiles, tile columns, shots), in as many launches as grid.y,
// which holds 65535, asks for: the kernels write only their own cells of fields that no other of their CTAs
// reads.  a.col0 is the first tile column of the launch; *launches counts them.
template <class Args>
inline cudaError_t launch_columns(const void* fn, int ntz, int ncol, int active, int threads, size_t smem, cudaStream_t st,
                                  const Args& args, int* launches) {
    Args a = args;
    for (a.col0 = 0; a.col0 < ncol; a.col0 += 65535) {
        const int n = ncol - a.col0 < 65535 ? ncol - a.col0 : 65535;
        if (cudaError_t e = launch(fn, dim3(ntz, n, active), threads, smem, st, a)) return e;
        ++*launches;
    }
    return cudaSuccess;
}

}  // namespace tile
}  // namespace sfd
