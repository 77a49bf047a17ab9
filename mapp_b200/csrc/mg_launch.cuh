// Launches with overlapping starts (programmatic dependent launch).
//
// The library's calls are chains of short kernels, and at small sizes the gaps
// between them (the next grid is set up only when the last block of the one
// before has drained) cost as much as the kernels.  c_d_calc and calc_g, sixteen
// kernels in all: 182 us with plain launches and 171 with overlapping starts at
// 2048 sites, 312 and 288 at 32000.  A kernel queued by launch_dep is set up
// while the one before it runs; its blocks wait in dep_sync, its first
// statement, until everything before it in the stream is complete and visible.
// (Two kernels split dep_sync: k_mlp_train reads its rows before the wait and
// k_mlp_adam lets the next step be set up before it waits; what makes that safe
// stands at each, and the first step of a run is not queued this way.)
// Behind a copy or an event it starts as any other launch does.
//
// Such a kernel is resident while the one before it still writes its inputs, so
// it reads what an earlier kernel of the chain writes with plain loads (or from
// L2, __ldcg): the read-only path (__ldg, ld.global.nc, and a kernel parameter
// that is const and __restrict__, which the compiler may turn into it) asks for
// data that does not change while the kernel lives, and is not ordered by the
// wait.  It is for the potential tables alone.
#pragma once

#include <cuda_runtime.h>

#include "mg_internal.h"

namespace mg {

// first statement of the kernels that launch_dep queues (a plain launch passes
// through it): waits for the work before this kernel, then lets the next
// kernel's blocks be set up
__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void dep_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void dep_sync()
{
    dep_wait();
    dep_start();
}

template <typename T>
struct same_type {
    using type = T;
};

template <typename... P>
inline cudaError_t launch_dep(void (*kern)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t st,
                              typename same_type<P>::type... args)
{
    cudaLaunchAttribute dep;
    dep.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    dep.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &dep;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, args...);
}

// For the precision and learned forms' persistent kernels: queued with an
// overlapping start only while the grid is at most one block per SM.  Most of
// them keep the potential tables or the network in shared memory, as many blocks
// an SM as that allows, and a full grid set up beside the blocks of a kernel that
// left most of the SM to the L1 does not find the shared memory for all its blocks
// and runs in two rounds: precision form, 256000 sites, k_dmd32_dens and
// k_dmd32_force queued early 780-810 us a call instead of 630.  Kernels that live
// off the L1 (the EAM, FS and plain DMD passes) are queued by launch_dep with full
// grids: 256000 atoms 351 us instead of 353-358, 256000 sites 1412 instead of
// 1423-1431.  The learned form's k_mlp_rows, k_mlp_densities and k_dmd32_pass2 stand
// between the two; queued early they make no difference (62500 sites 953-980 us, 957-962
// plainly; 500000 sites 6325-6374 and 6336-6348), so they go with their neighbours.
template <typename... P>
inline cudaError_t launch_full(void (*kern)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t st,
                                typename same_type<P>::type... args)
{
    if (grid <= (unsigned)num_sms()) return launch_dep(kern, grid, block, smem, st, args...);
    kern<<<grid, block, smem, st>>>(args...);
    return cudaGetLastError();
}

}  // namespace mg
