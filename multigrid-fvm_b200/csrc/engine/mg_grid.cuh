// mg_grid.cuh — index domains, programmatic launch and launch helpers shared by the
// engine's kernel files.
#pragma once

#include "mg_cells.cuh"

namespace mg {

struct Dom { int i0, j0, wi, wj; };

static __device__ __forceinline__ Dom dom_all(const LevelDev &L) { return {0, 0, L.npx, L.npy}; }
static __device__ __forceinline__ Dom dom_interior(const LevelDev &L) { return {1, 1, L.npx - 2, L.npy - 2}; }
static __device__ __forceinline__ Dom dom_flux(const LevelDev &L) { return {0, 0, L.npx - 1, L.npy - 1}; }
// sweep extent of each equation (solve_u/v/pprime/sc :701, :710, :725, :735)
static __device__ __forceinline__ Dom dom_eq(const LevelDev &L, int e)
{
    if (e == EQ_U) return {1, 1, L.npx - 3, L.npy - 2};
    if (e == EQ_V) return {1, 1, L.npx - 2, L.npy - 3};
    return dom_interior(L);
}

static __device__ __forceinline__ bool cell_at(const Dom &d, int t, int &i, int &j)
{
    if (d.wi <= 0 || d.wj <= 0 || t >= d.wi * d.wj) return false;
    j = d.j0 + t / d.wi;
    i = d.i0 + t % d.wi;
    return true;
}

static __device__ __forceinline__ int nth_eq(int mask, int k)
{
    for (int e = 0; e < 4; ++e)
        if ((mask >> e) & 1) {
            if (k == 0) return e;
            --k;
        }
    return -1;
}

// ---------------------------------------------- programmatic dependent launch
// The V-cycle's kernels are launched with programmatic stream serialization (when the
// schedule's `pdl` switch is on), so a kernel's CTAs may be scheduled while its
// predecessor is still running.  Two rules keep that in order:
//   * every thread waits (pdl_enter: until the launch before has completed and its writes
//     are visible; a no-op without the attribute) before the kernel's own dependent launch
//     is let begin, so all launches but the one directly before have completed by then;
//   * before that wait a kernel writes nothing, and reads only what the launch directly
//     before it does not write: its level's description and masks, case state that only
//     other launches set (stopped_before), and in the EARLY instantiations operands, where
//     the schedule says which launch comes before (after_smoother and the launches of one
//     smoothing, mg_context.cu).  A launch put in between, or a kernel that lets its
//     dependents begin before its own wait, breaks this silently.
static __device__ __forceinline__ void pdl_enter()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Whether a launch of this mode may leave a case out, read before it waits for the launch
// before it: `done` is set by the launch that ends a cycle, which is directly followed by
// the first launch of level 0 (that takes `gone`, or reads `done` after its wait) or by an
// op.  The blocks of a stopped case end there, before they load anything: a cycle of 64
// stopped 256^2 cases takes 0.28 ms against 1.52 where the flag was read along with the
// data, of two 52 us against 115 (a running one 2.25 ms and 227 us).
static __device__ __forceinline__ bool stopped_before(const CaseState &S, int mode)
{
    return (S.done != 0) & (mode > M_OP_C);
}

// Launch `k` on `st`, with programmatic stream serialization when `pdl` (the kernel
// may then be scheduled while its predecessor runs; it waits in pdl_enter()).
template <typename... KP, typename... A>
static cudaError_t launch_k(bool pdl, void (*k)(KP...), dim3 g, int b, int smem, cudaStream_t st, A... args)
{
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = g;
    c.blockDim = dim3((unsigned)b, 1, 1);
    c.dynamicSmemBytes = (size_t)smem;
    c.stream = st;
    c.attrs = at;
    c.numAttrs = pdl ? 1 : 0;
    return cudaLaunchKernelEx(&c, k, static_cast<KP>(args)...);
}

}  // namespace mg
