// mg_reduce.cuh — fixed-order block reductions and the end of a V-cycle.
#pragma once

#include "mg_grid.cuh"

namespace mg {

// ------------------------------------------------------------ reductions
template <int NV>
static __device__ __forceinline__ void block_sum(double (&v)[NV])
{
    __shared__ double red[32][NV];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int k = 0; k < NV; ++k)
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
    __syncthreads();
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < NV; ++k) red[warp][k] = v[k];
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int k = 0; k < NV; ++k) {
            v[k] = lane < nw ? red[lane][k] : 0.0;
            for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], o);
        }
    }
    __syncthreads();
}

// Write this block's NV partial sums; returns true (in every thread) for the last
// block to arrive, which then sees every block's partials.
template <int NV>
static __device__ __forceinline__ bool publish_partials(double *partials, unsigned *counter, const double (&v)[NV],
                                                 int nblocks)
{
    __shared__ int is_last;
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < NV; ++k) partials[blockIdx.x * RED_STRIDE + k] = v[k];
        __threadfence();
        unsigned prev = atomicAdd(counter, 1u);
        is_last = (prev == (unsigned)nblocks - 1u);
    }
    __syncthreads();
    if (is_last) __threadfence();
    return is_last != 0;
}

template <int NV>
static __device__ __forceinline__ void gather_partials(const double *partials, int nblocks, double (&v)[NV])
{
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = 0.0;
    for (int b = threadIdx.x; b < nblocks; b += blockDim.x)
#pragma unroll
        for (int k = 0; k < NV; ++k) v[k] += __ldcg(&partials[b * RED_STRIDE + k]);
    block_sum<NV>(v);
}

// The reference's stop test (:247-248) on the cycle's mass error, or that it is not finite.
static __device__ __forceinline__ bool stops_on_error(const CaseDev &C, double err)
{
    return (C.stop_enabled != 0) & (!isfinite(err) | (err < C.convergence));
}

// History entry and that stop test when the fixed-point change is not tracked: one thread
// per case.
static __device__ __forceinline__ void end_of_cycle_err_only(const CaseDev &C, CaseState &ST)
{
    const double err = ST.last_err;
    const int k = ST.ncyc;
    if (k < C.hist_cap) {
        C.hist_err[k] = err;
        C.hist_delta[k] = 0.0;
    }
    ST.ncyc = k + 1;
    const bool finite = isfinite(err);
    if (!finite) ST.status |= CASE_NONFINITE;
    if (stops_on_error(C, err)) {
        ST.done = 1;
        if (finite) ST.status |= CASE_CONVERGED_REF;
    }
    ST.have_prev = 0;
}

// End of a V-cycle on the level-0 interior: relative change of u, v, sc and of p
// with its mean removed against the previous cycle, the history entry, the stop
// rule, and prev <- current.  p sums are shifted by the previous cycle's means so a
// uniform pressure drift does not cancel catastrophically.
// The fixed-point change (four norms over level 0 and their block reduction) is
// computed only while a solve with fp_tol > 0 runs; otherwise the cycle only records
// its mass error.
// `cell`: this thread has level-0 cell (i, j); nb blocks take part.  `stops`: stops_on_error
// of ST.last_err, read with the data the caller waits for anyway.
static __device__ __forceinline__ void end_of_cycle(const CaseDev &C, CaseState &ST, bool stops, bool cell, int i, int j,
                                                    int nb)
{
    if (!(C.fp_tol > 0.0)) {
        if (!stops) {
            if (blockIdx.x == 0 && threadIdx.x == 0) end_of_cycle_err_only(C, ST);
            return;
        }
        // Every block of this launch reads ST.done when it begins and does its part of the
        // cycle unless it is set, so only the last one to get here may set it.  (Other cycles
        // go without the counter.)
        __syncthreads();
        if (threadIdx.x != 0) return;
        __threadfence();
        if (atomicAdd(&C.counters[1], 1u) != (unsigned)nb - 1u) return;
        C.counters[1] = 0;
        end_of_cycle_err_only(C, ST);
        return;
    }
    const LevelDev &L = C.lv[0];
    const Dom d = dom_interior(L);
    const int n = d.wi * d.wj;
    const double kd = ST.shift_d, kp = ST.shift_p;
    double a[10];
#pragma unroll
    for (int k = 0; k < 10; ++k) a[k] = 0.0;
    if (cell) {
        const int q = j * L.npx + i;
        const int cur[3] = {S_U, S_V, S_SC}, prv[3] = {S_PREV_U, S_PREV_V, S_PREV_SC};
#pragma unroll
        for (int f = 0; f < 3; ++f) {
            double x = MGF(L, cur[f])[q], y = MGF(L, prv[f])[q], dd = x - y;
            a[2 * f] = dd * dd;
            a[2 * f + 1] = x * x;
            MGF(L, prv[f])[q] = x;
        }
        double x = MGF(L, S_P)[q], y = MGF(L, S_PREV_P)[q];
        double dd = (x - y) - kd, e = x - kp;
        a[6] = dd; a[7] = dd * dd; a[8] = e; a[9] = e * e;
        MGF(L, S_PREV_P)[q] = x;
    }
    block_sum<10>(a);
    if (!publish_partials<10>(C.partials, &C.counters[1], a, nb)) return;
    double s[10];
    gather_partials<10>(C.partials, nb, s);
    if (threadIdx.x != 0) return;
    C.counters[1] = 0;
    const double N = (double)n;
    double worst = 0.0;
    for (int f = 0; f < 4; ++f) {
        double num, den;
        if (f < 3) { num = s[2 * f]; den = s[2 * f + 1]; }
        else {
            num = s[7] - s[6] * s[6] / N;
            den = s[9] - s[8] * s[8] / N;
            if (num < 0.0) num = 0.0;
        }
        double r = num == 0.0 ? 0.0 : (den <= 0.0 ? (double)INFINITY : sqrt(num / den));
        if (r > worst || r != r) worst = r;
    }
    const double err = ST.last_err;
    const int k = ST.ncyc;
    const double delta = ST.have_prev ? worst : 0.0;
    if (k < C.hist_cap) {
        C.hist_err[k] = err;
        C.hist_delta[k] = delta;
    }
    ST.ncyc = k + 1;
    ST.shift_d = kd + s[6] / N;
    ST.shift_p = kp + s[8] / N;
    const bool finite = isfinite(err) && isfinite(delta);
    if (!finite) ST.status |= CASE_NONFINITE;
    if (C.stop_enabled) {
        if (!finite) ST.done = 1;
        else if (err < C.convergence) { ST.done = 1; ST.status |= CASE_CONVERGED_REF; }
        else if (C.fp_tol > 0.0 && ST.have_prev && delta < C.fp_tol) { ST.done = 1; ST.status |= CASE_CONVERGED_FP; }
    }
    ST.have_prev = 1;
}

}  // namespace mg
