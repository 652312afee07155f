// mg_tangent.cu — the two ends of a forward-mode gradient, one block a direction: seeding
// and the objective's derivative.  Both were host loops over the directions (a strided copy
// a level and a wait; two whole fields read back): 60 us and 45 us a direction where the 66
// directions of a 64 x 64 grid now take a launch each.
#include "mg_kernels.cuh"
#include "mg_tangent.cuh"

namespace mg {

namespace {
constexpr int TBLOCK = 128;
}

// The seeded face's 1 on level 0, and on every coarser level the average of the two faces
// it covers (rest_geom, Version-6-26-04.c:1391-1473, as k_rest_geom).
__global__ void __launch_bounds__(TBLOCK) k_seed_tangent(const CaseDev *__restrict__ cs, const CaseTan *__restrict__ ts)
{
    const CaseDev &C = cs[blockIdx.x];
    const CaseTan &T = ts[blockIdx.x];
    if (T.face < 0) return;
    if (threadIdx.x == 0) T.lv[0].t[S_U][(T.face + 1) * C.lv[0].npx] = 1.0;
    for (int ig = 1; ig < C.ngrid; ++ig) {
        __syncthreads();
        const double *f = T.lv[ig - 1].t[S_U];
        double *k = T.lv[ig].t[S_U];
        const int nf = C.lv[ig - 1].npx, nk = C.lv[ig].npx;
        for (int j = 1 + threadIdx.x; j <= C.lv[ig].npy - 2; j += TBLOCK)
            k[j * nk] = 0.5 * (f[2 * j * nf] + f[(2 * j - 1) * nf]);
    }
}

// Row sums of one column each by three lanes, in row order (the host's objective_of).
__global__ void __launch_bounds__(TBLOCK)
    k_objective_tangent(const CaseDev *__restrict__ cs, CaseTan *ts)
{
    __shared__ double col[3][TBLOCK];
    const LevelDev &L = cs[blockIdx.x].lv[0];
    const double *p = ts[blockIdx.x].lv[0].t[S_P], *sc = ts[blockIdx.x].lv[0].t[S_SC];
    const int npx = L.npx, rows = L.npy - 2, t = threadIdx.x;
    double sum = 0.0;
    for (int j0 = 1; j0 <= rows; j0 += TBLOCK) {
        const int q = (j0 + t) * npx;
        if (j0 + t <= rows) {
            col[0][t] = p[q + 1];
            col[1][t] = p[q + npx - 2];
            col[2][t] = sc[q + npx - 1];
        }
        __syncthreads();
        if (t < 3)
            for (int k = 0; k < min(TBLOCK, rows - j0 + 1); ++k) sum += col[t][k];
        __syncthreads();
    }
    if (t < 3) col[t][0] = sum;
    __syncthreads();
    const double ny = (double)rows;
    if (t == 0) ts[blockIdx.x].dj = (col[0][0] / ny - col[1][0] / ny) + col[2][0] / ny;
}

cudaError_t launch_seed_tangent(const CaseDev *cs, const CaseTan *ts, int n, cudaStream_t s)
{
    k_seed_tangent<<<n, TBLOCK, 0, s>>>(cs, ts);
    return cudaGetLastError();
}

cudaError_t launch_objective_tangent(const CaseDev *cs, CaseTan *ts, int n, cudaStream_t s)
{
    k_objective_tangent<<<n, TBLOCK, 0, s>>>(cs, ts);
    return cudaGetLastError();
}

}  // namespace mg
