// mg_fast.cuh — how the V-cycle's grid-wide kernels reach memory, and their tile bodies.
//
// A grid-wide launch of a V-cycle is short: on a small batch it lasts little longer than
// its chain of dependent memory accesses, and on a large one it is bound by how many loads
// are in flight (the one-thread-per-cell-and-equation kernels ran at 1.1 instructions a
// cycle and a quarter of the DRAM bandwidth, waiting on six dependent round trips each).
// So these kernels wait on memory once:
//   * before waiting for the previous launch (programmatic dependent launch) a thread
//     copies its level's description (FastLevel) into registers: sizes, spacings and the
//     base and stride of the level's arrays, which no kernel writes;
//   * an array's address is base + slot * stride (the slots of a level lie at one stride
//     in the pool), so no pointer is loaded between the description and the data;
//   * a thread loads all it needs, then computes, then stores;
//   * the case's stop flag is read along with the description, and a stopped case's blocks
//     end there (stopped_before, mg_grid.cuh); in a launch that may follow the one that sets
//     it, it is read along with the data and guards the stores;
//   * a block covers a tile of 32 x 8 cells and shares what its cells need of each other
//     (fluxes, face conductances, fields) through shared memory: one thread forms all
//     three equations of its cell from some 20 loads instead of three threads with some
//     20 each, and each conductance is divided once.
#pragma once

#include "mg_cells.cuh"

namespace mg {

struct FastLevel {
    int npx, npy;
    unsigned sb;              // bytes from one slot's array to the next
    char *b;                  // the level's first array
    double dx, dy, rdx, rdy;  // spacings and their reciprocals
    double amu, amusc;
    const unsigned *seq;
    const int *tag, *pcode, *pfan;
};

__device__ __forceinline__ FastLevel fast_level(const LevelDev &L)
{
    return {L.npx, L.npy, L.sb, reinterpret_cast<char *>(L.f[0]), L.dx, L.dy, L.rdx, L.rdy, L.amu, L.amusc,
            L.seq, L.tag, L.pcode, L.pfan};
}

// Begins the loads of a kernel's description here, ahead of a branch on the case's stop
// flag, which the compiler would otherwise have them wait for: a V-cycle of 64 256^2 cases
// 2.264 ms against 2.311 with the assembly without it, 2.285 with the update.  (In the
// residual, the prolongation and the pair smoother it costs registers or time and is left
// out: 2.264 to 2.254 for the residual, 2.269 to 2.262 for the prolongation.)
__device__ __forceinline__ void begin_loads(const CaseDev &C, const FastLevel &L)
{
    asm volatile("" ::"r"(L.npx), "r"(L.npy), "r"(L.sb), "l"(L.b), "r"(C.ngrid), "r"(C.tail));
}

// access type over a FastLevel
struct Fast {
    using T = double;
    const FastLevel &L;
    __device__ __forceinline__ double *at(int s) const
    {
        return reinterpret_cast<double *>(L.b + (unsigned long long)(unsigned)s * L.sb);
    }
    __device__ __forceinline__ double ld(int s, int q) const { return at(s)[q]; }
    __device__ __forceinline__ void st(int s, int q, double v) const { at(s)[q] = v; }
    __device__ __forceinline__ double g(int s, int q) const { return at(s)[q]; }
    __device__ __forceinline__ double amu() const { return L.amu; }
    __device__ __forceinline__ double amusc() const { return L.amusc; }
};

// a / b where a may be zero or tiny (inside obstacles, where the compiled division would
// leave its fast path): through the reciprocal of b
__device__ __forceinline__ double quotient(double a, double b) { return div_by(a, make_recip(b)); }

// The FP32 operands of an equation's smoother at cell q (mixed precision; mg_kernels.cu)
// from its FP64 coefficients and source and the field around q (centre, w, e, s, n).
struct Around { double c, w, e, s, n; };
__device__ __forceinline__ void store_ops32(const Fast &io, int e, int q, const Coef &k, double su, bool jac,
                                            const Around &x)
{
    const double ap = jac ? k.ap + 1.0e-30 : k.ap;
    const double nb = k.aw * x.w + k.ae * x.e + k.as * x.s + k.an * x.n;
    const double r = (nb + su) - ap * x.c;
    const double v[NCOEF] = {k.aw, k.ae, k.as, k.an, 1.0 / ap, r};
#pragma unroll
    for (int a = 0; a < NCOEF; ++a) reinterpret_cast<float *>(io.at(co_slot(e, a)))[q] = (float)v[a];
}

// ------------------------------------------------------------------- tiles
constexpr int TX = 32, TY = 8;            // cells of a tile, one thread each
constexpr int TW = TX + 3;                // row pitch of its shared arrays (one cell of halo
                                          // on either side, two at the far ones)
__host__ __device__ __forceinline__ int tiles_of(int wi, int wj) { return ((wi + TX - 1) / TX) * ((wj + TY - 1) / TY); }

// A cell's surroundings in the shared arrays: fluxes cx, cy (fluxes :678-694) and the
// quotients area / spacing at offsets (di, dj).
template <int H>
struct TileGeo {
    double cx[H][TW], cy[H][TW], qx[H][TW], qy[H][TW];
};

// coef_u, coef_v, coef_sc (mg_cells.cuh) from the shared arrays, cell at [y][x]; `wall`:
// the quotient of the opposite wall's face area the first row (column) adds.
template <class G>
__device__ __forceinline__ Coef tile_coef_u(const G &g, int y, int x, double amu, bool top, bool bottom, double wall)
{
    const double cxm = 0.5 * (g.cx[y][x] + g.cx[y][x - 1]);
    const double cxp = 0.5 * (g.cx[y][x] + g.cx[y][x + 1]);
    const double cym = 0.5 * (g.cy[y - 1][x] + g.cy[y - 1][x + 1]);
    const double cyp = 0.5 * (g.cy[y][x] + g.cy[y][x + 1]);
    const double dxm = amu * g.qx[y][x], dym = amu * g.qy[y][x];
    Coef k;
    k.aw = hyb_p(cxm, dxm);
    k.ae = hyb_m(cxp, dxm);
    k.as = hyb_p(cym, dym);
    k.an = hyb_m(cyp, dym);
    k.ap = k.aw + k.ae + k.as + k.an;
    if (top) {
        k.an = k.an + dym;
        k.ap = k.ap + dym;
    }
    if (bottom) {
        const double add = amu * wall;
        k.as = k.as + add;
        k.ap = k.ap + add;
    }
    return k;
}
template <class G>
__device__ __forceinline__ Coef tile_coef_v(const G &g, int y, int x, double amu, bool right, bool left, double wall)
{
    const double cxm = 0.5 * (g.cx[y][x - 1] + g.cx[y + 1][x - 1]);
    const double cxp = 0.5 * (g.cx[y][x] + g.cx[y + 1][x]);
    const double cym = 0.5 * (g.cy[y][x] + g.cy[y - 1][x]);
    const double cyp = 0.5 * (g.cy[y][x] + g.cy[y + 1][x]);
    const double dx_ = amu * g.qx[y][x], dy_ = amu * g.qy[y][x];
    Coef k;
    k.aw = hyb_p(cxm, dx_);
    k.ae = hyb_m(cxp, dx_);
    k.as = hyb_p(cym, dy_);
    k.an = hyb_m(cyp, dy_);
    k.ap = k.aw + k.ae + k.as + k.an;
    if (right) {
        k.ae = k.ae + dy_;
        k.ap = k.ap + dy_;
    }
    if (left) {
        const double add = amu * wall;
        k.aw = k.aw + add;
        k.ap = k.ap + add;
    }
    return k;
}
template <class G>
__device__ __forceinline__ Coef tile_coef_sc(const G &g, int y, int x, double amusc, unsigned code)
{
    const double dxm = amusc * g.qx[y][x - 1], dym = amusc * g.qy[y - 1][x];
    const double dxp = amusc * g.qx[y][x], dyp = amusc * g.qy[y][x];
    Coef k;
    k.aw = hyb_p(g.cx[y][x - 1], dxm);
    k.ae = hyb_m(g.cx[y][x], dxp);
    k.as = hyb_p(g.cy[y - 1][x], dym);
    k.an = hyb_m(g.cy[y][x], dyp);
    k.ap = k.aw + k.ae + k.as + k.an;
    const int cnt = (int)(code >> 28);
    for (int t = 0; t < cnt; ++t) {
        const int d = (int)((code >> (2 * t)) & 3u);
        double add;
        if (d == 0)      { add = amusc * g.qx[y][x + 1]; k.ae = k.ae + add; }
        else if (d == 1) { add = amusc * g.qx[y][x - 1]; k.aw = k.aw + add; }
        else if (d == 2) { add = amusc * g.qy[y + 1][x]; k.an = k.an + add; }
        else             { add = amusc * g.qy[y - 1][x]; k.as = k.as + add; }
        k.ap = k.ap + add;
    }
    return k;
}
template <class A>
__device__ __forceinline__ Around tile_around(const A &a, int y, int x)
{
    return {a[y][x], a[y][x - 1], a[y][x + 1], a[y - 1][x], a[y + 1][x]};
}
// sum a_nb x_nb - ap x (the residuals' first part, :1494-1512)
__device__ __forceinline__ double stencil(const Coef &k, const Around &x)
{
    return k.aw * x.w + k.ae * x.e + k.as * x.s + k.an * x.n - k.ap * x.c;
}

// The momentum sources from operands loaded beforehand (umom :741-767, vmom :769-793);
// `area` is the face's own area, ax and ay both (for the body force).  k.ap becomes the
// relaxed, solid diagonal.
__device__ __forceinline__ double mom_source(const CaseDev &C, const Recip &rm, Coef &k, double area, double dp,
                                             double x, double res, double body, double sp)
{
    double su = area * dp;
    const double ap = div_by(k.ap, rm);
    su = su + (1.0 - C.relxm) * ap * x + res + body;
    k.ap = ap + sp;
    return su;
}

// Halo entry `h` of a tile (the cells around the TX x TY tile, `far` more beyond its far
// sides): its column and row in the shared arrays, entries 0 .. tile_halo(far) - 1.
__host__ __device__ constexpr int tile_halo(int far) { return (TX + 1 + far) * (1 + far) + TY * (1 + far); }
template <int FAR>
__device__ __forceinline__ void halo_at(int h, int &x, int &y)
{
    constexpr int W = TX + 1 + FAR;
    if (h < W * (1 + FAR)) {
        const int r = h / W;
        x = h % W;
        y = r == 0 ? 0 : TY + r;
    } else {
        const int g = h - W * (1 + FAR), c = g / TY;
        x = c == 0 ? 0 : TX + c;
        y = 1 + g % TY;
    }
}

}  // namespace mg
