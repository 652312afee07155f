// mg_smooth.cu — the register-blocked red-black Gauss-Seidel tile smoother.
//
// The tiles, halos, units and windows of k_smooth (mg_kernels.cu: a tile plus a halo of one
// cell a unit, every unit on a window one cell narrower on each cut side), with a block of
// 2 x 4 cells in a thread's registers: field values, coefficients, sources and reciprocals.
// A unit updates the block's four cells of one colour from registers; only the neighbours
// outside the block come from shared memory (6 loads for 4 updates) and every new value is
// stored there once: 2.5 shared-memory accesses an update where k_smooth, a vertical pair a
// thread, makes 5.  A block's fixed register cost is shared by eight cells instead of two,
// so an SM holds 3024 cells (12 warps of 168 registers) where 1024 threads with a pair each
// hold 2048: a 54 x 56 region against 44 x 44, at ten units tiles of 33 x 35 against 24 x 24.
// The four quotients of a unit are formed without a branch between them, so their chains
// overlap; those outside markstein's range are mended behind one test.
//
// Bound by latency: a launch of one round of CTAs takes 4.6 us for the load phase, the
// reciprocals and the write-back, and 0.43 us a unit (12 warps wait on a chain of ten FP64
// operations, three shared-memory accesses and a barrier).  Ten p' units on level 0 of 64
// 256^2 obstacle cases: 231 us against 355 (k_smooth); five units: 105 against 164; two
// cases: 9.5 against 14.4.
//
// Regions start at an even column and row, so the colour of every cell of a block is known
// at compile time, and a block row's two cells are one aligned 16-byte load where the
// level's row length is even.  Shared rows keep their even columns, then their odd ones:
// the lanes of a warp, two columns apart, read consecutive doubles.  (Jacobi, which updates
// all eight cells from old values, needs more registers than there are and was slower than
// k_smooth.)
#include "mg_fast.cuh"
#include "mg_grid.cuh"
#include "mg_kernels.cuh"

#include <type_traits>

namespace mg {

namespace {

constexpr int BX = 2, BY = 4;                                       // cells of a thread's block
constexpr int QX = SMOOTH_Q_COLS / BX, QY = SMOOTH_Q_ROWS / BY;     // blocks of a region
static_assert(QX * QY <= SMOOTH_Q_THREADS, "a thread a block");

// shared-memory index of column 2 k + half of row r
__device__ __forceinline__ int sh(int r, int half, int k) { return (r * 2 + half) * QX + k; }

// One equation on one level: coefficients, where the field comes from and goes to (the same
// array only where one tile covers the domain), row length and the domain [1, dx1] x [1, dy1].
struct QIn {
    const double *co[NCOEF], *src;
    double *dst;
    int npx, dx1, dy1;
    bool vec;   // a block row's two cells may be loaded together (16-byte aligned)
};

// Tile (tx, ty) of tw x th cells.  `enter` waits for the launches before and says whether
// the case is still running.  EARLY: the coefficients are read before that.
template <bool EARLY, class Enter>
__device__ __forceinline__ void smooth_q_tile(const QIn &in, bool active, int tx, int ty, int tw, int th, int u0, int nu,
                                              Enter enter)
{
    __shared__ double smq[2 * QX * (SMOOTH_Q_ROWS + 2)];
    double *phi = smq + 2 * QX;   // a row of slack on either side
    const int npx = in.npx, dx1 = in.dx1, dy1 = in.dy1, t = threadIdx.x;
    const int x0 = 1 + tx * tw, y0 = 1 + ty * th;
    const int x1 = min(x0 + tw - 1, dx1), y1 = min(y0 + th - 1, dy1);
    const int cx0 = max(x0 - nu, 0) & ~1, cy0 = max(y0 - nu, 0) & ~1;
    const int rx1 = min(x1 + nu, dx1 + 1), ry1 = min(y1 + nu, dy1 + 1);
    const int qx = t % QX, qy = t / QX, i = cx0 + BX * qx, j = cy0 + BY * qy;
    const bool mine = active && qy < QY && i <= rx1 && j <= ry1;
    const int q0 = j * npx + i;
    const bool vec = in.vec;

    // cell (x, y) of the block: k[y][x] = aw .. an, su, b, y; v = field
    double w[BY][BX], ea[BY][BX], so[BY][BX], no[BY][BX], su[BY][BX], b[BY][BX], rc[BY][BX], v[BY][BX];
#pragma unroll
    for (int y = 0; y < BY; ++y)
#pragma unroll
        for (int x = 0; x < BX; ++x) {
            w[y][x] = ea[y][x] = so[y][x] = no[y][x] = v[y][x] = 0.0;
            su[y][x] = b[y][x] = 1.0;
        }
    auto load = [&](const double *p, double (&a)[BY][BX]) {
#pragma unroll
        for (int y = 0; y < BY; ++y)
            if (mine && j + y <= ry1) {
                const double *g = p + q0 + y * npx;
                if (vec) {
                    const double2 d = *reinterpret_cast<const double2 *>(g);
                    a[y][0] = d.x;
                    a[y][1] = d.y;
                } else {
                    a[y][0] = g[0];
                    if (i + 1 < npx) a[y][1] = g[1];
                }
            }
    };
    auto coefs = [&]() {
        load(in.co[CK_AP], b);
        load(in.co[CK_AW], w);
        load(in.co[CK_AE], ea);
        load(in.co[CK_AS], so);
        load(in.co[CK_AN], no);
        load(in.co[CK_SU], su);
    };
    if (EARLY) coefs();
    const bool live = enter();
    if (!active) return;
    load(in.src, v);
    if (!EARLY) coefs();
    if (!live) return;
    // cells outside the domain (the boundary ring, unused halo) are never updated; harmless
    // operands keep their dead updates on the division's fast path
#pragma unroll
    for (int y = 0; y < BY; ++y)
#pragma unroll
        for (int x = 0; x < BX; ++x) {
            const bool dom = mine && i + x >= 1 && i + x <= dx1 && j + y >= 1 && j + y <= dy1 && i + x <= rx1 && j + y <= ry1;
            if (!dom) b[y][x] = su[y][x] = 1.0;
            rc[y][x] = make_recip(b[y][x]).y;
        }
    if (qy < QY) {
#pragma unroll
        for (int y = 0; y < BY; ++y)
#pragma unroll
            for (int x = 0; x < BX; ++x) phi[sh(BY * qy + y, x, qx)] = v[y][x];
    }
    __syncthreads();
    for (int h = 1; h <= nu; ++h) {
        const int g = nu - h;
        const int xl = max(1, x0 - g), xr = min(dx1, x1 + g), yl = max(1, y0 - g), yr = min(dy1, y1 + g);
        bool ax[BX], ay[BY];
#pragma unroll
        for (int x = 0; x < BX; ++x) ax[x] = i + x >= xl && i + x <= xr;
#pragma unroll
        for (int y = 0; y < BY; ++y) ay[y] = j + y >= yl && j + y <= yr;
        // the block's cells of colour COL (0 red, 1 black): (x + y) & 1 == COL
        auto unit = [&](auto tag) {
            constexpr int COL = decltype(tag)::value;
            if (qy >= QY) return;
            double a[BY], z[BY];
            bool plain = true;
#pragma unroll
            for (int y = 0; y < BY; ++y) {
                const int x = (y + COL) & 1, r = BY * qy + y;
                const double pw = x == 0 ? phi[sh(r, 1, qx - 1)] : v[y][0];
                const double pe = x == 1 ? phi[sh(r, 0, qx + 1)] : v[y][1];
                const double ps = y == 0 ? phi[sh(r - 1, x, qx)] : v[y - 1][x];
                const double pn = y == BY - 1 ? phi[sh(r + 1, x, qx)] : v[y + 1][x];
                const Recip R{b[y][x], rc[y][x]};
                a[y] = (w[y][x] * pw + ea[y][x] * pe + so[y][x] * ps + no[y][x] * pn) + su[y][x];
                z[y] = markstein(a[y], R);
                plain &= div_plain(a[y], R);
            }
            if (!plain) {
#pragma unroll
                for (int y = 0; y < BY; ++y) {
                    const int x = (y + COL) & 1;
                    if (!div_plain(a[y], Recip{b[y][x], rc[y][x]})) z[y] = div_by_rare(a[y], b[y][x], rc[y][x]);
                }
            }
#pragma unroll
            for (int y = 0; y < BY; ++y) {
                const int x = (y + COL) & 1;
                if (ax[x] && ay[y]) {
                    v[y][x] = z[y];
                    phi[sh(BY * qy + y, x, qx)] = z[y];
                }
            }
        };
        if (((u0 + h - 1) & 1) == 0) unit(std::integral_constant<int, 0>{});
        else unit(std::integral_constant<int, 1>{});
        __syncthreads();
    }
    // the tile, plus the boundary ring where it touches it
    const int ox0 = x0 == 1 ? 0 : x0, ox1 = x1 == dx1 ? x1 + 1 : x1;
    const int oy0 = y0 == 1 ? 0 : y0, oy1 = y1 == dy1 ? y1 + 1 : y1;
    if (mine) {
#pragma unroll
        for (int y = 0; y < BY; ++y)
#pragma unroll
            for (int x = 0; x < BX; ++x)
                if (i + x >= ox0 && i + x <= ox1 && j + y >= oy0 && j + y <= oy1) in.dst[q0 + y * npx + x] = v[y][x];
    }
}

}  // namespace

// blockIdx.x: tile, .y: case, .z: equation of `mask`; `dir` 0: from the field to the
// equation's ping-pong buffer, 1: the reverse.  EARLY: a later launch of the smoothing.
template <bool EARLY>
__global__ void __launch_bounds__(SMOOTH_Q_THREADS, 1)
    k_smooth_q(const CaseDev *__restrict__ cs, CaseState *st, int ig, int mode, int mask, int u0, int nu, int dir,
               int tw, int th)
{
    const CaseDev &C = cs[blockIdx.y];
    const FastLevel L = fast_level(C.lv[ig]);
    const Fast io{L};
    const int e = nth_eq(mask, blockIdx.z);
    QIn in;
    in.npx = L.npx;
    in.dx1 = L.npx - (e == EQ_U ? 3 : 2);
    in.dy1 = L.npy - (e == EQ_V ? 3 : 2);
    in.vec = (L.npx & 1) == 0;
#pragma unroll
    for (int k = 0; k < NCOEF; ++k) in.co[k] = io.at(co_slot(e, k));
    in.src = io.at(dir == 1 ? eq_tmp(e) : eq_field(e));
    in.dst = io.at(dir == 0 ? eq_tmp(e) : eq_field(e));
    const int txn = max(1, (in.dx1 + tw - 1) / tw), tyn = (in.dy1 + th - 1) / th;
    const bool active = mode_active(C, ig, mode) && in.dx1 >= 1 && in.dy1 >= 1 && (int)blockIdx.x < txn * tyn;
    smooth_q_tile<EARLY>(in, active, blockIdx.x % txn, blockIdx.x / txn, tw, th, u0, nu, [&]() {
        pdl_enter();
        return !active || !st[blockIdx.y].done;
    });
}

// The same on a caller's own level.
template <bool EARLY>
__global__ void __launch_bounds__(SMOOTH_Q_THREADS, 1) r_smooth_q(QIn in, int u0, int nu, int tw, int th)
{
    const int txn = (in.dx1 + tw - 1) / tw;
    smooth_q_tile<EARLY>(in, true, blockIdx.x % txn, blockIdx.x / txn, tw, th, u0, nu, [&]() {
        pdl_enter();
        return true;
    });
}

cudaError_t launch_smooth_q(const Launch &X, const CaseDev *dc, CaseState *ds, const Sched &S, cudaStream_t st)
{
    if (X.a3 & 4)
        return launch_k(S.pdl, k_smooth_q<true>, X.grid, SMOOTH_Q_THREADS, 0, st, dc, ds, X.ig, X.mode, X.a0, X.a1, X.a2,
                        X.a3 & 3, X.bw, X.bh);
    return launch_k(S.pdl, k_smooth_q<false>, X.grid, SMOOTH_Q_THREADS, 0, st, dc, ds, X.ig, X.mode, X.a0, X.a1, X.a2,
                    X.a3 & 3, X.bw, X.bh);
}

// The plan of `units` half-sweeps over a domain of wi x wj cells of one equation on a
// caller's level, whose first and last launch read and write phi: one launch in place where
// a region holds the whole level, else an even number through a buffer of the level's size.
// Times in microseconds, as the schedule's for the engine's levels.
double raw_q_plan(int wi, int wj, int units, int &chunks, int &tw, int &th)
{
    if (wi + 2 <= SMOOTH_Q_COLS && wj + 2 <= SMOOTH_Q_ROWS) {
        chunks = 1;
        tw = wi;
        th = wj;
        return 4.6 + 0.43 * units;
    }
    double best = 1e300;
    auto side = [](int n, int most) { return (n + (n + most - 1) / most - 1) / ((n + most - 1) / most); };
    for (int c = 2; c <= units; c += 2) {
        const int u = (units + c - 1) / c, mx = SMOOTH_Q_COLS - 2 * u - 1, my = SMOOTH_Q_ROWS - 2 * u - 1;
        if (mx < 8 || my < 8) continue;
        const int w = side(wi, mx), h = side(wj, my);
        const long long tiles = (long long)((wi + w - 1) / w) * ((wj + h - 1) / h);
        const double t = c * (0.3 + (double)((tiles + 147) / 148) * (4.9 + 0.37 * u));
        if (t < best) {
            best = t;
            chunks = c;
            tw = w;
            th = h;
        }
    }
    return best;
}

cudaError_t raw_smooth_q(const double *const *co, double *phi, double *tmp, int npx, int wi, int wj, int units, int chunks,
                         int tw, int th, cudaStream_t st)
{
    QIn in;
    for (int k = 0; k < NCOEF; ++k) in.co[k] = co[k];
    in.npx = npx;
    in.dx1 = wi;
    in.dy1 = wj;
    in.vec = (npx & 1) == 0 && (((uintptr_t)phi | (uintptr_t)tmp) & 15) == 0;
    for (int k = 0; k < NCOEF; ++k) in.vec = in.vec && ((uintptr_t)co[k] & 15) == 0;
    const unsigned tiles = (unsigned)(((wi + tw - 1) / tw) * ((wj + th - 1) / th));
    int u0 = 0;
    for (int c = 0; c < chunks; ++c) {
        const int nu = units / chunks + (c < units % chunks ? 1 : 0);
        in.src = (c & 1) ? tmp : phi;
        in.dst = (c & 1) || chunks == 1 ? phi : tmp;
        const cudaError_t e = c == 0 ? launch_k(false, r_smooth_q<false>, dim3(tiles), SMOOTH_Q_THREADS, 0, st, in, u0, nu, tw, th)
                                     : launch_k(true, r_smooth_q<true>, dim3(tiles), SMOOTH_Q_THREADS, 0, st, in, u0, nu, tw, th);
        if (e != cudaSuccess) return e;
        u0 += nu;
    }
    return cudaSuccess;
}

}  // namespace mg
