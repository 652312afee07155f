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
    bool ring;  // dst takes the boundary ring too (it has it already where it is a caller's own field)
    bool vec;   // a block row's two cells may be loaded together (16-byte aligned)
};

// Tile (tx, ty) of tw x th cells with a halo of nu, and where in its region a thread's block
// lies: its first cell, and whether the region has it.
struct QTileAt {
    int x0, y0, x1, y1, cx0, cy0, rx1, ry1, i, j;
    bool mine;
};
__device__ __forceinline__ QTileAt tile_at(int dx1, int dy1, int tx, int ty, int tw, int th, int nu, int qx, int qy)
{
    QTileAt T;
    T.x0 = 1 + tx * tw;
    T.y0 = 1 + ty * th;
    T.x1 = min(T.x0 + tw - 1, dx1);
    T.y1 = min(T.y0 + th - 1, dy1);
    T.cx0 = max(T.x0 - nu, 0) & ~1;
    T.cy0 = max(T.y0 - nu, 0) & ~1;
    T.rx1 = min(T.x1 + nu, dx1 + 1);
    T.ry1 = min(T.y1 + nu, dy1 + 1);
    T.i = T.cx0 + BX * qx;
    T.j = T.cy0 + BY * qy;
    T.mine = qy < QY && T.i <= T.rx1 && T.j <= T.ry1;
    return T;
}

// A block's cells: cell (x, y) has k[y][x] of aw, ae, as, an, su, the diagonal b with its
// reciprocal rc, and the field v.
struct QBlock {
    double w[BY][BX], ea[BY][BX], so[BY][BX], no[BY][BX], su[BY][BX], b[BY][BX], rc[BY][BX], v[BY][BX];
};
__device__ __forceinline__ void clear_block(QBlock &B)
{
#pragma unroll
    for (int y = 0; y < BY; ++y)
#pragma unroll
        for (int x = 0; x < BX; ++x) {
            B.w[y][x] = B.ea[y][x] = B.so[y][x] = B.no[y][x] = B.v[y][x] = 0.0;
            B.su[y][x] = B.b[y][x] = 1.0;
        }
}
// The reciprocals, and the field into shared memory.  Cells outside the domain (the boundary
// ring, unused halo) are never updated; harmless operands keep their dead updates on the
// division's fast path.
__device__ __forceinline__ void prepare_block(QBlock &B, const QTileAt &T, int dx1, int dy1, double *phi, int qx, int qy)
{
#pragma unroll
    for (int y = 0; y < BY; ++y)
#pragma unroll
        for (int x = 0; x < BX; ++x) {
            const bool dom = T.mine && T.i + x >= 1 && T.i + x <= dx1 && T.j + y >= 1 && T.j + y <= dy1 &&
                             T.i + x <= T.rx1 && T.j + y <= T.ry1;
            if (!dom) B.b[y][x] = B.su[y][x] = 1.0;
            B.rc[y][x] = make_recip(B.b[y][x]).y;
        }
    if (qy < QY) {
#pragma unroll
        for (int y = 0; y < BY; ++y)
#pragma unroll
            for (int x = 0; x < BX; ++x) phi[sh(BY * qy + y, x, qx)] = B.v[y][x];
    }
}
// The units u0 .. u0 + nu - 1 (each between barriers; one precedes the first), then the tile,
// with `ring` plus the boundary ring where it touches it, to dst.
template <bool MEND>
__device__ __forceinline__ void smooth_block(QBlock &B, const QTileAt &T, int dx1, int dy1, int npx, double *phi, int qx,
                                             int qy, int u0, int nu, double *dst, bool ring)
{
    const int i = T.i, j = T.j, x0 = T.x0, x1 = T.x1, y0 = T.y0, y1 = T.y1;
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
                const double pw = x == 0 ? phi[sh(r, 1, qx - 1)] : B.v[y][0];
                const double pe = x == 1 ? phi[sh(r, 0, qx + 1)] : B.v[y][1];
                const double ps = y == 0 ? phi[sh(r - 1, x, qx)] : B.v[y - 1][x];
                const double pn = y == BY - 1 ? phi[sh(r + 1, x, qx)] : B.v[y + 1][x];
                const Recip R{B.b[y][x], B.rc[y][x]};
                a[y] = (B.w[y][x] * pw + B.ea[y][x] * pe + B.so[y][x] * ps + B.no[y][x] * pn) + B.su[y][x];
                z[y] = markstein(a[y], R);
                plain &= div_plain(a[y], R);
            }
            if (!plain) {
                bool rest = false;
#pragma unroll
                for (int y = 0; y < BY; ++y) {
                    const int x = (y + COL) & 1;
                    const Recip R{B.b[y][x], B.rc[y][x]};
                    if (div_plain(a[y], R)) continue;
                    if (!MEND) {
                        z[y] = div_by_rare(a[y], R.b, R.y);
                        continue;
                    }
                    // as div_by_rare, of the four cells without a call
                    const double q = markstein(a[y] * 0x1p600, R), c = q * 0x1p-600;
                    const bool zero = a[y] == 0.0;
                    z[y] = zero ? a[y] * R.y : c;
                    if ((__double2hiint(R.y) == 0) | (!zero & ((fabs(a[y]) >= 0x1p-918) | (fabs(fma(-c, 0x1p600, q)) == 0x1p-475))))
                        rest = true;
                }
                if (rest) {
#pragma unroll
                    for (int y = 0; y < BY; ++y) {
                        const int x = (y + COL) & 1;
                        z[y] = div_by(a[y], Recip{B.b[y][x], B.rc[y][x]});
                    }
                }
            }
#pragma unroll
            for (int y = 0; y < BY; ++y) {
                const int x = (y + COL) & 1;
                if (ax[x] && ay[y]) {
                    B.v[y][x] = z[y];
                    phi[sh(BY * qy + y, x, qx)] = z[y];
                }
            }
        };
        if (((u0 + h - 1) & 1) == 0) unit(std::integral_constant<int, 0>{});
        else unit(std::integral_constant<int, 1>{});
        __syncthreads();
    }
    const int ox0 = ring && x0 == 1 ? 0 : x0, ox1 = ring && x1 == dx1 ? x1 + 1 : x1;
    const int oy0 = ring && y0 == 1 ? 0 : y0, oy1 = ring && y1 == dy1 ? y1 + 1 : y1;
    if (T.mine) {
#pragma unroll
        for (int y = 0; y < BY; ++y)
#pragma unroll
            for (int x = 0; x < BX; ++x)
                if (i + x >= ox0 && i + x <= ox1 && j + y >= oy0 && j + y <= oy1) dst[(j + y) * npx + i + x] = B.v[y][x];
    }
}

// Tile (tx, ty) of a CTA that takes one.  `enter` waits for the launches before and says
// whether the case is still running.  EARLY: the coefficients are read before that.
template <bool EARLY, class Enter>
__device__ __forceinline__ void smooth_q_tile(const QIn &in, bool active, int tx, int ty, int tw, int th, int u0, int nu,
                                              Enter enter)
{
    __shared__ double smq[2 * QX * (SMOOTH_Q_ROWS + 2)];
    double *phi = smq + 2 * QX;   // a row of slack on either side
    const int npx = in.npx, t = threadIdx.x, qx = t % QX, qy = t / QX;
    const QTileAt T = tile_at(in.dx1, in.dy1, tx, ty, tw, th, nu, qx, qy);
    const int q0 = T.j * npx + T.i;
    QBlock B;
    clear_block(B);
    auto load = [&](const double *p, double (&a)[BY][BX]) {
#pragma unroll
        for (int y = 0; y < BY; ++y)
            if (active && T.mine && T.j + y <= T.ry1) {
                const double *g = p + q0 + y * npx;
                if (in.vec) {
                    const double2 d = *reinterpret_cast<const double2 *>(g);
                    a[y][0] = d.x;
                    a[y][1] = d.y;
                } else {
                    a[y][0] = g[0];
                    if (T.i + 1 < npx) a[y][1] = g[1];
                }
            }
    };
    auto coefs = [&]() {
        load(in.co[CK_AP], B.b);
        load(in.co[CK_AW], B.w);
        load(in.co[CK_AE], B.ea);
        load(in.co[CK_AS], B.so);
        load(in.co[CK_AN], B.no);
        load(in.co[CK_SU], B.su);
    };
    if (EARLY) coefs();
    const bool live = enter();
    if (!active) return;
    load(in.src, B.v);
    if (!EARLY) coefs();
    if (!live) return;
    prepare_block(B, T, in.dx1, in.dy1, phi, qx, qy);
    __syncthreads();
    smooth_block<false>(B, T, in.dx1, in.dy1, npx, phi, qx, qy, u0, nu, in.dst, in.ring);
}

__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

// Wait for the mbarrier's phase of parity `par` with at most `polls` polls; false on timeout.
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned par, int polls)
{
    for (int it = 0; it < polls; ++it) {
        unsigned done;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(done)
                     : "r"(bar), "r"(par)
                     : "memory");
        if (done) return true;
    }
    return false;
}
__device__ __forceinline__ void copy_box(void *to, const CUtensorMap *map, int x, int y, int slot, unsigned bar)
{
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(smem_addr(to)), "l"(map), "r"(x), "r"(y), "r"(slot), "r"(bar)
                 : "memory");
}

// where the field lies after the coefficients of a box (a copy lands on a 128-byte boundary)
__host__ __device__ constexpr int ahead_field(int box) { return (NCOEF * box + 15) & ~15; }

__device__ __forceinline__ void copy_async16(void *to, const void *from)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(to)), "l"(from) : "memory");
}

}  // namespace

// The tiles of a launch that has more of them than SMs, by a CTA an SM that takes every
// gridDim.x-th of the table `tab`.  While a tile is smoothed, one thread has the next one's
// coefficients and field copied (TMA) into shared memory, from where the threads fetch their
// blocks, and the table entry after that: only the first tile's way from memory is waited
// for.  Tiles of cases that have stopped are left out.  `maps` has each case's two tensor
// maps with a box of bw x bh cells (even bw: a box starts at an even column).  A copy that
// does not land within `polls` polls: CASE_WAIT_TIMEOUT, as k_smooth_tma.
// A tile takes 3.5 us and 0.37 a unit here, 4.9 and 0.37 with a CTA a tile (k_smooth_q),
// bound by the copies (25 MB a round of CTAs) and the fetch that waits for them.  Level 0 of
// 64 256^2 obstacle cases: five p' units 88 us against 111, four of u, v, sc 225 against 300;
// a V-cycle 2.36 ms against 2.60, of 8 cases 0.447 against 0.454.  (Copies by every thread,
// cp.async, were no faster than none ahead: issuing them holds up the units' accesses.  Tiles
// drawn from a counter: two ahead, so that the draw is not waited for, they balance no better.)
template <bool EARLY>
__global__ void __launch_bounds__(SMOOTH_Q_THREADS, 1)
    k_smooth_qs(const QTile *__restrict__ tab, int ntab, const SmoothMap *__restrict__ maps, CaseState *st,
                int u0, int nu, int dir, int tw, int th, int bw, int bh, int polls)
{
    extern __shared__ __align__(128) double ahead[];   // coefficients, then the field
    __shared__ double smq[2 * QX * (SMOOTH_Q_ROWS + 2)];
    constexpr int KEPT = SMOOTH_Q_THREADS - 32;   // flags
    __shared__ QTile entry[3];   // of the s-th tile this CTA takes, in s % 3
    __shared__ int there[3];     // there is one
    __shared__ int last;         // which of the CTA's share of the table was fetched last
    __shared__ unsigned running[KEPT / 32];   // bit k of these: the k-th of that share is of a case that has not stopped
    __shared__ __align__(8) unsigned long long mbar;
    double *phi = smq + 2 * QX;
    const int t = threadIdx.x, qx = t % QX, qy = t / QX, box = bw * bh, fbox = ahead_field(box);
    const unsigned bar = smem_addr(&mbar);
    // the s-th tile's entry, the share's k-th
    auto fetch = [&](int s, int k) {
        last = k;
        const int n = blockIdx.x + k * gridDim.x;
        there[s % 3] = n < ntab;
        if (n >= ntab) return;
        for (int c = 0; c < (int)sizeof(QTile) / 16; ++c)
            copy_async16(reinterpret_cast<char *>(&entry[s % 3]) + 16 * c, reinterpret_cast<const char *>(tab + n) + 16 * c);
    };
    // the first of the share's from the k-th on whose case runs
    auto next = [&](int k) {
        while (k < KEPT) {
            const unsigned w = running[k / 32] >> (k % 32);
            if (w) return k + __ffs(w) - 1;
            k = (k / 32 + 1) * 32;
        }
        return k;
    };
    auto first_cell = [&](int n0, int n) { return max(1 + n0 * n - nu, 0) & ~1; };
    auto coefs = [&](const QTile &N) {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                     ::"r"(bar), "r"((unsigned)((NCOEF + 1) * box * sizeof(double)))
                     : "memory");
        copy_box(ahead, &maps[N.icase].coef, first_cell(N.tx, tw), first_cell(N.ty, th), co_slot(N.e, CK_AW), bar);
    };
    auto field = [&](const QTile &N) {
        copy_box(ahead + fbox, &maps[N.icase].field, first_cell(N.tx, tw), first_cell(N.ty, th),
                 dir == 1 ? eq_tmp(N.e) : eq_field(N.e), bar);
    };
    if (t == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        entry[0] = tab[blockIdx.x];
        if (EARLY) coefs(entry[0]);
        fetch(1, 1);
    }
    // the first tile is on its way without a look at its case; of the rest, those of cases
    // that have stopped are left out (beyond the flags kept they are taken, and not smoothed)
    bool stopped = false;
    if (t >= 32) {
        const int n = blockIdx.x + (t - 32) * gridDim.x;
        stopped = n < ntab && st[tab[n].icase].done;
        const unsigned w = __ballot_sync(0xffffffffu, n < ntab && !stopped);
        if ((t & 31) == 0) running[t / 32 - 1] = w;
    }
    pdl_enter();
    if (t == 0) {
        if (!EARLY) coefs(entry[0]);
        field(entry[0]);
    }
    const bool some = __syncthreads_or(stopped);   // tiles may have to be left out
    if (some && t == 0 && next(1) != 1) {          // (not the one fetched beforehand)
        asm volatile("cp.async.wait_all;" ::: "memory");
        fetch(1, next(1));
    }
    for (int s = 0;; ++s) {
        const QTile now = entry[s % 3];
        const int dx1 = now.npx - (now.e == EQ_U ? 3 : 2), dy1 = now.npy - (now.e == EQ_V ? 3 : 2);
        const QTileAt T = tile_at(dx1, dy1, now.tx, now.ty, tw, th, nu, qx, qy);
        const bool live = !st[now.icase].done;
        QBlock B;
        clear_block(B);
        const bool landed = mbar_wait(bar, s & 1, polls);
        auto load = [&](int at, double (&a)[BY][BX]) {
#pragma unroll
            for (int y = 0; y < BY; ++y)
                if (T.mine && T.j + y <= T.ry1) {
                    const double2 d = *reinterpret_cast<const double2 *>(ahead + at + (BY * qy + y) * bw + BX * qx);
                    a[y][0] = d.x;
                    a[y][1] = d.y;
                }
        };
        load(CK_AP * box, B.b);
        load(CK_AW * box, B.w);
        load(CK_AE * box, B.ea);
        load(CK_AS * box, B.so);
        load(CK_AN * box, B.no);
        load(CK_SU * box, B.su);
        load(fbox, B.v);
        prepare_block(B, T, dx1, dy1, phi, qx, qy);
        if (t == 0) asm volatile("cp.async.wait_all;" ::: "memory");   // entry s + 1
        // one decision for the whole block; after it, `ahead` has been read
        if (!__syncthreads_and(landed)) {
            if (t == 0) atomicOr(&st[now.icase].status, (int)CASE_WAIT_TIMEOUT);
            mbar_wait(bar, s & 1, TMA_WAIT_POLLS);
            return;
        }
        const bool more = there[(s + 1) % 3];
        if (t == 0 && more) {
            coefs(entry[(s + 1) % 3]);
            field(entry[(s + 1) % 3]);
            fetch(s + 2, some ? next(last + 1) : s + 2);
        }
        if (live)
            smooth_block<true>(B, T, dx1, dy1, now.npx, phi, qx, qy, u0, nu,
                         reinterpret_cast<double *>(now.b + (unsigned long long)(unsigned)(dir == 0 ? eq_tmp(now.e) : eq_field(now.e)) * now.sb), true);
        else
            __syncthreads();   // (phi has been read before it is written again)
        if (!more) return;
    }
}

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
    in.ring = true;
    in.vec = (L.npx & 1) == 0;
#pragma unroll
    for (int k = 0; k < NCOEF; ++k) in.co[k] = io.at(co_slot(e, k));
    in.src = io.at(dir == 1 ? eq_tmp(e) : eq_field(e));
    in.dst = io.at(dir == 0 ? eq_tmp(e) : eq_field(e));
    const int txn = max(1, (in.dx1 + tw - 1) / tw), tyn = (in.dy1 + th - 1) / th;
    const bool stopped = stopped_before(st[blockIdx.y], mode);
    begin_loads(C, L);
    if (stopped) {
        pdl_enter();
        return;
    }
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

// Mixed precision: the same blocks, regions and units on the FP32 operands and corrections of
// k_smooth_f32 (mg_kernels.cu), with its `flags` and its bits; a division less, so no
// reciprocals, and half the registers: two CTAs an SM, one's loads under the other's units.
// A thread's eight cells take their operands in 28 paired loads where k_smooth_f32's pair a
// thread had 2048 cells an SM, most of them halo at ten units.  Bound by the operands' way
// from memory (4 us a round of CTAs).  Level 0 of 12 256^2 cases: u, v, sc and p' 95 us in four
// launches against 206 in three; a V-cycle 0.474 ms against 0.654, of one 1024^2 case 0.646.
template <bool EARLY>
__global__ void __launch_bounds__(SMOOTH_Q_THREADS, 2)
    k_smooth_q32(const CaseDev *__restrict__ cs, CaseState *st, int ig, int mode, int mask, int u0, int nu, int flags,
                 int tw, int th)
{
    __shared__ float smq[2 * QX * (SMOOTH_Q_ROWS + 2)];
    float *del = smq + 2 * QX;   // a row of slack on either side
    const CaseDev &C = cs[blockIdx.y];
    const FastLevel L = fast_level(C.lv[ig]);
    const Fast io{L};
    const int e = nth_eq(mask, blockIdx.z), npx = L.npx, t = threadIdx.x, qx = t % QX, qy = t / QX;
    const int dx1 = npx - (e == EQ_U ? 3 : 2), dy1 = L.npy - (e == EQ_V ? 3 : 2);
    const int txn = max(1, (dx1 + tw - 1) / tw), tx = blockIdx.x % txn, ty = blockIdx.x / txn;
    const bool stopped = stopped_before(st[blockIdx.y], mode);
    begin_loads(C, L);
    if (stopped) {
        pdl_enter();
        return;
    }
    const bool active = mode_active(C, ig, mode) && dx1 >= 1 && dy1 >= 1 && ty * th < dy1;
    const bool first = (flags & 1) != 0, last = (flags & 2) != 0;
    const QTileAt T = tile_at(dx1, dy1, tx, ty, tw, th, nu, qx, qy);
    const int i = T.i, j = T.j, q0 = j * npx + i;
    auto buf = [&](int b) { return reinterpret_cast<float *>(io.at(eq_tmp(e))) + (b ? (size_t)npx * L.npy : 0); };
    // cell (x, y) of the block: aw, ae, as, an, 1 / ap, r; v the correction
    float w[BY][BX], ea[BY][BX], so[BY][BX], no[BY][BX], ra[BY][BX], rs[BY][BX], v[BY][BX];
    auto load = [&](const float *p, float (&a)[BY][BX]) {
#pragma unroll
        for (int y = 0; y < BY; ++y) {
            a[y][0] = a[y][1] = 0.0f;
            if (active && T.mine && j + y <= T.ry1) {
                // (a level that has a coarser one has an even number of cells a row)
                const float2 d = *reinterpret_cast<const float2 *>(p + q0 + y * npx);
                a[y][0] = d.x;
                a[y][1] = d.y;
            }
        }
    };
    auto op = [&](int k) { return reinterpret_cast<const float *>(io.at(co_slot(e, k))); };
    auto operands = [&]() {
        load(op(CK_AW), w);
        load(op(CK_AE), ea);
        load(op(CK_AS), so);
        load(op(CK_AN), no);
        load(op(CK_AP), ra);
        load(op(CK_SU), rs);
    };
    if (EARLY) operands();
    pdl_enter();
    if (!active) return;
    const bool live = !st[blockIdx.y].done;
    if (!EARLY) operands();
    if (first) {
#pragma unroll
        for (int y = 0; y < BY; ++y) v[y][0] = v[y][1] = 0.0f;
    } else {
        load(buf((flags & 4) ? 1 : 0), v);
    }
    if (!live) return;
    if (qy < QY) {
#pragma unroll
        for (int y = 0; y < BY; ++y)
#pragma unroll
            for (int x = 0; x < BX; ++x) del[sh(BY * qy + y, x, qx)] = v[y][x];
    }
    __syncthreads();
    for (int h = 1; h <= nu; ++h) {
        const int g = nu - h;
        const int xl = max(1, T.x0 - g), xr = min(dx1, T.x1 + g), yl = max(1, T.y0 - g), yr = min(dy1, T.y1 + g);
        bool ax[BX], ay[BY];
#pragma unroll
        for (int x = 0; x < BX; ++x) ax[x] = i + x >= xl && i + x <= xr;
#pragma unroll
        for (int y = 0; y < BY; ++y) ay[y] = j + y >= yl && j + y <= yr;
        auto unit = [&](auto tag) {
            constexpr int COL = decltype(tag)::value;
            if (qy >= QY) return;
            float z[BY];
#pragma unroll
            for (int y = 0; y < BY; ++y) {
                const int x = (y + COL) & 1, r = BY * qy + y;
                const float pw = x == 0 ? del[sh(r, 1, qx - 1)] : v[y][0];
                const float pe = x == 1 ? del[sh(r, 0, qx + 1)] : v[y][1];
                const float ps = y == 0 ? del[sh(r - 1, x, qx)] : v[y - 1][x];
                const float pn = y == BY - 1 ? del[sh(r + 1, x, qx)] : v[y + 1][x];
                z[y] = (w[y][x] * pw + ea[y][x] * pe + so[y][x] * ps + no[y][x] * pn + rs[y][x]) * ra[y][x];
            }
#pragma unroll
            for (int y = 0; y < BY; ++y) {
                const int x = (y + COL) & 1;
                if (ax[x] && ay[y]) {
                    v[y][x] = z[y];
                    del[sh(BY * qy + y, x, qx)] = z[y];
                }
            }
        };
        if (((u0 + h - 1) & 1) == 0) unit(std::integral_constant<int, 0>{});
        else unit(std::integral_constant<int, 1>{});
        __syncthreads();
    }
    // the tile, and zero on the boundary ring where it touches it
    const int ox0 = T.x0 == 1 ? 0 : T.x0, ox1 = T.x1 == dx1 ? dx1 + 1 : T.x1;
    const int oy0 = T.y0 == 1 ? 0 : T.y0, oy1 = T.y1 == dy1 ? dy1 + 1 : T.y1;
    float *dst = buf((flags & 4) ? 0 : 1);
    double *phi = io.at(eq_field(e));
    const bool add = last && e != EQ_PP;
    if (T.mine) {
        auto out = [&](int x, int y) { return i + x >= ox0 && i + x <= ox1 && j + y >= oy0 && j + y <= oy1; };
        auto dom = [&](int x, int y) { return i + x >= 1 && i + x <= dx1 && j + y >= 1 && j + y <= dy1; };
        double f[BY][BX];   // (all read before the first is written: the loads stay together)
#pragma unroll
        for (int y = 0; y < BY; ++y)
#pragma unroll
            for (int x = 0; x < BX; ++x) f[y][x] = add && out(x, y) && dom(x, y) ? phi[q0 + y * npx + x] : 0.0;
#pragma unroll
        for (int y = 0; y < BY; ++y)
#pragma unroll
            for (int x = 0; x < BX; ++x)
                if (out(x, y)) {
                    const int q = q0 + y * npx + x;
                    dst[q] = dom(x, y) ? v[y][x] : 0.0f;
                    if (add && dom(x, y)) phi[q] = f[y][x] + (double)v[y][x];
                }
    }
}

cudaError_t launch_smooth_q32(const Launch &X, const CaseDev *dc, CaseState *ds, const Sched &S, cudaStream_t st)
{
    return launch_k(S.pdl, (X.a3 & 8) ? k_smooth_q32<true> : k_smooth_q32<false>, X.grid, SMOOTH_Q_THREADS, 0, st, dc, ds,
                    X.ig, X.mode, X.a0, X.a1, X.a2, X.a3 & 7, X.bw, X.bh);
}

cudaError_t configure_smooth_q()
{
    cudaError_t e = cudaSuccess;
    for (const void *k : {(const void *)k_smooth_qs<false>, (const void *)k_smooth_qs<true>})
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (ahead_field(SMOOTH_Q_COLS * SMOOTH_Q_ROWS) + SMOOTH_Q_COLS * SMOOTH_Q_ROWS) * (int)sizeof(double));
    return e;
}

cudaError_t launch_smooth_q(const Launch &X, const CaseDev *dc, CaseState *ds, const Sched &S, cudaStream_t st)
{
    if (X.a4) {
        const int bw = X.box >> 16, bh = X.box & 0xffff;
        if (!X.ptr || !X.tiles || bw > SMOOTH_Q_COLS || bh > SMOOTH_Q_ROWS) return cudaErrorInvalidValue;
        return launch_k(S.pdl, (X.a3 & 4) ? k_smooth_qs<true> : k_smooth_qs<false>, X.grid, SMOOTH_Q_THREADS,
                        (ahead_field(bw * bh) + bw * bh) * (int)sizeof(double), st, (const QTile *)X.tiles, X.a4,
                        (const SmoothMap *)X.ptr, ds, X.a1, X.a2, X.a3 & 3, X.bw, X.bh, bw, bh, S.tma_wait_polls);
    }
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
        in.ring = in.dst != phi;
        const cudaError_t e = c == 0 ? launch_k(false, r_smooth_q<false>, dim3(tiles), SMOOTH_Q_THREADS, 0, st, in, u0, nu, tw, th)
                                     : launch_k(true, r_smooth_q<true>, dim3(tiles), SMOOTH_Q_THREADS, 0, st, in, u0, nu, tw, th);
        if (e != cudaSuccess) return e;
        u0 += nu;
    }
    return cudaSuccess;
}

}  // namespace mg
