// mg_tile.cu — the tile kernels of a V-cycle: assembly, restriction, prolongation (see
// mg_fast.cuh for how they reach memory).  blockIdx.x is a tile of the case's level,
// blockIdx.y the case; a thread forms every equation of its cell.
#include "mg_grid.cuh"
#include "mg_fast.cuh"
#include "mg_kernels.cuh"
#include "mg_reduce.cuh"

namespace mg {

namespace {

constexpr int NT = TX * TY;

// Fluxes and conductance quotients of one cell into the shared arrays.
template <class G>
__device__ __forceinline__ void put_geo(G &g, int y, int x, const FastLevel &L, double u, double v, double ax,
                                        double ay, double &cx, double &cy)
{
    cx = 0.5 * u * ax;
    cy = 0.5 * v * ay;
    g.cx[y][x] = cx;
    g.cy[y][x] = cy;
    g.qx[y][x] = div_by(ax, Recip{L.dx, L.rdx});
    g.qy[y][x] = div_by(ay, Recip{L.dy, L.rdy});
}

}  // namespace

// The assembly of a level visit (REST false): fluxes, coefu + umom, coefv + vmom, coefsc +
// scalar, the scalar outflow ghost (AsmBits `what`, all four parts).  REST true, on the
// coarse level ig + 1 of a restriction: coarse fluxes, the FAS defects from the sums of fine
// residuals k_tile_restv left in the level's ping-pong buffers and, with `what`, the coarse
// level's first assembly: a cell's coefficients serve both its residual and its assembly.
// F32: mixed precision, FP32 smoother operands instead of the FP64 coefficient sets.
// Bound by memory latency, then bandwidth.  Level 0 of 64 256^2 cases (34 FP64 words a cell,
// 176 us at the measured copy rate): 269 us, against 446 us with a thread per cell and
// equation (k_asm), which loads the same neighbourhood three times and divides for every
// use of a conductance; the restriction's coarse side 88 us against 208 (k_restrict).
template <bool REST, bool F32>
__global__ void __launch_bounds__(NT, 3)
    k_tile_asm(const CaseDev *__restrict__ cs, CaseState *st, int ig, int mode, unsigned what)
{
    constexpr bool FIELDS = REST || F32;
    __shared__ TileGeo<TY + 2> g;
    __shared__ double fu[FIELDS ? TY + 2 : 1][TW], fv[FIELDS ? TY + 2 : 1][TW], fs[FIELDS ? TY + 2 : 1][TW];
    const CaseDev &C = cs[blockIdx.y];
    const FastLevel L = fast_level(C.lv[REST ? ig + 1 : ig]);
    const Fast io{L};
    const int nx = L.npx, ny = L.npy, t = threadIdx.x, txn = max(1, (nx + TX - 1) / TX);
    const int i0 = (blockIdx.x % txn) * TX, j0 = (blockIdx.x / txn) * TY;
    // (the level-0 assembly comes right after the launch that sets `done`, so it takes `gone`)
    const bool first = !REST && ig == 0 && mode == M_DOWN;
    const bool stopped = first ? st[blockIdx.y].gone != 0 : stopped_before(st[blockIdx.y], mode);
    begin_loads(C, L);
    if (stopped) {
        pdl_enter();
        return;
    }
    const bool active = mode_active(C, ig, mode) && j0 < ny;
    if (REST && !mode_active(C, ig + 1, M_DOWN)) what = 0;
    const bool assemble = !REST || what != 0, sc_out = (what & A_SC_OUTFLOW) && C.ibc_xp == 4;
    const bool jac = (what & A_JAC) != 0;
    const Recip rm{C.relxm, C.rrelxm};
    pdl_enter();
    if (!active) return;
    const bool live = !st[blockIdx.y].done;

    const int x = 1 + t % TX, y = 1 + t / TX, i = i0 - 1 + x, j = j0 - 1 + y, q = j * nx + i;
    const bool own = i < nx && j < ny;
    const bool in = i >= 1 && j >= 1 && i <= nx - 2 && j <= ny - 2;
    const bool eu = in && i <= nx - 3, ev = in && j <= ny - 3;
    double u = 0, v = 0, ax = 0, ay = 0, p = 0, pe = 0, pn = 0, sc = 0, spu = 0, spv = 0, spsc = 0;
    double ru = 0, rv = 0, rs = 0, wu = 0, wv = 0, ghost = 0;
    unsigned code = 0;
    if (own) {
        u = io.ld(S_U, q);
        v = io.ld(S_V, q);
        ax = io.g(S_AREAX, q);
        ay = io.g(S_AREAY, q);
        if (FIELDS) sc = io.ld(S_SC, q);
    }
    if (in) {
        p = io.ld(S_P, q);
        pe = io.ld(S_P, q + 1);
        pn = io.ld(S_P, q + nx);
        if (assemble) {
            spu = io.g(S_SPU, q);
            spv = io.g(S_SPV, q);
            spsc = io.g(S_SPSC, q);
        }
        if (L.seq) code = L.seq[q];
        ru = io.ld(REST ? S_TMP0 : S_RESU, q);
        rv = io.ld(REST ? S_TMP1 : S_RESV, q);
        rs = io.ld(REST ? S_TMP2 : S_RESSC, q);
        if (j == 1) wu = io.g(S_AREAY, (ny - 2) * nx + i);
        if (i == 1) wv = io.g(S_AREAY, j * nx + nx - 2);
    }
    // the scalar's outflow ghost (:1226); in a restriction it is read, in the defect of the
    // cell west of it, so that cell's thread writes it, and the corners' their own
    const bool gown = sc_out && own && i == nx - 1 && (!REST || j == 0 || j == ny - 1);
    const bool gwest = REST && sc_out && in && i == nx - 2;
    if (gown) ghost = io.ld(S_SC, q - 1);
    int hx = 0, hy = 0;
    bool halo = false;
    double hu = 0, hv = 0, hax = 0, hay = 0, hs = 0;
    if (t < tile_halo(1)) {
        halo_at<1>(t, hx, hy);
        const int hi = i0 - 1 + hx, hj = j0 - 1 + hy;
        halo = hi >= 0 && hj >= 0 && hi < nx && hj < ny;
        if (halo) {
            const int hq = hj * nx + hi;
            hu = io.ld(S_U, hq);
            hv = io.ld(S_V, hq);
            hax = io.g(S_AREAX, hq);
            hay = io.g(S_AREAY, hq);
            if (FIELDS) hs = io.ld(S_SC, hq);
        }
    }
    double cx = 0, cy = 0;
    if (own) {
        put_geo(g, y, x, L, u, v, ax, ay, cx, cy);
        if (FIELDS) {
            fu[y][x] = u;
            fv[y][x] = v;
            fs[y][x] = sc;
        }
    }
    if (halo) {
        double a, b;
        put_geo(g, hy, hx, L, hu, hv, hax, hay, a, b);
        if (FIELDS) {
            fu[hy][hx] = hu;
            fv[hy][hx] = hv;
            fs[hy][hx] = hs;
        }
    }
    __syncthreads();
    if (!live) return;
    if (own && i <= nx - 2 && j <= ny - 2) {
        io.st(S_CX, q, cx);
        io.st(S_CY, q, cy);
    }
    auto emit = [&](int e, const Coef &k, double su, const Around &a) {
        if (F32) store_ops32(io, e, q, k, su, jac, a);
        else store_coef(io, e, q, k, su);
    };
    if (eu) {
        Coef k = tile_coef_u(g, y, x, L.amu, j == ny - 2, j == 1, j == 1 ? div_by(wu, Recip{L.dy, L.rdy}) : 0.0);
        const double body = C.dpdxm * ax * ay;
        Around a{};
        if (FIELDS) a = tile_around(fu, y, x);
        if (REST) {
            ru = ru - (stencil(k, a) + ax * (p - pe) + body);
            io.st(S_RESU, q, ru);
        }
        if (assemble) {
            const double su = mom_source(C, rm, k, ax, p - pe, u, ru, body, spu);
            emit(EQ_U, k, su, a);
            io.st(S_APU, q, k.ap);
        }
    }
    if (ev) {
        Coef k = tile_coef_v(g, y, x, L.amu, i == nx - 2, i == 1, i == 1 ? div_by(wv, Recip{L.dy, L.rdy}) : 0.0);
        const double body = C.dpdym * ax * ay;
        Around a{};
        if (FIELDS) a = tile_around(fv, y, x);
        if (REST) {
            rv = rv - (stencil(k, a) + ay * (p - pn) + body);
            io.st(S_RESV, q, rv);
        }
        if (assemble) {
            const double su = mom_source(C, rm, k, ay, p - pn, v, rv, body, spv);
            emit(EQ_V, k, su, a);
            io.st(S_APV, q, k.ap);
        }
    }
    if (in) {
        Coef k = tile_coef_sc(g, y, x, L.amusc, code);
        Around a{};
        if (FIELDS) a = tile_around(fs, y, x);
        if (REST) {
            rs = rs - stencil(k, a);
            io.st(S_RESSC, q, rs);
        }
        if (assemble) {
            k.ap = k.ap + spsc;
            if (FIELDS && sc_out && i == nx - 2) a.e = a.c;   // its ghost is (being) set to it
            emit(EQ_SC, k, spsc * C.sc_obs + rs, a);
        }
        if (gwest) io.st(S_SC, q + 1, sc);
    }
    if (gown) io.st(S_SC, q, ghost);
}

// The fine side of a restriction: restv :1354-1389, fluxes(fine) :216, the fine residuals
// of restr{u,v,sc} and their sums over each coarse cell's fine cells (:1546-1563,
// :1722-1738, :1634-1647), left in the coarse level's ping-pong buffers (free between
// smoothing calls).  A tile is 32 x 8 interior fine cells from an odd column and row, so it
// holds whole coarse cells; a coarse u face also takes the residuals of the column east of
// them, a v face those of the row north, which two warps form besides their own.  The fine
// residuals stay in shared memory (k_restv_fluxes writes them out for k_restrict to read):
// 215 us against 410 on level 0 of 64 256^2 cases.
__global__ void __launch_bounds__(NT, 3)
    k_tile_restv(const CaseDev *__restrict__ cs, CaseState *st, int ig, int mode)
{
    constexpr int H = TY + 3;
    __shared__ TileGeo<H> g;
    __shared__ double fu[H][TW], fv[H][TW], fs[H][TW], fp[H][TW], fax[H][TW], fay[H][TW];
    __shared__ double su[TY][TX + 1], sv[TY + 1][TX], ss[TY][TX];   // residuals of the tile
    const CaseDev &C = cs[blockIdx.y];
    const FastLevel L = fast_level(C.lv[ig]), LK = fast_level(C.lv[ig + 1]);
    const Fast F{L}, K{LK};
    begin_loads(C, LK);
    const int nx = L.npx, ny = L.npy, t = threadIdx.x, txn = max(1, (nx - 2 + TX - 1) / TX);
    const int i0 = 1 + (blockIdx.x % txn) * TX, j0 = 1 + (blockIdx.x / txn) * TY;
    const bool stopped = stopped_before(st[blockIdx.y], mode);
    begin_loads(C, L);
    if (stopped) {
        pdl_enter();
        return;
    }
    const bool active = mode_active(C, ig, mode) && j0 <= ny - 2;
    pdl_enter();
    if (!active) return;
    const bool live = !st[blockIdx.y].done;

    const int x = 1 + t % TX, y = 1 + t / TX, i = i0 - 1 + x, j = j0 - 1 + y, q = j * nx + i;
    const bool in = i <= nx - 2 && j <= ny - 2;
    double u = 0, v = 0, ax = 0, ay = 0, p = 0, sc = 0, ru = 0, rv = 0, rs = 0, wu = 0, wv = 0;
    unsigned code = 0;
    if (i < nx && j < ny) {
        u = F.ld(S_U, q);
        v = F.ld(S_V, q);
        ax = F.g(S_AREAX, q);
        ay = F.g(S_AREAY, q);
        p = F.ld(S_P, q);
        sc = F.ld(S_SC, q);
    }
    if (in) {
        ru = F.ld(S_RESU, q);
        rv = F.ld(S_RESV, q);
        rs = F.ld(S_RESSC, q);
        if (L.seq) code = L.seq[q];
        if (j == 1) wu = F.g(S_AREAY, (ny - 2) * nx + i);
        if (i == 1) wv = F.g(S_AREAY, j * nx + nx - 2);
    }
    // the residuals beyond the tile: v of the row north (warp 0), u of the column east (warp 1)
    const int ex = t < TX ? 1 + t : TX + 1, ey = t < TX ? TY + 1 : 1 + t - TX;
    const int ei = i0 - 1 + ex, ej = j0 - 1 + ey, eq = ej * nx + ei;
    const bool xv = t < TX && ei <= nx - 2 && ej <= ny - 3;
    const bool xu = t >= TX && t < TX + TY && ei <= nx - 3 && ej <= ny - 2;
    double er = 0, ew = 0;
    if (xv) {
        er = F.ld(S_RESV, eq);
        if (ei == 1) ew = F.g(S_AREAY, ej * nx + nx - 2);
    }
    if (xu) {
        er = F.ld(S_RESU, eq);
        if (ej == 1) ew = F.g(S_AREAY, (ny - 2) * nx + ei);
    }
    // this thread's coarse cell: restv by 64 threads, the sums by 64 threads an equation
    const int ce = t / (NT / 4), cl = t % (NT / 4), ic = i0 / 2 + 1 + cl % (TX / 2), jc = j0 / 2 + 1 + cl / (TX / 2);
    const int qc = jc * LK.npx + ic, cx_ = 2 + 2 * (cl % (TX / 2)), cy_ = 2 + 2 * (cl / (TX / 2));
    const bool coarse = ic <= LK.npx - 2 && jc <= LK.npy - 2;
    double axc = 0, ayc = 0;
    if (coarse && ce == 3) {
        axc = K.g(S_AREAX, qc);
        ayc = K.g(S_AREAY, qc);
    }
    int hx = 0, hy = 0, hq = 0;
    bool halo = false, hring = false;
    double hu = 0, hv = 0, hax = 0, hay = 0, hp = 0, hs = 0;
    if (t < tile_halo(2)) {
        halo_at<2>(t, hx, hy);
        const int hi = i0 - 1 + hx, hj = j0 - 1 + hy;
        halo = hi < nx && hj < ny;
        hring = halo && (hi == 0 || hj == 0) && hi <= nx - 2 && hj <= ny - 2;
        if (halo) {
            hq = hj * nx + hi;
            hu = F.ld(S_U, hq);
            hv = F.ld(S_V, hq);
            hax = F.g(S_AREAX, hq);
            hay = F.g(S_AREAY, hq);
            hp = F.ld(S_P, hq);
            hs = F.ld(S_SC, hq);
        }
    }
    auto put = [&](int yy, int xx, double pu, double pv, double pax, double pay, double pp, double ps, double &a,
                   double &b) {
        put_geo(g, yy, xx, L, pu, pv, pax, pay, a, b);
        fu[yy][xx] = pu;
        fv[yy][xx] = pv;
        fax[yy][xx] = pax;
        fay[yy][xx] = pay;
        fp[yy][xx] = pp;
        fs[yy][xx] = ps;
    };
    double cx, cy, hcx, hcy;
    put(y, x, u, v, ax, ay, p, sc, cx, cy);
    if (halo) put(hy, hx, hu, hv, hax, hay, hp, hs, hcx, hcy);
    __syncthreads();
    if (live) {
        if (in) {
            F.st(S_CX, q, cx);
            F.st(S_CY, q, cy);
        }
        if (hring) {
            F.st(S_CX, hq, hcx);
            F.st(S_CY, hq, hcy);
        }
    }
    const Recip rdy{L.dy, L.rdy};
    auto resid_u = [&](int yy, int xx, int gj, double res, double wall) {
        const Coef k = tile_coef_u(g, yy, xx, L.amu, gj == ny - 2, gj == 1, gj == 1 ? div_by(wall, rdy) : 0.0);
        const double a = fax[yy][xx];
        double r = stencil(k, tile_around(fu, yy, xx)) + a * (fp[yy][xx] - fp[yy][xx + 1]);
        r = r + res + C.dpdxm * a * fay[yy][xx];
        return a == 0.0 ? 0.0 : r;
    };
    auto resid_v = [&](int yy, int xx, int gi, double res, double wall) {
        const Coef k = tile_coef_v(g, yy, xx, L.amu, gi == nx - 2, gi == 1, gi == 1 ? div_by(wall, rdy) : 0.0);
        const double a = fay[yy][xx];
        double r = stencil(k, tile_around(fv, yy, xx)) + a * (fp[yy][xx] - fp[yy + 1][xx]);
        r = r + res + C.dpdym * fax[yy][xx] * a;
        return a == 0.0 ? 0.0 : r;
    };
    if (in && i <= nx - 3) su[y - 1][x - 1] = resid_u(y, x, j, ru, wu);
    if (in && j <= ny - 3) sv[y - 1][x - 1] = resid_v(y, x, i, rv, wv);
    if (in) ss[y - 1][x - 1] = stencil(tile_coef_sc(g, y, x, L.amusc, code), tile_around(fs, y, x)) + rs;
    if (xv) sv[TY][ex - 1] = resid_v(ey, ex, ei, er, ew);
    if (xu) su[ey - 1][TX] = resid_u(ey, ex, ej, er, ew);
    __syncthreads();
    if (!live || !coarse) return;
    // fine cell (2 ic, 2 jc) is at (cy_, cx_) of the field arrays, (cy_ - 1, cx_ - 1) of the residuals'
    const int a = cx_ - 1, b = cy_ - 1;
    if (ce == 0) {
        if (ic <= LK.npx - 3)
            K.st(S_TMP0, qc,
                 (su[b][a] + su[b - 1][a]) + 0.5 * (su[b][a - 1] + su[b - 1][a - 1] + su[b][a + 1] + su[b - 1][a + 1]));
    } else if (ce == 1) {
        if (jc <= LK.npy - 3)
            K.st(S_TMP1, qc,
                 (sv[b][a] + sv[b][a - 1]) + 0.5 * (sv[b - 1][a] + sv[b - 1][a - 1] + sv[b + 1][a] + sv[b + 1][a - 1]));
    } else if (ce == 2) {
        K.st(S_TMP2, qc, ss[b][a] + ss[b - 1][a] + ss[b][a - 1] + ss[b - 1][a - 1]);
    } else {
        const double cu = quotient(fu[cy_][cx_] * fax[cy_][cx_] + fu[cy_ - 1][cx_] * fax[cy_ - 1][cx_], axc + 1.0e-30);
        const double cv = quotient(fv[cy_][cx_] * fay[cy_][cx_] + fv[cy_][cx_ - 1] * fay[cy_][cx_ - 1], ayc + 1.0e-30);
        const double cp = 0.25 * (fp[cy_][cx_] + fp[cy_][cx_ - 1] + fp[cy_ - 1][cx_] + fp[cy_ - 1][cx_ - 1]);
        const double cs_ = 0.25 * (fs[cy_][cx_] + fs[cy_][cx_ - 1] + fs[cy_ - 1][cx_] + fs[cy_ - 1][cx_ - 1]);
        K.st(S_U, qc, cu);
        K.st(S_V, qc, cv);
        K.st(S_P, qc, cp);
        K.st(S_SC, qc, cs_);
        // the fine level does not change until the prolongation back into it, so these are
        // the R(x_f) the corrections subtract (prol_corr's r, same operations)
        K.st(S_RU, qc, cu);
        K.st(S_RV, qc, cv);
        K.st(S_RP, qc, cp);
        K.st(S_RSC, qc, cs_);
    }
}

// The prolongation into level ig as a gather (cell_prol_apply_io: the additions of the
// reference's scatter in its order).  The tile's 18 x 6 coarse corrections are formed once
// in shared memory (FUSED: coarse state minus the R(x_f) restv saved, written back for the
// tile's own coarse cells; else read from cell_prol_corr's arrays), each with the solid
// flags that zero it, instead of up to nine times from global memory (45 loads a cell;
// level 0 of 64 256^2 cases: 121 us against 233).  END: into level 0,
// followed by the end of the cycle; every thread reads back only the cell it just wrote.
template <bool FUSED, bool END>
__global__ void __launch_bounds__(NT, 4) k_tile_prol(const CaseDev *__restrict__ cs, CaseState *st, int ig, int mode)
{
    constexpr int CW = TX / 2 + 2, CH = TY / 2 + 2;
    __shared__ double ku[CH][CW], kv[CH][CW], kp[CH][CW], ks[CH][CW];
    __shared__ unsigned char zu[CH][CW], zv[CH][CW];
    const CaseDev &C = cs[blockIdx.y];
    const FastLevel L = fast_level(C.lv[ig]), LK = fast_level(C.lv[ig + 1]);
    const Fast F{L}, K{LK};
    const int nx = L.npx, ny = L.npy, nxc = LK.npx, nyc = LK.npy, t = threadIdx.x, txn = max(1, (nx - 2 + TX - 1) / TX);
    const int i0 = 1 + (blockIdx.x % txn) * TX, j0 = 1 + (blockIdx.x / txn) * TY;
    const bool stopped = stopped_before(st[blockIdx.y], mode);
    if (stopped) {
        pdl_enter();
        return;
    }
    const bool active = mode_active(C, ig, mode) && j0 <= ny - 2;
    pdl_enter();
    if (!active) return;
    const bool live = !st[blockIdx.y].done, stops = END && stops_on_error(C, st[blockIdx.y].last_err);
    const int x = t % TX, y = t / TX, i = i0 + x, j = j0 + y, q = j * nx + i;
    const bool in = i <= nx - 2 && j <= ny - 2;
    double u = 0, v = 0, p = 0, sc = 0;
    if (in) {
        u = F.ld(S_U, q);
        v = F.ld(S_V, q);
        p = F.ld(S_P, q);
        sc = F.ld(S_SC, q);
    }
    if (t < CW * CH) {
        const int a = t % CW, b = t / CW, ic = i0 / 2 + a, jc = j0 / 2 + b, qc = jc * nxc + ic;
        if (ic < nxc && jc < nyc) {
            const bool ci = ic >= 1 && ic <= nxc - 2, cj = jc >= 1 && jc <= nyc - 2;
            const bool du = FUSED && cj && ic >= 1 && ic <= nxc - 3, dv = FUSED && ci && jc >= 1 && jc <= nyc - 3,
                       dc = FUSED && ci && cj;
            double xu = K.ld(du ? S_U : S_CU, qc), yu = du ? K.ld(S_RU, qc) : 0.0;
            double xv = K.ld(dv ? S_V : S_CV, qc), yv = dv ? K.ld(S_RV, qc) : 0.0;
            double xp = K.ld(dc ? S_P : S_CP, qc), yp = dc ? K.ld(S_RP, qc) : 0.0;
            double xs = K.ld(dc ? S_SC : S_C, qc), ys = dc ? K.ld(S_RSC, qc) : 0.0;
            double mu = 0.0, mv = 0.0;
            if (ci && cj) {
                mu = F.g(S_SPU, 2 * jc * nx + 2 * ic);
                mv = F.g(S_SPV, 2 * jc * nx + 2 * ic);
            }
            if (du) xu = xu - yu;
            if (dv) xv = xv - yv;
            if (dc) {
                xp = xp - yp;
                if (mu > 1.0e10) xp = 0.0;
                xs = xs - ys;
            }
            ku[b][a] = xu;
            kv[b][a] = xv;
            kp[b][a] = xp;
            ks[b][a] = xs;
            zu[b][a] = mu > 1.0e10;
            zv[b][a] = mv > 1.0e10;
            if (FUSED && live && a >= 1 && a <= TX / 2 && b >= 1 && b <= TY / 2 && ci && cj) {
                if (ic <= nxc - 3) K.st(S_CU, qc, xu);
                if (jc <= nyc - 3) K.st(S_CV, qc, xv);
                K.st(S_CP, qc, xp);
                K.st(S_C, qc, xs);
            }
        }
    }
    __syncthreads();
    if (in && live) {
        const double f1 = 3. / 4., f2 = 1. / 4., g1 = 9. / 16., g2 = 3. / 16., g3 = 3. / 16., g4 = 1. / 16.;
        // coarse cell (ic, jc) of the fine pair this cell belongs to, the next one on the
        // cell's own side (in, jn), in shared coordinates (the tile starts at an odd cell)
        const int a = (x + 2) / 2, b = (y + 2) / 2;
        const int an = (i & 1) == 0 ? a + 1 : a - 1, bn = (j & 1) == 0 ? b + 1 : b - 1;
        // u faces, i in [1, nx-3]: prolu :1782-1814.  An even face takes the correction of
        // its coarse column, an odd one half of each of its neighbours'.
        if (i <= nx - 3) {
            if ((i & 1) == 0) {
                double c = f1 * ku[b][a] + f2 * ku[bn][a];
                if (zu[b][a]) c = 0.0;
                u = u + c;
            } else {
                if (i > 1) {
                    double c = f1 * ku[b][a - 1] + f2 * ku[bn][a - 1];
                    if (zu[b][a - 1]) c = 0.0;
                    u = u + 0.5 * c;
                }
                if ((i + 1) / 2 <= nxc - 3) {
                    double c = f1 * ku[b][a] + f2 * ku[bn][a];
                    if (zu[b][a]) c = 0.0;
                    u = u + 0.5 * c;
                }
            }
            F.st(S_U, q, u);
        }
        // v faces, j in [1, ny-3]: prolv :1861-1888
        if (j <= ny - 3) {
            if ((j & 1) == 0) {
                double c = f1 * kv[b][a] + f2 * kv[b][an];
                if (zv[b][a]) c = 0.0;
                v = v + c;
            } else {
                if (j > 1) {
                    double c = f1 * kv[b - 1][a] + f2 * kv[b - 1][an];
                    if (zv[b - 1][a]) c = 0.0;
                    v = v + 0.5 * c;
                }
                if ((j + 1) / 2 <= nyc - 3) {
                    double c = f1 * kv[b][a] + f2 * kv[b][an];
                    if (zv[b][a]) c = 0.0;
                    v = v + 0.5 * c;
                }
            }
            F.st(S_V, q, v);
        }
        // p and sc cells: prolp :1933-1958, prolsc :1999-2025
        p = p + (g1 * kp[b][a] + g2 * kp[b][an] + g3 * kp[bn][a] + g4 * kp[bn][an]);
        sc = sc + (g1 * ks[b][a] + g2 * ks[b][an] + g3 * ks[bn][a] + g4 * ks[bn][an]);
        F.st(S_P, q, p);
        F.st(S_SC, q, sc);
    }
    if (END && live) end_of_cycle(C, st[blockIdx.y], stops, in, i, j, tiles_of(nx - 2, ny - 2));
}

cudaError_t launch_tile(const Launch &X, const CaseDev *dc, CaseState *ds, const Sched &S, cudaStream_t st)
{
    const bool pdl = S.pdl;
    switch (X.kernel) {
    case K_ASM:
        if (X.a0 & A_F32) return launch_k(pdl, k_tile_asm<false, true>, X.grid, NT, 0, st, dc, ds, X.ig, X.mode, (unsigned)X.a0);
        return launch_k(pdl, k_tile_asm<false, false>, X.grid, NT, 0, st, dc, ds, X.ig, X.mode, (unsigned)X.a0);
    case K_RESTV_FLUXES: return launch_k(pdl, k_tile_restv, X.grid, NT, 0, st, dc, ds, X.ig, X.mode);
    case K_RESTRICT:
        if (X.a0 & A_F32) return launch_k(pdl, k_tile_asm<true, true>, X.grid, NT, 0, st, dc, ds, X.ig, X.mode, (unsigned)X.a0);
        return launch_k(pdl, k_tile_asm<true, false>, X.grid, NT, 0, st, dc, ds, X.ig, X.mode, (unsigned)X.a0);
    case K_PROL_APPLY:
        if (X.a0) return launch_k(pdl, k_tile_prol<true, false>, X.grid, NT, 0, st, dc, ds, X.ig, X.mode);
        return launch_k(pdl, k_tile_prol<false, false>, X.grid, NT, 0, st, dc, ds, X.ig, X.mode);
    case K_PROL_APPLY_END:
        if (X.a0) return launch_k(pdl, k_tile_prol<true, true>, X.grid, NT, 0, st, dc, ds, 0, X.mode);
        return launch_k(pdl, k_tile_prol<false, true>, X.grid, NT, 0, st, dc, ds, 0, X.mode);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace mg
