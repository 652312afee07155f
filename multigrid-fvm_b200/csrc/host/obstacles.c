/*
 * obstacles.c — the two sequential obstacle loops of the reference, turned into
 * data the GPU can apply in parallel with the same result bit for bit.
 *
 * 1. update()'s pressure copy (Version-6-26-04.c:1153-1177).  For every obstacle in
 *    list order the reference copies into its bottom row from the row below, its
 *    top row from the row above, its left column from the left and its right column
 *    from the right; later copies overwrite earlier ones and may read cells earlier
 *    copies wrote.  Replaying the copies on cell labels gives, for every written
 *    cell, the cell whose pre-copy value it ends up holding; the GPU then does
 *    p[dst] = p_before[src].  If some source is itself a destination the gather
 *    must read all sources before writing (flag `hazard`).
 *
 * 2. coefsc()'s obstacle-face diffusion (:939-963).  Every obstacle cell adds a
 *    diffusion term to the east coefficient of its west neighbour, the west
 *    coefficient of its east neighbour, the north coefficient of its south
 *    neighbour and the south coefficient of its north neighbour, and each time the
 *    same term to that neighbour's ap.  FP addition is order-dependent, so for every
 *    receiving cell the additions are recorded in loop order as 2-bit codes
 *    (0: from the east cell into ae, 1: from the west cell into aw, 2: from the
 *    north cell into an, 3: from the south cell into as), up to 14 per cell, count
 *    in the top 4 bits.  Cells on the boundary ring are dropped: no routine reads
 *    their coefficients.
 */
#include "mgfvm_host.h"

#include <stdlib.h>
#include <string.h>

#define SEQ_MAX 14

/* Sets of cells, 64 to a word: the lists below are read off them in ascending order, for
 * the few cells an obstacle touches, without a pass over the level (64 cases of 256 x 256
 * with 20 obstacles each, all levels: 10 ms; by passes and sorts 51). */
typedef unsigned long long cellset;
#define ADD_CELL(set, q) ((set)[(q) >> 6] |= 1ull << ((q) & 63))
#define HAS_CELL(set, q) (((set)[(q) >> 6] >> ((q) & 63)) & 1)
#define EACH_CELL(set, words, q)                                                     \
    for (size_t w_ = 0; w_ < (words); ++w_)                                          \
        for (unsigned long long b_ = (set)[w_]; b_; b_ &= b_ - 1)                    \
            for (int q = (int)(w_ * 64) + __builtin_ctzll(b_), once_ = 1; once_; once_ = 0)

int mgfvm_build_obstacle_prog(const mgfvm_config *c, int ig, mgfvm_obstacle_prog *out)
{
    memset(out, 0, sizeof *out);
    if (c->nobs <= 0 || ig >= c->ig_obs) return MGFVM_OK;
    int nx = c->nfx / (1 << ig) + 2, ny = c->nfy / (1 << ig) + 2;
    size_t n = (size_t)nx * ny;
    int *origin = (int *)malloc(sizeof(int) * n);
    const size_t words = (n + 63) / 64;
    cellset *sets = (cellset *)calloc(3 * words, sizeof(cellset));
    cellset *written = sets, *added = sets + words, *owner = sets + 2 * words;
    unsigned *seq = (unsigned *)calloc(n, sizeof(unsigned));
    if (!origin || !sets || !seq) {
        free(origin); free(sets); free(seq);
        return mgfvm_fail(MGFVM_ENOMEM, "obstacle program: out of host memory");
    }
    for (size_t q = 0; q < n; ++q) origin[q] = (int)q;

    int overflow = 0, maxa = 0;
    for (int k = 0; k < c->nobs; ++k) {
        int r[4];
        mgfvm_obstacle_range(c, k, ig, r);
        int is = r[0], ie = r[1], js = r[2], je = r[3];
        /* pressure copies, in the reference's order */
        for (int i = is; i <= ie; ++i) { int d = js * nx + i; origin[d] = origin[d - nx]; ADD_CELL(written, d); }
        for (int i = is; i <= ie; ++i) { int d = je * nx + i; origin[d] = origin[d + nx]; ADD_CELL(written, d); }
        for (int j = js; j <= je; ++j) { int d = j * nx + is; origin[d] = origin[d - 1]; ADD_CELL(written, d); }
        for (int j = js; j <= je; ++j) { int d = j * nx + ie; origin[d] = origin[d + 1]; ADD_CELL(written, d); }
        /* diffusion additions, i outer and j inner as in :941-962: what a cell receives from
         * this obstacle comes from its west, south, north, east neighbour, in that order */
        if (ie < is || je < js) continue;
        for (int j = js > 1 ? js - 1 : 1; j <= je + 1 && j <= ny - 2; ++j) {
            const int in = j >= js && j <= je, lo = in ? is - 1 : is, hi = in ? ie + 1 : ie;
            const int sn = j - 1 >= js && j - 1 <= je, nn = j + 1 >= js && j + 1 <= je;
            for (int i = lo > 1 ? lo : 1; i <= hi && i <= nx - 2; ++i) {
                const int x = j * nx + i, col = i >= is && i <= ie;
                unsigned code = 0, k2 = 0;
                if (in && i - 1 >= is && i - 1 <= ie) { code = 1; k2 = 2; }
                if (sn && col) { code |= 3u << k2; k2 += 2; }
                if (nn && col) { code |= 2u << k2; k2 += 2; }
                if (in && i + 1 >= is && i + 1 <= ie) k2 += 2;
                const unsigned s = seq[x], cnt = s >> 28, now = cnt + k2 / 2;
                if (now > SEQ_MAX) { overflow = 1; continue; }
                seq[x] = (s & 0x0FFFFFFFu) | (code << (2 * cnt)) | (now << 28);
                if ((int)now > maxa) maxa = (int)now;
                if (s == 0 && now) ADD_CELL(added, x);
            }
        }
    }
    if (overflow) {
        free(origin); free(sets); free(seq);
        return mgfvm_fail(MGFVM_EUNSUPPORTED,
                          "level %d: a cell receives more than %d obstacle-face additions "
                          "(overlapping obstacles)", ig, SEQ_MAX);
    }
    int ncopy = 0, nseq = 0;
    EACH_CELL(written, words, q) if (origin[q] != q) ++ncopy;
    for (size_t w = 0; w < words; ++w) nseq += __builtin_popcountll(added[w]);
    out->dst = (int *)malloc(sizeof(int) * (size_t)(ncopy ? ncopy : 1));
    out->src = (int *)malloc(sizeof(int) * (size_t)(ncopy ? ncopy : 1));
    out->cells = (int *)malloc(sizeof(int) * (size_t)(nseq ? nseq : 1));
    out->codes = (unsigned *)malloc(sizeof(unsigned) * (size_t)(nseq ? nseq : 1));
    if (!out->dst || !out->src || !out->cells || !out->codes) {
        free(origin); free(sets); free(seq);
        mgfvm_free_obstacle_prog(out);
        return mgfvm_fail(MGFVM_ENOMEM, "obstacle program: out of host memory");
    }
    int m = 0;
    EACH_CELL(written, words, q)
        if (origin[q] != q) { out->dst[m] = q; out->src[m] = origin[q]; ++m; }
    int hazard = 0, outlet = 0;
    for (int k = 0; k < m; ++k) {
        int s = out->src[k];
        if (HAS_CELL(written, s) && origin[s] != s) hazard = 1;
        if (out->dst[k] % nx >= nx - 2 || s % nx >= nx - 2) outlet = 1;
    }
    out->touches_outlet = outlet;
    out->ncopy = m;
    out->hazard = hazard;
    if (!hazard && m > 0) {
        /* group the copies by owner: the source when interior, else the interior cell
         * next to it (sources are at most one cell outside an interior obstacle) */
        int *place = (int *)calloc(n, sizeof(int)), *own = (int *)malloc(sizeof(int) * (size_t)m);
        out->owners = (int *)malloc(sizeof(int) * (size_t)m);
        out->fan = (int *)malloc(sizeof(int) * 2 * (size_t)m);
        if (!place || !own || !out->owners || !out->fan) {
            free(place); free(own); free(origin); free(sets); free(seq);
            mgfvm_free_obstacle_prog(out);
            return mgfvm_fail(MGFVM_ENOMEM, "obstacle program: out of host memory");
        }
        for (int k = 0; k < m; ++k) {
            const int s0 = out->src[k], si = s0 % nx, sj = s0 / nx;
            const int oi = si < 1 ? 1 : (si > nx - 2 ? nx - 2 : si);
            const int oj = sj < 1 ? 1 : (sj > ny - 2 ? ny - 2 : sj);
            own[k] = oj * nx + oi;
            ++place[own[k]];
            ADD_CELL(owner, own[k]);
        }
        int at = 0;
        EACH_CELL(owner, words, q) { const int c1 = place[q]; place[q] = at; at += c1; }   /* counting sort */
        for (int k = 0; k < m; ++k) {
            const int to = place[own[k]]++;
            out->owners[to] = own[k];
            out->fan[2 * to] = out->dst[k];
            out->fan[2 * to + 1] = own[k] == out->src[k] ? -1 : out->src[k];
        }
        for (int k = 0; k < m; ++k)
            if (k == m - 1 || out->owners[k + 1] != out->owners[k]) out->fan[2 * k] |= PFAN_LAST;
        free(place); free(own);
    }
    m = 0;
    EACH_CELL(added, words, q) { out->cells[m] = q; out->codes[m] = seq[q]; ++m; }
    out->nseq = m;
    out->max_adds = maxa;
    free(origin); free(sets); free(seq);
    return MGFVM_OK;
}

void mgfvm_free_obstacle_prog(mgfvm_obstacle_prog *p)
{
    if (!p) return;
    free(p->dst); free(p->src); free(p->cells); free(p->codes); free(p->owners); free(p->fan);
    memset(p, 0, sizeof *p);
}
