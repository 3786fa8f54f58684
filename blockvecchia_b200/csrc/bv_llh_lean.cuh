// bv_llh_lean.cuh -- the default FP64 block evaluation: the left-looking
// blocked Cholesky of bv_llh_big.cuh (same augmented system, panels, slab and
// shared-memory layout) run by small CTAs of 96-256 threads, several per SM,
// so that the pivot chains of several blocks overlap on one SM.
//
// Per 16-column panel p, warp 0 factors panel p's diagonal block and solves
// the rows below it while the other warps bring panel p+1 up to date.  An
// update warp takes tiles of 8 rows x 16 columns of panel p+1 and keeps a
// tile's entries in the DMMA accumulators from their generation to their last
// update from the slab:
//   * the lane that holds entry (i, j) in the m8n8k4 accumulator layout
//     evaluates its covariance (four independent entries per lane, so the
//     square-root and exponential chains overlap) -- the panel never makes
//     the round trip through shared memory between generation and update.
//     One tile at a time: two at once, with eight entries in flight, ran n =
//     1M, cs = 200 in 44.3 ms against 34.8 -- their unrolled code overflowed
//     the instruction cache (13% of the warps' stall cycles) and 128
//     registers;
//   * panels 0..p-1 are applied straight from the CTA's slab (L2-resident),
//     the next panel's fragments loaded while the current one is applied.
//     The accumulators hold the entries negated, so D = A B + D subtracts
//     each product in place without negating an operand; rounding is
//     symmetric, so the bits are those of x - a b.
// Then panel p goes to the slab and panel p+1 takes panel p's update from
// shared memory.
//
// Per element the operations and their order do not depend on the CTA size,
// the tile count or where the entry was generated, so every variant gives
// the same bits.
#pragma once

#include "bv_llh_big.cuh"

namespace bv {

// How a block's entries are generated: on 2-D locations in the update warps'
// accumulators, the closed forms and (through the table) a general nu; with a
// third coordinate (cov_xyz, long) through shared memory.  Each is a kernel of
// its own: with a call of K_nu beside it (inlined or not) the closed forms'
// kernel spills 500-900 bytes per thread (n = 1M, cs = 200: 55 against 44 ms).
enum LeanGen : int { kGenClosed = 0, kGenGeneral = 1, kGenXYZ = 2 };

// Dynamic shared memory of a launch whose largest block has M = max_m; a
// general nu takes the table's window too where it fits in `avail` (a block
// without room for it reads the table from global memory).
inline size_t lean_smem(int gen, int max_m, int nz, size_t avail)
{
    const size_t b = big_layout(max_m, 0, nz, 0).total;
    return gen == kGenGeneral ? std::max(b, std::min(avail, b + kTabWinBytes)) : b;
}

// Variants of the streamed kernel, threads x CTAs per SM (the handles' and the
// server's kernel arrays begin with these): 128 registers per thread, 204 for
// the last.
enum LeanShape : int { kLean96 = 0, kLean160 = 1, kLean256 = 2, kLean128 = 3, kLean160Wide = 4, kLeanShapes = 5 };

// The variant for a launch of `blocks` blocks, the largest of M = max_m.  More
// and larger CTAs per SM as long as two panels per CTA fit its shared memory:
// four up to M ~ 185, three up to ~ 250, two beyond; a panel of a small block
// has too few tiles for more than two update warps; a launch of at most two
// blocks per SM wants each block short.  Entries generated through shared
// memory (a third coordinate) are a larger share of the update warps' work.
// Kernel ms on 148 SMs at 96 x 5 / 160 x 3 / 256 x 2 / 128 x 4 / 160 x 2:
//   cs =  60, 150 blocks (M <=  82):    .041 / .036 / .034 / .036 / .031
//   cs = 120, 300 blocks (M <= 137):    .086 / .064 / .064 / .070 / .061
//   cs = 120, 500 blocks (M <= 137):    .099 / .107 / .109 / .092 / .107
//   cs =  60, 5k blocks (M <=  77):     0.24 / 0.32 / 0.42 / 0.26 / 0.37
//   cs =  80, 10k blocks (M <=  97):    0.74 / 0.81 / 1.08 / 0.73 / 1.01
//   cs = 120, 20k blocks (M <= 137):    2.49 / 2.73 / 3.48 / 2.42 / 3.29
//   cs = 160, 10k blocks (M <= 177):    2.59 / 2.33 / 2.58 / 2.22 / 2.76
//   cs = 200, 100k blocks (M <= 217):   46.7 / 33.7 / 37.3 / 37.4 / 42.2
//   cs = 240, 10k blocks (M <= 257):    7.28 / 5.21 / 5.26 / 5.77 / 6.25
//   cs = 300, 1.5k blocks (M <= 322):   2.88 / 1.84 / 1.43 / 2.09 / 1.84
//   cs = 300, 20k blocks (M <= 317):    33.4 / 20.9 / 17.1 / 24.1 / 20.8
// nu = 0.8:
//   cs =  60, 5k blocks (M <=  77):     0.35 / 0.42 / 0.53 / 0.36 / 0.44
//   cs =  80, 10k blocks (M <=  97):    0.95 / 1.06 / 1.34 / 0.93 / 1.13
//   cs = 120, 10k blocks (M <= 137):    1.76 / 1.70 / 2.05 / 1.59 / 1.96
//   cs = 200, 10k blocks (M <= 217):    5.37 / 4.29 / 4.60 / 4.53 / 4.84
//   cs = 300, 20k blocks (M <= 317):    35.7 / 23.8 / 20.8 / 26.8 / 23.3
// space-time:
//   cs =  30, 2.5k blocks (M <=  44):   0.20 / 0.21 / 0.23 / 0.19 / 0.26
//   cs =  47, 250 blocks (M <=  61):    .099 / .062 / .052 / .073 / .063
//   cs =  60, 500 blocks (M <=  74):    .142 / .138 / .117 / .117 / .140
//   cs =  60, 2.5k blocks (M <=  74):   0.51 / 0.46 / 0.47 / 0.46 / 0.59
//   cs = 100, 2.5k blocks (M <= 114):   1.10 / 0.96 / 0.93 / 0.98 / 1.27
//   cs = 200, 2.5k blocks (M <= 214):   5.43 / 3.23 / 3.01 / 3.91 / 4.34
inline int lean_table(int gen, int max_m, size_t blocks, int sms)
{
    const bool few = blocks <= 2 * (size_t)sms;
    if (gen == kGenXYZ) return (max_m <= 90 && !few) ? kLean128 : kLean256;
    if (max_m > 250) return kLean256;
    if (few) return kLean160Wide;
    return max_m <= 85 ? kLean96 : (max_m <= 185 ? kLean128 : kLean160);
}

// The static shared scratch the streamed path needs (a subset of
// BlockShared), for kernels that run only this path.
struct alignas(16) LeanShared {
    double Lt[kNB][kNB];  // factored diagonal block, transposed
    double inv[kNB];      // 1 / L_jj (0: failed pivot)
    double ex[4][8];      // factor_panel's exchange of a 4 x 4 diagonal block
    double red[2];        // the server's flag between blocks
    unsigned status;
    int task;
};

__device__ __forceinline__ double2 ldcg2(const double *p)
{
    return __ldcg(reinterpret_cast<const double2 *>(p));
}

__device__ __forceinline__ double2 ld2(const double *p) { return *reinterpret_cast<const double2 *>(p); }

// A lane's place in an 8-row tile (DMMA m8n8k4: row l >> 2, column pair
// 2 (l & 3)).  Tiles start at multiples of 8 rows, so the slab swizzle is a
// constant of the lane: columns 2 c4, 2 c4 + 1 at o0, 8 + 2 c4, + 1 at o1.
struct TileLane {
    int r8, c4, o0, o1;
    __device__ __forceinline__ TileLane()
    {
        const int lane = threadIdx.x & 31;
        r8 = lane >> 2;
        c4 = lane & 3;
        o0 = swz(r8, 2 * c4);
        o1 = swz(r8, 8 + 2 * c4);
    }
};

// Entries of NTILE tiles of the panel starting at row and column n0, negated:
// tile m's rows i0 + m * rstep + r8, columns n0 + 8 nj + 2 c4 + e.  Rows
// beyond the block and entries above the diagonal are zeros; row M holds the
// observations; columns beyond the block are unspecified (never used).  The
// values are those of gen_column for the closed forms (nu = 1/2, 3/2, 5/2),
// which share the distance and the exponential; the 4 NTILE entries of a lane
// are independent chains.
template <int NTILE>
__device__ __forceinline__ void gen_tiles(double (&d)[NTILE][2][2], const double *X, const double *Y,
                                          const double *Z, int M, int n0, int i0, int rstep,
                                          const TileLane &L, const MaternParams *mp)
{
    const int kind = __ldg(&mp->nu_kind);
    const double range = __ldg(&mp->range), inv_range = __ldg(&mp->inv_range);
    double xj[4], yj[4];
#pragma unroll
    for (int nj = 0; nj < 2; ++nj) {
        const double2 a = ld2(X + n0 + 8 * nj + 2 * L.c4), b = ld2(Y + n0 + 8 * nj + 2 * L.c4);
        xj[2 * nj] = a.x;
        xj[2 * nj + 1] = a.y;
        yj[2 * nj] = b.x;
        yj[2 * nj + 1] = b.y;
    }
    double r[NTILE][4];
#pragma unroll
    for (int m = 0; m < NTILE; ++m) {
        const int i = min(i0 + m * rstep + L.r8, M - 1);
        const double xi = X[i], yi = Y[i];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const double dx = xj[c] - xi, dy = yj[c] - yi;
            r[m][c] = div_by_recip(__dsqrt_rn(__fma_rn(dx, dx, __dmul_rn(dy, dy))), range, inv_range);
        }
    }
    if (!__ldg(&mp->scale_is_one)) {
        const double ds = __ldg(&mp->dist_scale), inv_ds = __ldg(&mp->inv_ds);
#pragma unroll
        for (int m = 0; m < NTILE; ++m)
#pragma unroll
            for (int c = 0; c < 4; ++c) r[m][c] = div_by_recip(r[m][c], ds, inv_ds);
    }
    const double sigma2 = __ldg(&mp->sigma2);
#pragma unroll
    for (int m = 0; m < NTILE; ++m)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const double e = exp(-r[m][c]);
            d[m][c >> 1][c & 1] = e;
        }
    if (kind == kNuThreeHalves) {
#pragma unroll
        for (int m = 0; m < NTILE; ++m)
#pragma unroll
            for (int c = 0; c < 4; ++c) d[m][c >> 1][c & 1] *= __dadd_rn(1.0, r[m][c]);
    } else if (kind == kNuFiveHalves) {
#pragma unroll
        for (int m = 0; m < NTILE; ++m)
#pragma unroll
            for (int c = 0; c < 4; ++c)
                d[m][c >> 1][c & 1] *=
                    __fma_rn(r[m][c], __dmul_rn(r[m][c], 1.0 / 3.0), __dadd_rn(1.0, r[m][c]));
    }
#pragma unroll
    for (int m = 0; m < NTILE; ++m)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            double &v = d[m][c >> 1][c & 1];
            v = (r[m][c] == 0.0) ? -sigma2 : __dmul_rn(-sigma2, v);
        }
    const double nugget = __ldg(&mp->nugget);
#pragma unroll
    for (int m = 0; m < NTILE; ++m) {
        const int i = i0 + m * rstep + L.r8;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int j = n0 + 8 * (c >> 1) + 2 * L.c4 + (c & 1);
            double &v = d[m][c >> 1][c & 1];
            if (i >= M) v = (i == M) ? -Z[j] : 0.0;
            else if (j >= i) v = (j == i) ? __dsub_rn(v, nugget) : 0.0;
        }
    }
}

// The general-nu table's part in shared memory for one block: octaves
// [base / 8, base / 8 + kTabWinOct) of the squared distance's exponent field.
struct KWindow {
    const double2 *win;  // [kTabPairs][kTabWinN]; nullptr: no room for it
    const double2 *tab;  // the whole table, in global memory
    int base;            // (exponent field << 3) of the window's first interval
};

// The same entries for a general nu, through the table (bv_ktab.cuh): the
// squared distance's exponent and top three mantissa bits give the interval.
// The loads are 16-byte shared-memory reads at random intervals (about three
// wavefronts per quarter-warp), the lanes' polynomials independent chains.
template <int NTILE>
__device__ __forceinline__ void gen_tiles_table(double (&d)[NTILE][2][2], const double *X, const double *Y,
                                                const double *Z, int M, int n0, int i0, int rstep,
                                                const TileLane &L, const MaternParams *mp, const KWindow &kw)
{
    double s[NTILE][4], t[NTILE][4];
    int k[NTILE][4];
    unsigned out = 0;  // entries of this lane outside the window
    {
        double xj[4], yj[4];
#pragma unroll
        for (int nj = 0; nj < 2; ++nj) {
            const double2 a = ld2(X + n0 + 8 * nj + 2 * L.c4), b = ld2(Y + n0 + 8 * nj + 2 * L.c4);
            xj[2 * nj] = a.x;
            xj[2 * nj + 1] = a.y;
            yj[2 * nj] = b.x;
            yj[2 * nj + 1] = b.y;
        }
#pragma unroll
        for (int m = 0; m < NTILE; ++m) {
            const int i = min(i0 + m * rstep + L.r8, M - 1);
            const double xi = X[i], yi = Y[i];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const double dx = xj[c] - xi, dy = yj[c] - yi;
                s[m][c] = __fma_rn(dx, dx, __dmul_rn(dy, dy));
                const int kk = (__double2hiint(s[m][c]) >> 17) - kw.base;
                const bool in = (unsigned)kk < (unsigned)kTabWinN;
                if (!in && s[m][c] != 0.0) out |= 1u << (4 * m + c);
                k[m][c] = in ? kk : 0;
                t[m][c] = ktab_t(s[m][c], 3);
                d[m][c >> 1][c & 1] = 0.0;
            }
        }
    }
    if (kw.win) {
#pragma unroll
        for (int h = kTabPairs - 1; h >= 0; --h)
#pragma unroll
            for (int m = 0; m < NTILE; ++m)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const double2 q = kw.win[h * kTabWinN + k[m][c]];
                    double &v = d[m][c >> 1][c & 1];
                    v = fma(fma(v, t[m][c], q.y), t[m][c], q.x);
                }
    } else {
        out = (1u << (4 * NTILE)) - 1;
    }
    const double sigma2 = __ldg(&mp->sigma2), nugget = __ldg(&mp->nugget);
    const bool any = __any_sync(0xffffffffu, out != 0);
#pragma unroll
    for (int m = 0; m < NTILE; ++m) {
        const int i = i0 + m * rstep + L.r8;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int j = n0 + 8 * (c >> 1) + 2 * L.c4 + (c & 1);
            double &v = d[m][c >> 1][c & 1];
            if (any && (out >> (4 * m + c) & 1u)) v = ktab_entry(s[m][c], mp, kw.tab);
            if (s[m][c] == 0.0) v = -sigma2;
            if (i >= M) v = (i == M) ? -Z[j] : 0.0;
            else if (j >= i) v = (j == i) ? __dsub_rn(v, nugget) : 0.0;
        }
    }
}

// Fragments of one slab panel for a group of NTILE tiles: B, the 16 rows n0..
// that every tile of the panel multiplies by, through L1 (n = 1M, cs = 200:
// 51.2 against 51.8 ms through L2 only); A, each tile's own rows, read once
// per panel, L2 only.  This CTA wrote both before the last barrier, from
// this SM.  Rows beyond the block read the following panel's memory (panel
// q + 1 holds at least 18 rows whenever panel q is applied); they only reach
// rows and columns that are never stored or never used.
// kShared: the panels are in shared memory (the one-warp kernel).
template <int NTILE, bool kShared>
struct Frags {
    double2 b[2][2], a[NTILE][2];
    __device__ __forceinline__ void load(const double *pb, const double *pa, int tstep, const TileLane &L)
    {
#pragma unroll
        for (int nj = 0; nj < 2; ++nj) {
            b[0][nj] = ld2(pb + 128 * nj + L.o0);
            b[1][nj] = ld2(pb + 128 * nj + L.o1);
        }
#pragma unroll
        for (int m = 0; m < NTILE; ++m) {
            a[m][0] = kShared ? ld2(pa + m * tstep + L.o0) : ldcg2(pa + m * tstep + L.o0);
            a[m][1] = kShared ? ld2(pa + m * tstep + L.o1) : ldcg2(pa + m * tstep + L.o1);
        }
    }
    // A lane's DMMA steps 2h and 2h+1 use the adjacent columns k = 8h + 2 c4
    // + {0, 1}, one 16-byte load for both.
    __device__ __forceinline__ void apply(double (&d)[NTILE][2][2]) const
    {
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
#pragma unroll
            for (int m = 0; m < NTILE; ++m)
#pragma unroll
                for (int nj = 0; nj < 2; ++nj)
                    dmma_8x8x4(d[m][nj][0], d[m][nj][1], (kk & 1) ? a[m][kk >> 1].y : a[m][kk >> 1].x,
                               (kk & 1) ? b[kk >> 1][nj].y : b[kk >> 1][nj].x);
    }
};

// NTILE tiles (first tile at row i0, the others rstep rows further each) take
// panels 0..p-1 from the slab.  Row i of panel q is at slab + 16 (q (Mp - 8q
// - 8) + i).
template <int NTILE, bool kShared = false>
__device__ __forceinline__ void update_tiles(double (&d)[NTILE][2][2], const double *slab, int Mp, int p,
                                             int n0, int i0, int rstep, const TileLane &L)
{
    if (p <= 0) return;
    const double *pb = slab + 16 * (n0 + L.r8), *pa = slab + 16 * (i0 + L.r8);
    const int tstep = 16 * rstep;
    int step = 16 * (Mp - 16);  // from panel q to q + 1
    Frags<NTILE, kShared> f0, f1;
    f0.load(pb, pa, tstep, L);
    for (int q = 0; q < p; q += 2) {
        if (q + 1 < p) {
            pb += step;
            pa += step;
            step -= 256;
            f1.load(pb, pa, tstep, L);
        }
        f0.apply(d);
        if (q + 1 < p) {
            if (q + 2 < p) {
                pb += step;
                pa += step;
                step -= 256;
                f0.load(pb, pa, tstep, L);
            }
            f1.apply(d);
        }
    }
}

// Panel p+1 (rows n0..): its tiles evaluated by the lanes that hold them, or
// (kGenXYZ) read from the shared panel (generated there, positive), panels
// 0..p-1 applied, the negated entries into nxt; panel 0 (p = -1, a general
// nu) in its own sign.  Warps [w0, w0 + nw) take tiles t, t + nw, ...
template <int NTILE, int GEN>
__device__ __forceinline__ void next_tiles(double *nxt, const double *X, const double *Y, const double *Z,
                                           const double *slab, int M, int p, int n0, int t0, int nw,
                                           const TileLane &L, const MaternParams *mp, const KWindow &kw)
{
    const int Mp = M + 1, i0 = n0 + 8 * t0, rstep = 8 * nw;
    double d[NTILE][2][2];
    if constexpr (GEN == kGenClosed) {
        gen_tiles<NTILE>(d, X, Y, Z, M, n0, i0, rstep, L, mp);
    } else if constexpr (GEN == kGenGeneral) {
        gen_tiles_table<NTILE>(d, X, Y, Z, M, n0, i0, rstep, L, mp, kw);
    } else {
#pragma unroll
        for (int m = 0; m < NTILE; ++m) {
            const double *row = nxt + 16 * (min(i0 + m * rstep + L.r8, M) - n0);
#pragma unroll
            for (int nj = 0; nj < 2; ++nj) {
                const double2 v = ld2(row + (nj ? L.o1 : L.o0));
                d[m][nj][0] = -v.x;
                d[m][nj][1] = -v.y;
            }
        }
    }
    update_tiles<NTILE>(d, slab, Mp, p, n0, i0, rstep, L);
    if (GEN == kGenGeneral && p < 0) {
#pragma unroll
        for (int m = 0; m < NTILE; ++m)
#pragma unroll
            for (int nj = 0; nj < 2; ++nj) {
                d[m][nj][0] = -d[m][nj][0];
                d[m][nj][1] = -d[m][nj][1];
            }
    }
#pragma unroll
    for (int m = 0; m < NTILE; ++m) {
        const int i = i0 + m * rstep + L.r8;
        if (i < Mp) {
            double *row = nxt + 16 * (i - n0);
            *reinterpret_cast<double2 *>(row + L.o0) = make_double2(d[m][0][0], d[m][0][1]);
            *reinterpret_cast<double2 *>(row + L.o1) = make_double2(d[m][1][0], d[m][1][1]);
        }
    }
}

template <int GEN>
__device__ __forceinline__ void next_panel(double *nxt, const double *X, const double *Y, const double *Z,
                                           const double *slab, int M, int p, int n0, int w0, int nw,
                                           const MaternParams *mp, const KWindow &kw)
{
    const TileLane L;
    const int ntiles = (M + 8 - n0) >> 3;  // rows n0..M
    for (int t0 = (threadIdx.x >> 5) - w0; t0 < ntiles; t0 += nw)
        next_tiles<1, GEN>(nxt, X, Y, Z, slab, M, p, n0, t0, nw, L, mp, kw);
}

// Panel p+1 (negated in nxt, rows n0..M) takes panel p's update from cur
// (rows k0.., panel p's B rows n0..n0+15): the products are summed from zero
// and subtracted, entries back to their own sign.  Tiles dealt to all warps.
template <int NT>
__device__ __forceinline__ void last_update(double *nxt, const double *cur, int M, int k0, int n0)
{
    const TileLane L;
    const int x = (L.r8 & 3) << 2;
    const double *brow = cur + 16 * (n0 - k0 + L.r8) + L.c4;
    double b[4][2];
#pragma unroll
    for (int kk = 0; kk < 4; ++kk)
#pragma unroll
        for (int nj = 0; nj < 2; ++nj)
            b[kk][nj] = (n0 + 8 * nj + L.r8 <= M) ? brow[128 * nj + ((4 * kk) ^ x)] : 0.0;
    for (int i0 = n0 + 8 * (threadIdx.x >> 5); i0 <= M; i0 += NT / 4) {
        const int i = i0 + L.r8;
        const bool in = i <= M;
        const double *arow = cur + 16 * (min(i, M) - k0) + L.c4;
        double acc[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            const double a = arow[(4 * kk) ^ x];
#pragma unroll
            for (int nj = 0; nj < 2; ++nj) dmma_8x8x4(acc[nj][0], acc[nj][1], a, b[kk][nj]);
        }
        if (in) {
            double2 *d0 = reinterpret_cast<double2 *>(nxt + 16 * (i - n0) + L.o0);
            double2 *d1 = reinterpret_cast<double2 *>(nxt + 16 * (i - n0) + L.o1);
            const double2 v0 = *d0, v1 = *d1;
            *d0 = make_double2(-v0.x - acc[0][0], -v0.y - acc[0][1]);
            *d1 = make_double2(-v1.x - acc[1][0], -v1.y - acc[1][1]);
        }
    }
}

// A row of 16 swizzled doubles (absolute row r) to and from registers.
__device__ __forceinline__ void load_row(const double *row, int r, double (&v)[kNB])
{
    const int x = (r & 3) << 2;
#pragma unroll
    for (int h = 0; h < kNB / 2; ++h) {
        const double2 t = ld2(row + ((2 * h) ^ x));
        v[2 * h] = t.x;
        v[2 * h + 1] = t.y;
    }
}

__device__ __forceinline__ void store_row(double *row, int r, const double (&v)[kNB])
{
    const int x = (r & 3) << 2;
#pragma unroll
    for (int h = 0; h < kNB / 2; ++h)
        *reinterpret_cast<double2 *>(row + ((2 * h) ^ x)) = make_double2(v[2 * h], v[2 * h + 1]);
}

// The diagonal block of panel p (rows k0.., kb <= 16 columns) and the 16 rows
// below it, by one warp, in place: lane r owns row k0 + r of cur.  The element
// operations and their order are factor_rows' (lagged Crout: the products over
// k < c - 1 in four partial sums by k mod 4, the k = c - 1 product last).
//
// The warp's time is the dependent chain of 16 pivots (an FP64 rsqrt is ~60
// cycles, a shuffle 26 and more when the SM's shared-memory pipe is busy) and
// the fetch of its code.  Four columns are done per round, one round's code
// looped: the lanes' partial sums over the earlier columns are formed by
// themselves, the 4 x 4 diagonal block's go to every lane through `ex`, and
// every lane factors that block redundantly and applies it to its own row --
// two shared-memory exchanges per four pivots instead of eight to thirty-two
// shuffles per pivot, no divergent branches, and the finished columns read
// back from the panel instead of held in registers (a lane above its diagonal
// reads what it finds there: its entry is set to zero).
//
// sh.Lt receives the factor transposed (zeros above the diagonal and beyond
// kb), sh.inv 1 / L_qq (0: failed).
//
// kUnroll: 1, one round's code (n = 200k, cs = 120, 128 x 4: 2.67 ms with an
// unrolled column-by-column factorization by shuffles, 2.45 with this), or 4,
// unrolled for the shapes that leave few warps on an SM (150 blocks, cs = 60,
// 160 x 2: .0356 looped, .0312 unrolled).
template <int kUnroll>
static __device__ __forceinline__ unsigned factor_phase(double *cur, int M, int k0, int kb, int mc,
                                                        LeanShared &sh)
{
    const int lane = threadIdx.x & 31;
    const bool low = lane < kNB;
    const bool valid = low ? lane < kb : (kb == kNB && k0 + lane <= M);
    const int x = (lane & 3) << 2;  // k0 is a multiple of 16
    double *row = cur + (valid ? lane : 0) * 16;
    unsigned st = 0;
#pragma unroll kUnroll
    for (int c0 = 0; c0 < kNB; c0 += 4) {
        double a[4][4], last = 0.0, vlast = 0.0;
        {
            const double2 u0 = ld2(row + (c0 ^ x)), u1 = ld2(row + ((c0 ^ x) + 2));
            const double u[4] = {u0.x, u0.y, u1.x, u1.y};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                a[c][0] = (valid && c0 + c < kb && (!low || c0 + c <= lane)) ? u[c] : 0.0;
                a[c][1] = a[c][2] = a[c][3] = 0.0;
            }
        }
#pragma unroll kUnroll
        for (int k = 0; k < c0; k += 4) {
            const bool end = k + 4 == c0;
            const double2 v0 = ld2(row + (k ^ x)), v1 = ld2(row + ((k ^ x) + 2));
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const double v = (j & 2) ? ((j & 1) ? v1.y : v1.x) : ((j & 1) ? v0.y : v0.x);
                const double2 p = ld2(&sh.Lt[k + j][c0]), q = ld2(&sh.Lt[k + j][c0 + 2]);
                if (j == 3 && end) {  // column c0's last product follows its sum
                    last = p.x;
                    vlast = v;
                } else {
                    a[0][j] = fma(-v, p.x, a[0][j]);
                }
                a[1][j] = fma(-v, p.y, a[1][j]);
                a[2][j] = fma(-v, q.x, a[2][j]);
                a[3][j] = fma(-v, q.y, a[3][j]);
            }
        }
        // Columns c0, c0+1: complete sums but for the products of this round;
        // c0+2, c0+3: partial sums 0, 1 and the sum of 2 and 3.
        const double s0 = fma(-vlast, last, (a[0][0] + a[0][1]) + (a[0][2] + a[0][3]));
        const double s1 = (a[1][0] + a[1][1]) + (a[1][2] + a[1][3]);
        const double g2[3] = {a[2][0], a[2][1], a[2][2] + a[2][3]};
        const double g3[3] = {a[3][0], a[3][1], a[3][2] + a[3][3]};
        if (lane >= c0 && lane < c0 + 4) {
            double2 *e = reinterpret_cast<double2 *>(sh.ex[lane - c0]);
            e[0] = make_double2(s0, s1);
            e[1] = make_double2(g2[0], g2[1]);
            e[2] = make_double2(g2[2], g3[0]);
            e[3] = make_double2(g3[1], g3[2]);
        }
        __syncwarp();
        const double2 e1 = ld2(&sh.ex[1][0]);
        const double2 e2a = ld2(&sh.ex[2][0]), e2b = ld2(&sh.ex[2][2]);
        const double2 e3a = ld2(&sh.ex[3][0]), e3b = ld2(&sh.ex[3][2]), e3c = ld2(&sh.ex[3][4]),
                      e3d = ld2(&sh.ex[3][6]);
        const double e0 = sh.ex[0][0], e2c = sh.ex[2][4];
        double piv[4], inv[4], w[4];
        bool ok[4];
        // A failed pivot's column is zero below it; rsqrt of 1 keeps the
        // evaluation branch-free.
        auto pivot = [&](int c, double y) {
            piv[c] = y;
            ok[c] = y > 0.0;
            const double z = rsqrt(ok[c] ? y : 1.0);
            inv[c] = ok[c] ? z : 0.0;
        };
        pivot(0, e0);
        const double l10 = e1.x * inv[0], l20 = e2a.x * inv[0], l30 = e3a.x * inv[0];
        w[0] = s0 * inv[0];
        pivot(1, fma(-l10, l10, e1.y));
        const double l21 = fma(-l20, l10, e2a.y) * inv[1], l31 = fma(-l30, l10, e3a.y) * inv[1];
        w[1] = fma(-w[0], l10, s1) * inv[1];
        pivot(2, fma(-l21, l21, (fma(-l20, l20, e2b.x) + e2b.y) + e2c));
        const double l32 = fma(-l31, l21, (fma(-l30, l20, e3b.x) + e3b.y) + e3c.x) * inv[2];
        w[2] = fma(-w[1], l21, (fma(-w[0], l20, g2[0]) + g2[1]) + g2[2]) * inv[2];
        pivot(3, fma(-l32, l32, (fma(-l30, l30, e3c.y) + fma(-l31, l31, e3d.x)) + e3d.y));
        w[3] = fma(-w[2], l32, (fma(-w[0], l30, g3[0]) + fma(-w[1], l31, g3[1])) + g3[2]) * inv[3];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int q = c0 + c;
            if (!ok[c] && q < kb) st |= (k0 + q < mc) ? 1u : 2u;
            w[c] = (lane > q) ? w[c] : ((lane == q) ? (ok[c] ? piv[c] * inv[c] : piv[c]) : 0.0);
            if (low) sh.Lt[q][lane] = (valid && q < kb) ? w[c] : 0.0;
            if (lane == q) sh.inv[q] = (q < kb) ? inv[c] : 0.0;
        }
        if (valid && lane >= c0) {
            *reinterpret_cast<double2 *>(row + (c0 ^ x)) = make_double2(w[0], w[1]);
            *reinterpret_cast<double2 *>(row + ((c0 ^ x) + 2)) = make_double2(w[2], w[3]);
        }
        __syncwarp();
    }
    return st;
}

// Row r below the diagonal block by forward substitution against L_kk.
// Columns beyond a partial panel have zeros in Lt and inv.
__device__ __forceinline__ void solve_row(const LeanShared &sh, double *row, int r)
{
    double w[kNB];
    load_row(row, r, w);
    double inv_q = sh.inv[0];
    double l_next = sh.Lt[0][1];
#pragma unroll
    for (int q = 0; q < kNB; ++q) {
        // The two operands on step q+1's dependent chain (1 / L_{q+1,q+1} and
        // L_{q+2,q+1}) are read one step ahead; the fence keeps the others
        // from being hoisted into spills.
        asm volatile("" ::: "memory");
        const double inv_cur = inv_q;
        const double l_cur = l_next;
        if (q + 1 < kNB) inv_q = sh.inv[q + 1];
        if (q + 2 < kNB) l_next = sh.Lt[q + 1][q + 2];
        double2 col[kNB / 2];
#pragma unroll
        for (int h = (q + 2) >> 1; h < kNB / 2; ++h) col[h] = ld2(&sh.Lt[q][2 * h]);
        w[q] *= inv_cur;
        if (q + 1 < kNB) w[q + 1] = fma(-w[q], l_cur, w[q + 1]);
#pragma unroll
        for (int c = q + 2; c < kNB; ++c) w[c] = fma(-w[q], (c & 1) ? col[c >> 1].y : col[c >> 1].x, w[c]);
    }
    store_row(row, r, w);
}

// log det of the conditional factor (positive pivots) and |u|^2 (row M) of the
// finished panels: one sum per 32 columns, by warps 0 .. kW-1 in turn, into
// sh.Lt (free by then); publish_block adds them in column order, so the value
// does not depend on the number of warps.
template <int kW>
__device__ __forceinline__ void column_sums(const double *slab, int M, int mc, int warp, LeanShared &sh)
{
    const int lane = threadIdx.x & 31, Mp = M + 1;
    for (int c = warp; mc + 32 * c < M; c += kW) {
        const int j = mc + 32 * c + lane;
        double ld = 0.0, qf = 0.0;
        if (j < M) {
            const int q = j / kNB, cc = j - q * kNB;
            const double *pq = slab + big_panel_base(q, Mp);
            const double dj = pq[(j - q * kNB) * 16 + swz(j, cc)];
            if (dj > 0) ld = log(dj * dj);
            const double u = pq[(M - q * kNB) * 16 + swz(M, cc)];
            qf = u * u;
        }
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) {
            ld += __shfl_xor_sync(0xffffffffu, ld, s);
            qf += __shfl_xor_sync(0xffffffffu, qf, s);
        }
        if (lane == 0) {
            (&sh.Lt[0][0])[c] = ld;
            (&sh.Lt[8][0])[c] = qf;
        }
    }
}

// The block's contribution and status (one thread, after column_sums).
__device__ __forceinline__ void publish_block(const LlhArgs &a, int b, int bs, const LeanShared &sh,
                                              unsigned status)
{
    double Ls = 0.0, Qs = 0.0;
    for (int c = 0; 32 * c < bs; ++c) {
        Ls += (&sh.Lt[0][0])[c];
        Qs += (&sh.Lt[8][0])[c];
    }
    const double v = -(Qs + Ls + (double)bs * a.log2pi) * 0.5;
    if (!isfinite(v)) status |= BV_ST_NONFINITE;
    a.block_llk[b] = v;
    a.block_status[b] = status | a.status_or;
}

// One block by the streamed path, run by a CTA of NT threads (warp 0 factors
// and solves, the other NT/32 - 1 warps generate and update).  smem: the
// dynamic area (big_layout(M, 0, nz, 0).total bytes); slab: this CTA's global
// slab (big_slab_doubles(M) doubles).
template <int NT, int MINB, int GEN>
__device__ __forceinline__ void process_block_lean(const LlhArgs &a, const MaternParams *mp, int b,
                                                          unsigned char *smem, double *slab, LeanShared &sh)
{
    static_assert(NT % 32 == 0 && NT > 32, "whole warps, at least one besides the factor warp");
    constexpr bool kXYZ3 = GEN == kGenXYZ;
    constexpr int kT = NT, kW = NT / 32;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int off = a.acc[b];
    const int bs = a.acc[b + 1] - off;
    const int mc = (b == 0) ? 0 : a.cs;
    const int M = mc + bs, Mp = M + 1;
    const int P = big_panels(M);
    const BigLayout l = big_layout(M, 0, kXYZ3 ? 1 : 0, 0);
    double *X = reinterpret_cast<double *>(smem + l.o_X);
    double *Y = reinterpret_cast<double *>(smem + l.o_Y);
    double *Z = reinterpret_cast<double *>(smem + l.o_Z);
    double *T = kXYZ3 ? reinterpret_cast<double *>(smem + l.o_T) : nullptr;
    double *cur = reinterpret_cast<double *>(smem + l.o_cur);
    double *nxt = reinterpret_cast<double *>(smem + l.o_next);

    // For the table the pad to whole panels repeats the last point (its
    // entries are never used, but stay in the range of the block's).
    const int *kidx = a.knn + (size_t)b * a.cs;
    for (int t = tid; t < (GEN == kGenGeneral ? P * kNB : M); t += kT) {
        const int u = (GEN == kGenGeneral) ? min(t, M - 1) : t;
        const int src = (u < mc) ? __ldg(kidx + u) : off + (u - mc);
        X[t] = __ldg(a.x + src);
        Y[t] = __ldg(a.y + src);
        Z[t] = __ldg(a.obs + src);
        if constexpr (kXYZ3) T[t] = __ldg(a.z + src);
    }
    __syncthreads();
    KWindow kw{nullptr, a.ktab, 0};
    if constexpr (GEN == kGenGeneral) {
        // Largest possible squared distance: the bounding box's diagonal.
        double x0 = X[0], x1 = x0, y0 = Y[0], y1 = y0;
        for (int t = lane; t < M; t += 32) {
            x0 = fmin(x0, X[t]);
            x1 = fmax(x1, X[t]);
            y0 = fmin(y0, Y[t]);
            y1 = fmax(y1, Y[t]);
        }
#pragma unroll
        for (int w = 16; w > 0; w >>= 1) {
            x0 = fmin(x0, __shfl_xor_sync(0xffffffffu, x0, w));
            x1 = fmax(x1, __shfl_xor_sync(0xffffffffu, x1, w));
            y0 = fmin(y0, __shfl_xor_sync(0xffffffffu, y0, w));
            y1 = fmax(y1, __shfl_xor_sync(0xffffffffu, y1, w));
        }
        const double dx = x1 - x0, dy = y1 - y0;
        const int e = (__double2hiint(fma(dx, dx, dy * dy)) >> 20) + 1;  // exponent field above it
        const int top = __ldg(&mp->kt_e1) + 1023;                        // of region 1's top
        const int first = max(min(e, top) - kTabWinOct, top - kTabOct1);
        unsigned dyn;
        asm("mov.u32 %0, %%dynamic_smem_size;" : "=r"(dyn));
        if (__ldg(&mp->kt_on) && l.total + kTabWinBytes <= dyn) {
            double2 *win = reinterpret_cast<double2 *>(smem + l.total);
            const double2 *src = a.ktab + 8 * (first - (top - kTabOct1));
            for (int t = tid; t < kTabPairs * kTabWinN; t += kT) {
                const int h = t / kTabWinN;
                win[t] = __ldg(src + h * kTabN + (t - h * kTabWinN));
            }
            kw.win = win;
            kw.base = 8 * first;
            __syncthreads();
        }
    }

    // Panel 0: thread t takes column t mod 16, every (kT/16)-th row; through
    // the table, the update warps' code makes it (in nxt) before the first
    // panel (for the closed forms that costs registers: C2's shape 3.17
    // against 2.96 ms).
    constexpr bool kFirst = GEN == kGenGeneral;
    if constexpr (!kFirst) {
        gen_column<kXYZ3>(cur, 0, X, Y, Z, T, M, Mp, 0, min(kNB, M), tid & 15, tid >> 4, kT >> 4, *mp);
        __syncthreads();
    }

    unsigned st = 0;  // warp 0: pivot flags
    for (int p = kFirst ? -1 : 0; p < P; ++p) {
        const int k0 = kFirst ? max(0, p * kNB) : p * kNB;
        const int kb = (kFirst && p < 0) ? 0 : min(kNB, M - k0);
        const int n0 = k0 + kb;                    // first row / column of panel p+1
        const int kb1 = max(0, min(kNB, M - n0));  // its width
        if (warp == 0) {
            if (!kFirst || p >= 0)
                st |= factor_phase<(NT * MINB > 320) ? 1 : 4>(cur, M, k0, kb, mc, sh);
        } else if (kb1 > 0) {
            if constexpr (kXYZ3) {
                const int u = tid - 32;
                gen_column<true>(nxt, n0, X, Y, Z, T, M, Mp, n0, kb1, u & 15, n0 + (u >> 4), (kT - 32) >> 4,
                                 *mp);
                update_warps_sync<NT>();
                next_panel<GEN>(nxt, X, Y, Z, slab, M, p, n0, 1, kW - 1, mp, kw);
            } else {
                next_panel<GEN>(nxt, X, Y, Z, slab, M, p, n0, 1, kW - 1, mp, kw);
            }
        }
        if (kFirst && p < 0) {
            __syncthreads();
            double *t = cur;
            cur = nxt;
            nxt = t;
            continue;
        }
        // The substitution needs only the factored diagonal block: warp 0
        // publishes it (named barrier 3 over the CTA: warp 0 arrives, the
        // others wait after their work on panel p+1) and goes on to its rows,
        // which overlap the other warps' generation and update.
        if (warp == 0) {
            __syncwarp();
            asm volatile("bar.arrive 3, %0;" ::"n"(NT) : "memory");
        } else {
            asm volatile("bar.sync 3, %0;" ::"n"(NT) : "memory");
        }
        // Rows below the diagonal block (after the 16 the factor warp solved
        // for a full panel).  Warp 0, idle for most of the phase before,
        // takes the first kSubstRows0 rows, the other warps the rest.
        const int rs0 = k0 + (kb == kNB ? 2 * kNB : kb);
        const int rw0 = min(Mp, rs0 + kSubstRows0);
        const int rend = (warp == 0) ? rw0 : Mp;
        for (int r = (warp == 0) ? rs0 + lane : rw0 + tid - 32; r < rend; r += (warp == 0) ? 32 : kT - 32)
            solve_row(sh, cur + (r - k0) * 16, r);
        if (warp == 0) {
            // Its rows to the slab while the others still update (after the
            // barrier, by all warps: n = 1M, cs = 200 34.6 against 33.7 ms).
            __syncwarp();
            const double2 *s2 = reinterpret_cast<const double2 *>(cur);
            double2 *g2 = reinterpret_cast<double2 *>(slab + big_panel_base(p, Mp));
            for (int e = lane; e < (rw0 - k0) * 8; e += 32) g2[e] = s2[e];
        }
        __syncthreads();
        // The other rows to the slab; panel p+1 takes panel p's update.
        if (rw0 < Mp) {
            const double2 *s2 = reinterpret_cast<const double2 *>(cur);
            double2 *g2 = reinterpret_cast<double2 *>(slab + big_panel_base(p, Mp));
            for (int e = (rw0 - k0) * 8 + tid; e < (Mp - k0) * 8; e += kT) g2[e] = s2[e];
        }
        if (kb1 > 0) last_update<NT>(nxt, cur, M, k0, n0);
        __syncthreads();
        double *t = cur;
        cur = nxt;
        nxt = t;
    }

    column_sums<kW>(slab, M, mc, warp, sh);
    if (warp == 0 && lane == 0 && st) atomicOr(&sh.status, st);
    __syncthreads();
    if (tid == 0) {
        publish_block(a, b, bs, sh, sh.status);
    }
}


// ---------------------------------------------------------------------------
// Small blocks: one warp per block.
//
// With M below ~50 a block has two or three panels of a few tiles each: the
// streamed kernel's CTA spends its time in barriers and on one warp's pivot
// chain while the others wait.  Here each warp works on a block of its own,
// with all its panels in shared memory (no slab, no copy, no block-wide
// barrier), so an SM overlaps the chains of 12 blocks instead of four.  The
// operations per element and their order are the streamed kernel's.  Kernel
// ms, 96-thread CTAs / one warp per block: classic, 30k blocks, cs = 30: 0.57
// / 0.32; cs = 10, 20k: 0.23 / 0.11; cs = 47, 30k: 0.89 / 0.61; 5k blocks of 4
// points, cs = 20: .099 / .058.  168 registers without spills (16 warps per SM
// at 128: 0.30-0.43).
// ---------------------------------------------------------------------------

constexpr int kWarpMaxM = 48;   // largest block (three panels)
constexpr int kWarpThreads = 128;

// Doubles of a warp's area: X, Y, Z padded to whole panels, then the panels
// and 16 rows of slack (a tile's rows beyond the block are read, not used).
__host__ __device__ inline size_t warp_area_doubles(int M)
{
    return (3 * 16 * (size_t)big_panels(M) + big_slab_doubles(M) + 256 + 15) & ~(size_t)15;
}

// Tiles t0, t0 + 1 (NTILE = 2) or t0 of panel p+1 (rows n0..): generated,
// panels 0..p applied, in place in the slab.
template <int NTILE>
__device__ __forceinline__ void warp_tiles(const double *X, const double *Y, const double *Z, double *slab,
                                           int M, int p, int n0, int t0, const TileLane &L,
                                           const MaternParams *mp)
{
    const int Mp = M + 1, i0 = n0 + 8 * t0;
    double d[NTILE][2][2];
    gen_tiles<NTILE>(d, X, Y, Z, M, n0, i0, 8, L, mp);
    update_tiles<NTILE, true>(d, slab, Mp, p, n0, i0, 8, L);
    double acc[NTILE][2][2];
#pragma unroll
    for (int m = 0; m < NTILE; ++m)
#pragma unroll
        for (int nj = 0; nj < 2; ++nj) acc[m][nj][0] = acc[m][nj][1] = 0.0;
    if (p >= 0) {
        // Panel p's products, summed from zero and subtracted.
        const double *cur = slab + 16 * (p * (Mp - 8 * p - 8)) + 16 * L.r8 + L.c4;
        const int x = (L.r8 & 3) << 2;
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            const int k = (4 * kk) ^ x;
            const double b0 = cur[16 * n0 + k], b1 = cur[16 * (n0 + 8) + k];
#pragma unroll
            for (int m = 0; m < NTILE; ++m) {
                const double a = cur[16 * (i0 + 8 * m) + k];
                dmma_8x8x4(acc[m][0][0], acc[m][0][1], a, b0);
                dmma_8x8x4(acc[m][1][0], acc[m][1][1], a, b1);
            }
        }
    }
    double *nxt = slab + big_panel_base(p + 1, Mp);
#pragma unroll
    for (int m = 0; m < NTILE; ++m) {
        const int i = i0 + 8 * m + L.r8;
        if (i < Mp) {
            double *row = nxt + 16 * (i - n0);
            *reinterpret_cast<double2 *>(row + L.o0) =
                make_double2(-d[m][0][0] - acc[m][0][0], -d[m][0][1] - acc[m][0][1]);
            *reinterpret_cast<double2 *>(row + L.o1) =
                make_double2(-d[m][1][0] - acc[m][1][0], -d[m][1][1] - acc[m][1][1]);
        }
    }
}

// One block (2-D, closed forms) by one warp; area: warp_area_doubles(M).
__device__ __forceinline__ void process_block_warp(const LlhArgs &a, const MaternParams *mp, int b, double *area,
                                                   LeanShared &sh)
{
    const int lane = threadIdx.x & 31;
    const int off = a.acc[b];
    const int bs = a.acc[b + 1] - off;
    const int mc = (b == 0) ? 0 : a.cs;
    const int M = mc + bs, Mp = M + 1, P = big_panels(M);
    double *X = area, *Y = X + 16 * P, *Z = Y + 16 * P, *slab = Z + 16 * P;
    const int *kidx = a.knn + (size_t)b * a.cs;
    for (int t = lane; t < M; t += 32) {
        const int src = (t < mc) ? __ldg(kidx + t) : off + (t - mc);
        X[t] = __ldg(a.x + src);
        Y[t] = __ldg(a.y + src);
        Z[t] = __ldg(a.obs + src);
    }
    __syncwarp();
    const TileLane L;
    unsigned st = 0;
    for (int p = -1; p < P; ++p) {
        const int k0 = max(0, p * kNB), kb = (p < 0) ? 0 : min(kNB, M - k0), n0 = k0 + kb;
        if (p >= 0) {
            double *cur = slab + big_panel_base(p, Mp);
            st |= factor_phase<4>(cur, M, k0, kb, mc, sh);
            __syncwarp();
            for (int r = k0 + (kb == kNB ? 2 * kNB : kb) + lane; r < Mp; r += 32)
                solve_row(sh, cur + (r - k0) * 16, r);
            __syncwarp();
        }
        if (n0 < M) {
            const int ntiles = (Mp - n0 + 7) >> 3;
            for (int t0 = 0; t0 < ntiles; t0 += 2) {
                if (t0 + 1 < ntiles)
                    warp_tiles<2>(X, Y, Z, slab, M, p, n0, t0, L, mp);
                else
                    warp_tiles<1>(X, Y, Z, slab, M, p, n0, t0, L, mp);
            }
            __syncwarp();
        }
    }
    column_sums<1>(slab, M, mc, 0, sh);
    __syncwarp();
    if (lane == 0) publish_block(a, b, bs, sh, st);
    __syncwarp();
}

}  // namespace bv
