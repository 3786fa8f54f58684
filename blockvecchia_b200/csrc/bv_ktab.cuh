// bv_ktab.cuh -- the general-nu Matern covariance as a table of polynomials,
// built on the device for each evaluation's parameters.
//
// One entry by matern_general (Temme's series or Steed's algorithm) is a loop
// of ~15 steps with dependent divisions, several hundred FP64 instructions;
// a block of M = 310 points has 48,000 of them, a layout 10^8 and more, all
// of one function of one variable.  That function of the squared distance
//     f(s) = con r^nu K_nu(r),   r = sqrt(s) / range / dist_scale,
// is analytic away from s = 0, so on an interval [a, a (1 + 1/8)] its
// Chebyshev series of degree 11 is below 1e-16 relative (measured against
// 30-digit arithmetic for nu in [0.05, 6]: at most 9e-17 for r < 11.3, with
// 1/16 instead of 1/8 at most 1e-16 up to r = 32; to nu = 40 no more).  The
// table holds:
//   region 1: 8 intervals per octave of s, 32 octaves up to r ~ 8-11.3;
//   region 2: 16 intervals per octave, the next 3 octaves (r ~ 23-32).
// Entries outside it (r below ~1.7e-4 or beyond region 2) call
// matern_general.  An entry is then 6 16-byte loads and 12 fused
// multiply-adds, no square root and no division, and its rounding is that of
// the node values plus half an ulp.  The node values are matern_general's
// own; 16 nodes per interval for 12 coefficients average their rounding.
// Entries against 40 digits, rms through the table / evaluated directly: below
// r = 2 relative 3.8e-16 / 4.2e-16 at nu = 0.8 (0.3: 3.1 / 3.3, 1.2: 4.7 / 5.0,
// 6: 21 / 24), from there 6.7e-16 / 4.5e-16, the rounding being that of an
// interval's largest value and the values falling by up to e over it; of
// sigma2, over all distances, 3.1e-16 / 3.4e-16.  ~4,900 node evaluations
// replace the entries'.
#pragma once

#include "bv_matern.cuh"

namespace bv {

constexpr int kTabDeg = 11, kTabPairs = (kTabDeg + 1) / 2;
constexpr int kTabNodes = 16;
constexpr int kTabOct1 = 32, kTabOct2 = 3;
constexpr int kTabN1 = 8 * kTabOct1, kTabN2 = 16 * kTabOct2;
constexpr int kTabN = kTabN1 + kTabN2;            // intervals
constexpr int kTabEntries = kTabPairs * kTabN;    // double2s of a table
// The part of region 1 a CTA keeps in shared memory for a block: 12 octaves
// of s below the block's largest squared distance (distances down to 1/64 of
// it), the same layout with its own interval count.
constexpr int kTabWinOct = 12, kTabWinN = 8 * kTabWinOct;
constexpr int kTabWinBytes = kTabPairs * kTabWinN * (int)sizeof(double2);

// Region 1's top: the exponent e with 2^e <= (11.3 range dist_scale)^2.  No
// table where squared distances of that size leave the normal range, or where
// matern_general does at the table's lower end (r ~ 1.2e-4): it multiplies
// con r^nu, both tiny for a large nu, by K_nu(r) < 2^(nu-1) Gamma(nu) r^-nu,
// and a node that is not finite would take its whole interval with it,
// entries of larger r among them (at nu = 60 the entries from r = 3.1e-4 to
// 3.2e-4).  At sigma2 = 1 the line is at nu ~ 55.
inline void ktab_prepare(MaternParams &p)
{
    p.kt_on = 0;
    p.kt_e1 = 0;
    const double scale = p.range * p.dist_scale;
    const double top = 11.313708498984761 * scale;
    const double s = top * top;
    if (!(s > 1e-250 && s < 1e250)) return;
    const int e1 = std::ilogb(s);
    const double log_r = 0.5 * 0.6931471805599453 * (e1 - kTabOct1) - std::log(scale);
    const double log_pow = p.nu * log_r;                                                  // r^nu
    const double log_k = (p.nu - 1.0) * 0.6931471805599453 + std::lgamma(p.nu) - log_pow;  // above K_nu(r)
    if (log_pow < -690.0 || log_k > 700.0) return;
    if (p.sigma2 != 0.0 && std::log(std::fabs(p.con)) + log_pow < -690.0) return;
    p.kt_on = 1;
    p.kt_e1 = e1;
}

// Coefficients of the Chebyshev polynomials T_0 .. T_kTabDeg: T[k][j] t^j.
struct ChebTable {
    double t[kTabDeg + 1][kTabDeg + 1];
    constexpr ChebTable() : t()
    {
        t[0][0] = 1.0;
        t[1][1] = 1.0;
        for (int k = 2; k <= kTabDeg; ++k)
            for (int j = 0; j <= k; ++j) t[k][j] = (j > 0 ? 2.0 * t[k - 1][j - 1] : 0.0) - t[k - 2][j];
    }
};
static __constant__ ChebTable kCheb;

// One interval of one table by 16 lanes (a half-warp), lane i its node i:
// Chebyshev coefficients of the node values less a reference node's (so that
// rounding scales with the function's change over the interval), then the
// monomial coefficients of -f in t in [-1, 1].  Intervals [0, kTabN) over the
// grid's x, tables over its y.
__device__ __forceinline__ void ktab_build_interval(const MaternParams &mp, int idx, double2 *tab)
{
    const int i = threadIdx.x & 15;
    const unsigned mask = 0xffffu << (threadIdx.x & 16);
    const bool r1 = idx < kTabN1;
    const int sub = r1 ? 8 : 16, o = r1 ? idx : idx - kTabN1;
    const int e = mp.kt_e1 + (r1 ? o / 8 - kTabOct1 : o / 16);
    const double lo = ldexp(1.0 + (double)(o % sub) / sub, e), half = ldexp(0.5 / sub, e);
    const double t = cospi((2 * i + 1) * (1.0 / (2 * kTabNodes)));
    const double s = lo + half * (t + 1.0);
    double r = div_by_recip(__dsqrt_rn(s), mp.range, mp.inv_range);
    if (!mp.scale_is_one) r = div_by_recip(r, mp.dist_scale, mp.inv_ds);
    const double f = matern_general(r, mp);
    const double ref = __shfl_sync(mask, f, kTabNodes / 2, 16);
    const double g = f - ref;
    double c = 0.0;
    // From the highest degree down, the smallest terms first.
    for (int k = kTabDeg; k >= 0; --k) {
        double a = g * cospi(k * (2 * i + 1) * (1.0 / (2 * kTabNodes)));
#pragma unroll
        for (int w = 8; w > 0; w >>= 1) a += __shfl_xor_sync(mask, a, w, 16);
        a *= (k == 0 ? 1.0 : 2.0) / kTabNodes;
        if (i <= kTabDeg) c = fma(a, kCheb.t[k][i], c);
    }
    if (i == 0) c += ref;
    if (i <= kTabDeg) reinterpret_cast<double *>(tab + (i >> 1) * kTabN + idx)[i & 1] = -c;
}

constexpr int kTabThreads = 64;  // 4 intervals per CTA
constexpr int kTabCtas = (kTabN + kTabThreads / 16 - 1) / (kTabThreads / 16);

// The local coordinate t in [-1, 1] of s within its interval, 2^-b of an
// octave wide: the mantissa below its top b bits.
__device__ __forceinline__ double ktab_t(double s, int b)
{
    const unsigned hi = (unsigned)__double2hiint(s), lo = (unsigned)__double2loint(s);
    const unsigned mh = (__funnelshift_l(lo, hi, b) & 0xfffffu) | 0x3ff00000u;
    return fma(2.0, __hiloint2double((int)mh, (int)(lo << b)), -3.0);
}

// -f(s) for any s > 0 through the global table, or directly outside it.  Out
// of line: the rare entries outside a block's window.
static __device__ __noinline__ double ktab_entry(double s, const MaternParams *mp, const double2 *tab)
{
    const int hi = __double2hiint(s);
    if (mp->kt_on) {
        const int base = mp->kt_e1 + 1023;
        const int i1 = (hi >> 17) - 8 * (base - kTabOct1), i2 = (hi >> 16) - 16 * base;
        if ((unsigned)i1 < (unsigned)kTabN1 || (unsigned)i2 < (unsigned)kTabN2) {
            const bool in1 = (unsigned)i1 < (unsigned)kTabN1;
            const double2 *p = tab + (in1 ? i1 : kTabN1 + i2);
            const double t = ktab_t(s, in1 ? 3 : 4);
            double v = 0.0;
#pragma unroll
            for (int h = kTabPairs - 1; h >= 0; --h) {
                const double2 c = __ldg(p + h * kTabN);
                v = fma(fma(v, t, c.y), t, c.x);
            }
            return v;
        }
    }
    double r = div_by_recip(__dsqrt_rn(s), mp->range, mp->inv_range);
    if (!mp->scale_is_one) r = div_by_recip(r, mp->dist_scale, mp->inv_ds);
    return (r == 0.0) ? -mp->sigma2 : -matern_general(r, *mp);
}

}  // namespace bv
