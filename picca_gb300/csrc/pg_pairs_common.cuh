// FP32 pair geometry with guard bands, shared by the pair kernels that decide
// bins in FP32 and leave the pairs near an edge to FP64 (pg_pairs_fast.cu,
// which also sums in FP32, and pg_pairs_runs64.cu, which sums in FP64).
#pragma once

#include "pg_f64_bits.cuh"
#include "pg_internal.cuh"

namespace pg {
namespace {

constexpr float kMagic = 12582912.0f;        // 1.5 * 2^23
constexpr unsigned kMagicBits = 0x4B400000u;  // bits of 1.5 * 2^23
constexpr float kFar = 1e30f;                 // nB, t and z of an empty slot
constexpr float kMaxGuard = 0.05f;            // widest guard band (in bins)
// cos(1e-3): above it (angles below 1e-3 rad, and the reference's flat-sky
// branch below 2 arcsec) the pair kernels take cos and sin of half the angle
// from the angle itself, not from the half-angle identities
constexpr double kCosHalfAngleForm = 0.9999995;

struct FastConst {
    double inv_p, inv_t;    // histogram scales: r_par (mu with r-mu bins) and r_trans (r)
    double geom_p;          // scale of the staged r_par geometry (inv_p; the r scale with
                            // r-mu bins, where both coordinates are in r-bin units)
    float pc;               // r_par_min * inv_p + 1/2
    float g0_par;           // guard band of x' without the |rho1| term
    float g_rho;            // guard band of x' per unit of the work item's max |rho1|
    float h_tr;             // 1/2 - g_tr: |f| above this is near an r_trans edge
    float guard_z;          // guard on z1 + z2
    float zmin2, zmax2;     // 2 z_min, 2 z_max
    unsigned np, nt;
    int nbins;
    int hstride;            // histogram array stride (nbins rounded up to 4)
    int lower_exact;        // auto-correlation with r_par_min = 0: x = |p| >= 0, so
                            // the lower edge of bin 0 can never be crossed
    // r-mu binning: mu = r_par / r in bins of inv_mu = np / (mu_max - mu_min)
    float inv_mu, mu_off;   // mu_off = mu_min * inv_mu + 1/2
    float g_mu0;            // guard of x_mu without the r_par error term
};

// Guard of the r_par coordinate of one work item (see make_fast_const).
struct ParGuard {
    float h_par;      // 1/2 - g
    float low_clamp;  // -1/2 + 2 g (auto-correlation with r_par_min = 0)
    float guard_v;    // half-plate cut guard (in units of p)
    bool wide;        // the band reaches its limit: bins too narrow for FP32
};

__device__ __forceinline__ ParGuard par_guard(const FastConst *fcp, float max_rho) {
    float g = fcp->g0_par + fcp->g_rho * max_rho;
    ParGuard pg;
    pg.wide = !(g < kMaxGuard);
    if (pg.wide) g = kMaxGuard;  // absurd bin counts: almost everything is re-decided
    pg.h_par = 0.5f - g;
    pg.low_clamp = -0.5f + 2.f * g;
    pg.guard_v = g;
    return pg;
}

// par_guard for kernels whose every decision has to be the FP64 one: with bins
// too narrow for FP32 (100,000 of them or more in half a forest) no remainder
// is certain, and the caller does not skip pairs by FP32 searches.
__device__ __forceinline__ ParGuard par_guard_exact(const FastConst *fcp, float max_rho) {
    ParGuard pg = par_guard(fcp, max_rho);
    if (pg.wide) pg.h_par = -1.f;
    return pg;
}

// The distance that a forest's others are taken relative to: its middle pixel's,
// or 0 where that is not a number or infinite; *max_rho_bits then starts at
// infinity, so that the band is wide.
__device__ __forceinline__ double reference_distance(double middle, unsigned *max_rho_bits) {
    if (isfinite(middle)) return middle;
    atomicMax(max_rho_bits, 0x7F800000u);
    return 0.;
}

// x, or low where x is below it; NaN stays NaN (decided by no bin).
__device__ __forceinline__ float clamp_low(float x, float low) { return x < low ? low : x; }

// FP32 value of a weight that stays nonzero when the FP64 weight is nonzero
// (a weight below the FP32 range still counts its pairs, as in FP64).
__device__ __forceinline__ float weight32(double w) {
    const float f = f64_to_f32(w);  // subnormal results come as 0
    if (f != 0.f) return f;
    const float g = (float)w;
    if (g == 0.f && w != 0.) return w > 0 ? 1.401298464e-45f : -1.401298464e-45f;
    return g;
}

// x as an FP32 pair: hi the nearest FP32 (to the last bit on ties), lo the
// rest (hi + lo equal to x to about 2^-48 of |x|), by integer and FP32
// operations; values near the ends of the FP32 range by conversions.
__device__ __forceinline__ float2 split_near(double x) {
    const unsigned e = ((unsigned)__double2hiint(x) >> 20) & 0x7FFu;
    if (e - 949u > 200u && x != 0.) {
        const float hi = (float)x;
        return make_float2(hi, (float)(x - (double)hi));
    }
    const float2 t = split_f64(x);  // hi truncated
    const float hi = t.x + t.y;
    return make_float2(hi, t.y - (hi - t.x));
}

// round(x) (as unsigned; negative results wrap to large values) and the
// remainder x - round(x) in [-1/2, 1/2].
__device__ __forceinline__ unsigned round_rem(float x, float &rem) {
    const float y = x + kMagic;
    rem = x - (y - kMagic);
    return __float_as_uint(y) - kMagicBits;
}

struct CfPairCtx {
    int64_t a0, b0;
    double ang, c, s, zq2;
    bool shp;
};

// Number of leading entries of a non-increasing sequence x[0..n) (the .x
// field of the staged forest-2 records) above v (OR_EQUAL: not below v).
template <bool OR_EQUAL>
__device__ __forceinline__ int count_leading(const float4 *x, int n, float v) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        const float y = x[mid].x;
        if (OR_EQUAL ? y >= v : y > v) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// Guard bands. Let u = 2^-24 (the unit roundoff of FP32). For r_par: rho1
// and rho2 are the FP64 differences r - R (exact) rounded to FP32 (errors
// u|rho1|, u|rho2|); cp carries a relative error u, nB = -cp*rho2 another
// u|cp rho2|, and the FMA p = cp*rho1 + nB rounds once (u|p|). For a pair
// whose exact x lies in [-1, n + 1] (the others are rejected either way),
// |rho2| <= |rho1| + (n + 1)/cp, so p is within 4u(n + 1) + 3u cp|rho1| of
// the exact value; the rounding of pc = pmin + 1/2 and of the subtraction add
// u(|pmin| + 1/2) and u|x'|. With cp <= inv_p and a factor 2 of margin
//   g_par = 16 u (n + |pmin| + 2) + 8 u inv_p max|rho1| + 1e-6,
// the last term taken per work item (R is the middle pixel of forest 1, so
// max|rho1| is about half the forest's length). For x_tr the FP32 rounding
// of d1 and d2 (relative u), of st, of t = st*d2 - 1/2 (one FMA) and of the
// FMA st*d1 + t give <= 6u(|x_tr| + 1), and
//   g_tr = 16 u (n + 2) + 1e-6.
// round(x') and the remainder are exact (the magic-number add rounds to an
// integer and the subtraction is exact). The reference's own FP64 evaluation
// is within 1e-12 of the exact value, far inside these bands. With
// r_par_min = 0 in an auto-correlation x = |p| >= 0 and the lower edge of bin
// 0 cannot be crossed: x' is clamped from below at -1/2 + 2g, which keeps
// pairs with |p| < 2g (same-wavelength pixels give p = 0 exactly) in bin 0
// without flagging them.
inline FastConst make_fast_const(const Binning &b) {
    FastConst fc{};
    const double u = 1.0 / 16777216.0;
    fc.inv_p = (double)b.np / b.r_par_range;
    fc.inv_t = (double)b.nt / b.r_trans_max;
    fc.geom_p = fc.inv_p;
    const double pmin = b.r_par_min * fc.inv_p;
    fc.pc = (float)(pmin + 0.5);
    fc.g0_par = (float)(16 * u * (b.np + fabs(pmin) + 2) + 1e-6);
    fc.g_rho = (float)(8 * u * fc.inv_p);
    if (b.rmu) {
        // r-mu bins (py/picca/cf.py:354-358): r_par and r_trans are staged in
        // r-bin units, r = sqrt(r_par^2 + r_trans^2) and mu = r_par / r per
        // pair; the r_par histogram holds mu (scale 1). g0_par and g_rho
        // bound the absolute error of the staged r_par in r-bin units.
        fc.geom_p = fc.inv_t;
        fc.inv_p = 1.0;
        fc.pc = 0.5f;
        fc.g0_par = (float)(16 * u * (b.nt + 2) + 1e-6);
        fc.g_rho = (float)(8 * u * fc.inv_t);
        fc.inv_mu = (float)((double)b.np / b.r_par_range);
        fc.mu_off = (float)(b.r_par_min * (double)b.np / b.r_par_range + 0.5);
        fc.g_mu0 = (float)(16 * u * (b.np + fabs(b.r_par_min * b.np / b.r_par_range) + 2) + 1e-6);
    }
    double g_tr = 16 * u * (b.nt + 2) + 1e-6;
    // r-mu: r also carries the reciprocal square root and the sum of squares
    if (b.rmu) g_tr = 32 * u * (b.nt + 2) + 1e-6;
    if (!(g_tr < (double)kMaxGuard)) g_tr = kMaxGuard;
    fc.h_tr = (float)(0.5 - g_tr);
    fc.guard_z = 1e-5f;  // z1 + z2 < 20: FP32 error below 5e-6
    fc.zmin2 = (float)(2 * b.z_min);
    fc.zmax2 = (float)(2 * b.z_max);
    fc.np = (unsigned)b.np;
    fc.nt = (unsigned)b.nt;
    fc.nbins = b.nbins;
    fc.hstride = (b.nbins + 3) & ~3;
    fc.lower_exact = (!b.x_correlation && b.r_par_min == 0.0) ? 1 : 0;
    return fc;
}

// Whether FP32 decides the bins of any geometry outside the guard bands (bins
// along r_trans: all but 50,000 of them; r_par depends on the forest, see
// par_guard_exact).
[[maybe_unused]] inline bool fast_const_exact(const FastConst &fc) {
    return fc.h_tr > 0.5f - kMaxGuard && fc.g0_par < kMaxGuard;
}

}  // namespace
}  // namespace pg
