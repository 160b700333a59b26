// Batched Dr16 continuum fit (delta_extraction/expected_fluxes/utils.py:12-136
// and least_squares/least_squares_cont_model.py:65-197, paths under
// py/picca), the per-iteration histograms of Dr16ExpectedFlux and the final
// delta extraction.
//
// One warp fits one forest with
//     C = (a + b x) mc,      x = (L - Lmin)/(Lmax - Lmin),
//     D = eta/ivar + var_lss C^2 + fudge ivar C^4,
//     chi2 = sum (f - C)^2 / D + sum log D
// (the reference's chi2 - sum log w with w = 1/D): chi2, its gradient and
// Hessian in (a, b) in one pass over the pixels, warp sums, damped Newton
// steps (backtracking Armijo line search). The per-pixel terms are FP64
// (cont_fit64_kernel, PG_FIT_FP64, and forests too long for the mixed form) or
// FP32 (PG_FIT_MIXED). The reference minimises the same function with
// iminuit's MIGRAD.
#include <cuda_bf16.h>

#include <type_traits>

#include "pg_cont_common.cuh"
#include "pg_internal.cuh"

namespace pg {
namespace {

constexpr int kContBlock = 256;
constexpr int kContK = 7;  // pixels per lane held in registers (forests <= 224 pixels)
constexpr int kVarBins = 100;
constexpr double kVarPipeMin = -5.0;                  // log10(1e-5)
constexpr double kVarPipeMax = 0.30102999566398120;   // log10(2)

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// scipy interp1d(kind="linear", fill_value="extrapolate"): searchsorted
// (left) clipped to [1, n-1], then slope * (v - x_lo) + y_lo. The search
// compares keys that order like the doubles (integer pipe).
__device__ __forceinline__ double interp_linear(const double *__restrict__ x,
                                                const double *__restrict__ y, int n, double v) {
    const unsigned long long key = order_key(v);
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (order_key(x[mid]) < key) lo = mid + 1;
        else hi = mid;
    }
    int idx = lo < 1 ? 1 : (lo > n - 1 ? n - 1 : lo);
    const double xl = x[idx - 1], xh = x[idx], yl = y[idx - 1], yh = y[idx];
    const double slope = (yh - yl) / (xh - xl);
    return __dadd_rn(__dmul_rn(slope, __dsub_rn(v, xl)), yl);
}

// Piece of the variance functions that holds v (searchsorted right over the
// m + 1 breakpoints, the end pieces extrapolated).
__device__ __forceinline__ int ppoly_piece(const double *__restrict__ brk, int m, double v) {
    const unsigned long long key = order_key(v);
    int lo = 0, hi = m + 1;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (order_key(brk[mid]) <= key) lo = mid + 1;
        else hi = mid;
    }
    const int i = lo - 1;
    return i < 0 ? 0 : (i > m - 1 ? m - 1 : i);
}

// Cubic i of a coefficient array (highest power first) at dx.
__device__ __forceinline__ double ppoly_at(const double *__restrict__ coef, int m, int i,
                                           double dx) {
    return ((coef[i] * dx + coef[m + i]) * dx + coef[2 * m + i]) * dx + coef[3 * m + i];
}

struct ModelEval {
    double mc, eta, var_lss, fudge;
};

__device__ __forceinline__ ModelEval eval_model(const pg_cont_model &m, double ll, double zp1,
                                                double tc) {
    ModelEval e;
    e.mc = interp_linear(m.mean_cont_x, m.mean_cont_y, m.num_mean_cont, ll - zp1) * tc;
    if (m.use_constant_weight) {
        e.eta = 0.;
        e.var_lss = 1.;
        e.fudge = 0.;
    } else {
        const int mi = m.num_var_intervals, i = ppoly_piece(m.var_breaks, mi, ll);
        const double dx = ll - m.var_breaks[i];
        e.eta = ppoly_at(m.eta_coef, mi, i, dx);
        e.var_lss = ppoly_at(m.var_lss_coef, mi, i, dx);
        e.fudge = ppoly_at(m.fudge_coef, mi, i, dx);
    }
    return e;
}

// ---------------------------------------------------------------------------
// The FP64 fit
// ---------------------------------------------------------------------------
// Bound: the FP64 pipe (16 cycles a warp operation and SM). The line search
// near the optimum compares rounding noise, so the number of steps a forest
// takes follows the last bit of every term: all of the below gives the bits of
// the plain evaluation of the formulas.
//  * The derivatives are summed as halves: scaling by a power of two commutes
//    with rounding, and an addition of a scaled term is one FMA (exact
//    product, one rounding). The terms of fudge are skipped where it is 0 for
//    the whole forest (they add exact zeros).
//  * A backtracking trial forms chi2 only, the derivatives when it is taken.
//    The values at the last accepted point are those of the solution: no
//    evaluation after the loop.
//  * The six warp sums share the levels of one butterfly (8 additions instead
//    of 30; a + b = b + a).
//  * Searches compare integer keys; the mean continuum of a pixel is kept for
//    the continuum that is written.
//  * Pixel terms are in shared memory (slot k of lane l at k * 32 + l) rather
//    than 224 registers a thread, two pixels are evaluated at a time, and warps
//    draw forests from a counter.
// 20,011 forests of 160 pixels: 7.7 ms with terms in registers and static
// forests, 4.7 ms now; 5,000 forests of 600 pixels (a warp per 32 consecutive
// forests before, 40 CTAs): 24.7 ms, 5.0 ms.
constexpr int kLongK = 32;  // pixels per lane of the long form (up to 1,024)

template <int K>
constexpr int fit64_warps() { return K == kContK ? 16 : 4; }

// One forest's terms: mc, x mc, flux, eta / ivar, var_lss, fudge ivar.
struct FitTerms64 {
    const double *ja, *jb, *f, *q, *vl, *fi;
};

struct PixelTerms64 {
    double val, gh, hh;  // chi2 term, half derivatives in C
};

template <bool DERIVATIVES, bool FUDGE>
__device__ __forceinline__ PixelTerms64 pixel_terms64(const FitTerms64 &t, int e, double a,
                                                      double b, bool const_w) {
    PixelTerms64 o;
    const double c = a * t.ja[e] + b * t.jb[e];
    const double c2 = c * c;
    const double vl = t.vl[e];
    double d = t.q[e] + vl * c2, fc = 0.;
    if (FUDGE) {
        fc = t.fi[e] * c2;
        d = d + fc * c2;
    }
    const double r = t.f[e] - c;
    const double id = __drcp_rn(d);
    const double rid = r * id;
    o.val = r * rid + (const_w ? 0. : log(d));
    if (DERIVATIVES) {
        // hd = (dD/dC) / 2, h2 = (d2D/dC2) / 2
        double hd = vl * c, h2 = vl;
        if (FUDGE) {
            hd = fma(2., fc * c, hd);
            h2 = vl + (6. * t.fi[e]) * c2;
        }
        const double w = hd * id;
        const double r2 = rid * rid;
        const double p = r2 * hd;
        o.gh = (-rid - p) + w;
        double hh = fma(4., rid * w, id);
        hh = fma(4., p * w, hh);
        hh = hh - r2 * h2;
        hh = hh + h2 * id;
        o.hh = fma(-2., w * w, hh);
    }
    return o;
}

// Sums of one lane's pixels: chi2 and the half derivatives.
template <bool DERIVATIVES, bool FUDGE>
__device__ __forceinline__ void lane_sums64(const FitTerms64 &t, unsigned valid, int nk, double a,
                                            double b, bool const_w, double s[6]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int q = 0; q < 6; ++q) s[q] = 0.;
    auto add = [&](const PixelTerms64 &o, int e) {
        s[0] += o.val;
        if (DERIVATIVES) {
            const double ja = t.ja[e], jb = t.jb[e];
            s[1] += o.gh * ja;
            s[2] += o.gh * jb;
            const double ha = o.hh * ja;
            s[3] += ha * ja;
            s[4] += ha * jb;
            s[5] += (o.hh * jb) * jb;
        }
    };
    int k = 0;
#pragma unroll 1
    for (; k + 1 < nk; k += 2) {
        const int e = k * 32 + lane;
        const PixelTerms64 o0 = pixel_terms64<DERIVATIVES, FUDGE>(t, e, a, b, const_w);
        const PixelTerms64 o1 = pixel_terms64<DERIVATIVES, FUDGE>(t, e + 32, a, b, const_w);
        if ((valid >> k) & 1u) add(o0, e);
        if ((valid >> k) & 2u) add(o1, e + 32);
    }
    if (k < nk && ((valid >> k) & 1u)) {
        const int e = k * 32 + lane;
        add(pixel_terms64<DERIVATIVES, FUDGE>(t, e, a, b, const_w), e);
    }
}

// warp_sum of six values, in every lane: level by level of the same
// butterfly, each lane carrying only the values it is to deliver.
__device__ __forceinline__ void warp_sum6(double s[6]) {
    const int lane = threadIdx.x & 31;
    const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
    double v[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const double keep = b4 ? s[q + 3] : s[q], give = b4 ? s[q] : s[q + 3];
        v[q] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
    }
    // lanes without bit 3: v[0], v[1]; with it: v[2]
    const double k0 = b3 ? v[2] : v[0], g0 = b3 ? v[0] : v[2];
    double u0 = k0 + __shfl_xor_sync(0xffffffffu, g0, 8);
    const double u1 = v[1] + __shfl_xor_sync(0xffffffffu, v[1], 8);
    // lanes with bit 2 deliver v[1] (of the lanes without bit 3)
    const double k1 = b2 && !b3 ? u1 : u0, g1 = b2 ? u0 : (b3 ? u0 : u1);
    u0 = k1 + __shfl_xor_sync(0xffffffffu, g1, 4);
    u0 += __shfl_xor_sync(0xffffffffu, u0, 2);
    u0 += __shfl_xor_sync(0xffffffffu, u0, 1);
#pragma unroll
    for (int q = 0; q < 6; ++q)
        s[q] = __shfl_sync(0xffffffffu, u0, (q >= 3 ? 16 : 0) + (q % 3 == 2 ? 8 : 0) +
                                                (q % 3 == 1 ? 4 : 0));
}

template <bool DERIVATIVES>
__device__ __noinline__ void fit_sums64(const FitTerms64 &t, unsigned valid, int nk, double a,
                                        double b, bool const_w, bool fudge, double s[6]) {
    if (fudge) lane_sums64<DERIVATIVES, true>(t, valid, nk, a, b, const_w, s);
    else lane_sums64<DERIVATIVES, false>(t, valid, nk, a, b, const_w, s);
    if (!DERIVATIVES) {
        s[0] = warp_sum(s[0]);
        return;
    }
    warp_sum6(s);
#pragma unroll
    for (int q = 1; q < 6; ++q) s[q] *= 2.;
}

// Forests of at most 32 * kContK pixels (K = kContK; a warp draws `group`
// forests at a time) or of more, up to 32 * K (K = kLongK; draws
// of half a warp's share of what is left, down to one forest, whose lengths are
// looked at 32 at a time: a set without long forests is passed over in some
// thousand draws, and long ones are shared out singly at the end).
template <int K>
__global__ void __launch_bounds__(fit64_warps<K>() * 32) cont_fit64_kernel(
    const __grid_constant__ pg_spectra sp, const __grid_constant__ pg_cont_model m,
    const double *__restrict__ start, const int32_t *__restrict__ index, int64_t count,
    int max_iter, double tol, const __grid_constant__ pg_cont_fit out, int32_t *counter,
    int group, Scratch *scratch) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int S = 32 * K;
    const int lane = threadIdx.x & 31;
    double *slab = reinterpret_cast<double *>(smem) + (size_t)(threadIdx.x >> 5) * 6 * S;
    const FitTerms64 t = {slab, slab + S, slab + 2 * S, slab + 3 * S, slab + 4 * S, slab + 5 * S};
    const bool const_w = m.use_constant_weight != 0;
    const int nwarps = gridDim.x * (blockDim.x >> 5);
    int64_t w_next = 0, w_end = 0;
    unsigned todo = 0;
    for (;;) {
        int64_t w;
        if (K == kContK) {
            if (w_next == w_end) {
                int g = 0;
                if (lane == 0) g = atomicAdd(counter, 1);
                w_next = (int64_t)__shfl_sync(0xffffffffu, g, 0) * group;
                if (w_next >= count) break;
                w_end = min(count, w_next + group);
            }
            w = w_next++;
        } else {
            while (!todo) {
                if (w_next >= w_end) {
                    int t = 0;
                    if (lane == 0) t = atomicAdd(counter, 1);
                    t = __shfl_sync(0xffffffffu, t, 0);
                    unsigned left = (unsigned)count, size = max(1u, left / (2u * nwarps));
                    for (; t >= nwarps && left > size * nwarps; t -= nwarps) {
                        left -= size * nwarps;
                        size = max(1u, left / (2u * nwarps));
                    }
                    w_next = count - left + (int64_t)t * size;
                    if (w_next >= count) break;
                    w_end = min(count, w_next + size);
                }
                bool is_long = false;
                if (w_next + lane < w_end) {
                    const int64_t g = index ? (int64_t)index[w_next + lane] : w_next + lane;
                    is_long = sp.pix_offset[g + 1] - sp.pix_offset[g] > 32 * kContK;
                }
                todo = __ballot_sync(0xffffffffu, is_long);
                w_next += 32;
            }
            if (!todo) break;
            w = w_next - 32 + (__ffs(todo) - 1);
            todo &= todo - 1;
        }
        const int64_t f = index ? (int64_t)index[w] : w;
        const int64_t off = sp.pix_offset[f];
        const int64_t n64 = sp.pix_offset[f + 1] - off;
        if (K == kContK && n64 > S) continue;  // the other form's forest
        if (n64 <= 0 || n64 > S) {
            if (lane == 0) {
                if (n64 > 0) report_error(scratch, PG_ERR_UNSUPPORTED, (int32_t)f);
                out.zero_point[f] = NAN;
                out.slope[f] = NAN;
                out.chi2[f] = NAN;
                out.ndata[f] = 0;
                out.status[f] = 1;
                out.iterations[f] = 0;
            }
            continue;
        }
        const int n = (int)n64;
        const int nk = (n + 31) >> 5;
        const double zp1 = log10(1 + sp.z_qso[f]);
        const double ll_min = m.log_lambda_rest_min + zp1;
        const double ll_max = m.log_lambda_rest_max + zp1;
        unsigned valid = 0;
        bool fudge = false;
        double sfi = 0., si = 0.;
        __syncwarp();
        for (int k = 0; k < nk; ++k) {
            const int p = lane + 32 * k, e = k * 32 + lane;
            double ja = 0., jb = 0., fl = 0., q = 1., vl = 0., fi = 0.;
            if (p < n) {
                const double ll = sp.log_lambda[off + p];
                const double iv = sp.ivar[off + p];
                fl = sp.flux[off + p];
                sfi += fl * iv;
                si += iv;
                if (iv > 0) {
                    const ModelEval ev = eval_model(m, ll, zp1, sp.transmission_correction[off + p]);
                    const double x = (ll - ll_min) / (ll_max - ll_min);
                    ja = ev.mc;
                    jb = x * ev.mc;
                    if (!const_w) {
                        q = ev.eta / iv;
                        vl = ev.var_lss;
                        fi = ev.fudge * iv;
                    }
                    valid |= 1u << k;
                    fudge |= fi != 0.;
                }
            }
            slab[e] = ja; slab[S + e] = jb; slab[2 * S + e] = fl;
            slab[3 * S + e] = q; slab[4 * S + e] = vl; slab[5 * S + e] = fi;
        }
        fudge = __any_sync(0xffffffffu, fudge);
        sfi = warp_sum(sfi);
        si = warp_sum(si);
        const double a0 = sfi / si;  // utils.py:92
        // ndata: pixels with a positive weight at the reference's starting
        // point (a0, 0) (cont_model.py:88-92)
        int nd = 0;
        for (int k = 0; k < nk; ++k) {
            if ((valid >> k) & 1u) {
                const int e = k * 32 + lane;
                const double c = a0 * t.ja[e];
                const double d = t.q[e] + t.vl[e] * c * c + t.fi[e] * c * c * c * c;
                nd += (d > 0.) ? 1 : 0;
            }
        }
        nd = __reduce_add_sync(0xffffffffu, nd);
        double a = a0, b = 0.;
        if (start) {
            a = start[2 * f];
            b = m.order == 0 ? 0. : start[2 * f + 1];
        }
        double s[6];
        fit_sums64<true>(t, valid, nk, a, b, const_w, fudge, s);
        int it = 0;
        // max_iter == 0 with a start: evaluate the model at the given (a, b)
        bool converged = max_iter == 0 && start != nullptr;
        for (; it < max_iter; ++it) {
            double da, db;
            if (m.order == 0) {
                da = s[3] > 0 ? -s[1] / s[3] : -s[1];
                db = 0.;
            } else {
                const double det = s[3] * s[5] - s[4] * s[4];
                if (det > 0 && s[3] > 0) {
                    da = -(s[5] * s[1] - s[4] * s[2]) / det;
                    db = -(s[3] * s[2] - s[4] * s[1]) / det;
                } else {
                    const double scale = fmax(fabs(s[3]), fabs(s[5]));
                    da = -s[1] / (scale > 0 ? scale : 1.);
                    db = -s[2] / (scale > 0 ? scale : 1.);
                }
                if (da * s[1] + db * s[2] >= 0) {  // not a descent direction
                    const double scale = fmax(fabs(s[3]), fabs(s[5]));
                    da = -s[1] / (scale > 0 ? scale : 1.);
                    db = -s[2] / (scale > 0 ? scale : 1.);
                }
            }
            const double slope_dir = da * s[1] + db * s[2];
            double step = 1.;
            double trial[6];
            bool accepted = false;
            for (int ls = 0; ls < 40; ++ls) {
                const double at = a + step * da, bt = b + step * db;
                if (ls == 0) fit_sums64<true>(t, valid, nk, at, bt, const_w, fudge, trial);
                else fit_sums64<false>(t, valid, nk, at, bt, const_w, fudge, trial);
                if (isfinite(trial[0]) && trial[0] <= s[0] + 1e-4 * step * slope_dir) {
                    if (ls > 0) fit_sums64<true>(t, valid, nk, at, bt, const_w, fudge, trial);
                    accepted = true;
                    break;
                }
                step *= 0.5;
            }
            if (!accepted) {
                converged = fabs(s[1]) + fabs(s[2]) < 1e-6 * fmax(1., fabs(s[0]));
                break;
            }
            a += step * da;
            b += step * db;
#pragma unroll
            for (int k = 0; k < 6; ++k) s[k] = trial[k];
            if (fabs(step * da) < tol * fmax(1., fmax(fabs(a), fabs(b))) &&
                fabs(step * db) < tol * fmax(1., fmax(fabs(a), fabs(b)))) {
                converged = true;
                ++it;
                break;
            }
        }
        // the continuum with the reference's operation order
        // (cont_model.py:138-144); s holds chi2 at (a, b)
        bool negative = false, all_zero = true;
        for (int k = 0; k < nk; ++k) {
            const int p = lane + 32 * k;
            if (p >= n) continue;
            const double ll = sp.log_lambda[off + p];
            const double mc = ((valid >> k) & 1u)
                                  ? t.ja[k * 32 + lane]
                                  : interp_linear(m.mean_cont_x, m.mean_cont_y, m.num_mean_cont,
                                                  ll - zp1) * sp.transmission_correction[off + p];
            const double line = b * (ll - ll_min) / (ll_max - ll_min) + a;
            const double c = line * mc;
            if (out.continuum) out.continuum[off + p] = c;
            negative |= c < 0;
            all_zero &= c == 0;
        }
        negative = __any_sync(0xffffffffu, negative);
        all_zero = __all_sync(0xffffffffu, all_zero);
        if (lane == 0) {
            int status = converged ? 0 : 1;
            if (negative) status = 2;
            if (all_zero) status = 3;
            out.zero_point[f] = status == 0 ? a : NAN;
            out.slope[f] = status == 0 ? b : NAN;
            out.chi2[f] = status == 0 ? s[0] : NAN;
            out.ndata[f] = nd;
            out.status[f] = status;
            out.iterations[f] = it;
        }
    }
}

template <int K>
int launch_fit64(const pg_spectra &sp, const pg_cont_model &m, const double *start,
                 const int32_t *index, int64_t count, int max_iter, double tol,
                 const pg_cont_fit &out, int32_t *counter, Scratch *scratch, int num_sms,
                 cudaStream_t stream) {
    // few forests: one warp a forest, spread over the SMs (each has one FP64 pipe;
    // 100 forests in CTAs of 16 warps: 785 us, 434 us spread)
    const int64_t share = (count + num_sms - 1) / num_sms;
    const int warps = (int)(share < fit64_warps<K>() ? share : fit64_warps<K>());
    constexpr size_t warp_bytes = (size_t)6 * 32 * K * sizeof(double);
    const size_t smem = warps * warp_bytes;
    cudaError_t err = cudaFuncSetAttribute(cont_fit64_kernel<K>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)(fit64_warps<K>() * warp_bytes));
    if (err != cudaSuccess) return check_cuda(err);
    int64_t blocks = (count + warps - 1) / warps;
    if (blocks > num_sms) blocks = num_sms;
    // forests drawn one at a time, several where there are many (a draw by
    // every warp for each of them would queue at the counter)
    int64_t group = count / (blocks * warps * 16);
    group = group < 1 ? 1 : (group > 32 ? 32 : group);
    cont_fit64_kernel<K><<<(unsigned)blocks, warps * 32, smem, stream>>>(
        sp, m, start, index, count, max_iter, tol, out, counter, (int)group, scratch);
    return check_cuda(cudaGetLastError());
}

// ---------------------------------------------------------------------------
// Mixed-precision fit (PG_FIT_MIXED): FP32 per-pixel terms, FP32 lane and
// warp sums, FP64 2x2 Newton solve. GB300 executes FP64 at 1/64 of the FP32
// rate, so the per-pixel work avoids FP64 except for the three differences
// whose operands are close (the rest-frame argument of the mean continuum,
// its offset from the interpolation node, and the offset from the forest's
// lower wavelength limit). The model tables are copied to shared memory in
// FP32 (plus the FP64 nodes of the mean continuum and per-interval slopes
// computed in FP64), so the interpolation searches use FP32 comparisons.
// Newton steps larger than 1e-3 of max(1, |a|, |b|) are damped by an Armijo
// line search on chi2; smaller steps, inside the region of quadratic
// convergence, are taken in full, because there the change of chi2 is below
// the resolution of FP32 sums. The iteration stops when the step is below
// max(tol, 1e-6) * max(1, |a|, |b|): the error left is about the square of
// the last step plus the FP32 rounding of the gradient (about 1e-8
// relative). The reported chi2 sums the FP32 terms with compensation; the
// continuum is (b x + a) mc in FP32, stored as FP64.
// ---------------------------------------------------------------------------
// One lane's pixels of the mixed fit, in the warp's shared-memory slab
// (slot k of lane l at k * 32 + l: conflict-free, and no lane reads another
// lane's entries). Unused and masked slots hold mc = 0, f = 0, q = 1,
// vl = fi = 0 and contribute exactly nothing.
struct FitSlab {
    float4 *a;  // mc, x, f, q
    float2 *b;  // vl, fi
};

constexpr size_t kFitSlabBytes = (size_t)kContK * 32 * (sizeof(float4) + sizeof(float2));

// chi2 (with want_val), gradient and Hessian in (a, b) of one lane's pixels,
// summed over the warp: s = {chi2, ga, gb, haa, hab, hbb}. The per-pixel
// algebra with h = dD/dC / 2, e = h / D:
//     dchi2/dC / 2   = e - r/D (1 + r h / D)
//     d2chi2/dC2 / 2 = 1/D + h' (1/D - (r/D)^2) + e (4 (r/D)(1 + r h/D) - 2 e)
// where h' = d2D/dC2 / 2 = vl + 6 fi C^2. Without want_val (the Newton
// iterations near the optimum) the reciprocal is the approximate one (two
// ulps) and chi2 itself is not formed.
__device__ __noinline__ void fit_terms(const FitSlab &px, int lane, int nk, float a, float b,
                                          bool const_w, bool want_val, float s[6]) {
    float val = 0.f, ga = 0.f, gb = 0.f, haa = 0.f, hab = 0.f, hbb = 0.f;
#pragma unroll 1
    for (int k = 0; k < nk; ++k) {
        const float4 pa = px.a[k * 32 + lane];
        const float2 pb = px.b[k * 32 + lane];
        const float c = pa.x * fmaf(b, pa.y, a);
        const float c2 = c * c;
        const float t1 = fmaf(pb.y, c2, pb.x);
        const float d = fmaf(t1, c2, pa.w);
        const float hd = c * fmaf(pb.y, c2, t1);                         // (dD/dC) / 2
        const float h2 = fmaf(4.f * pb.y, c2, fmaf(pb.y, c2, t1));       // vl + 6 fi C^2
        const float r = pa.z - c;
        const float id = want_val ? 1.f / d : __fdividef(1.f, d);
        const float rid = r * id;
        const float e = hd * id;
        const float w1 = fmaf(rid, hd, 1.f);
        const float g = fmaf(-rid, w1, e);
        const float hh = fmaf(h2, fmaf(-rid, rid, id), id) + e * fmaf(4.f * rid, w1, -2.f * e);
        const float gj = g * pa.x;
        ga += gj;
        gb = fmaf(gj, pa.y, gb);
        const float hj = hh * pa.x * pa.x;
        haa += hj;
        const float hjx = hj * pa.y;
        hab += hjx;
        hbb = fmaf(hjx, pa.y, hbb);
        if (want_val) val += fmaf(r, rid, const_w ? 0.f : logf(d));
    }
    // gradient and Hessian of chi2 (the factors 2 of the half-derivatives)
    s[0] = val;
    s[1] = 2.f * ga; s[2] = 2.f * gb;
    s[3] = 2.f * haa; s[4] = 2.f * hab; s[5] = 2.f * hbb;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int q = 0; q < 6; ++q) s[q] += __shfl_xor_sync(0xffffffffu, s[q], o);
    }
}

constexpr int kFitGroup = 8;  // forests per work item of the mixed fit

struct FitSlot {
    int64_t f, off;
    int n, nd, status, it, write;
    float lm_hi, lm_lo;     // Lmin = rest-frame start + log10(1 + z), two floats
    float ah, al, bh, bl;   // the start, then the result (two-float sums)
    float cs, ce;           // chi2 (compensated)
};

// Mixed-precision fit: FP32 per-pixel terms, (a, b) as two-float sums.
// Forests are handed out kFitGroup at a time from a work counter; the
// per-forest FP64 scalars (log10(1 + z), the start, the outputs) are
// computed by the group's lanes in parallel rather than by one lane per
// forest.
//
// cert_chi2 > 0 selects the certificate stop of the warm-started fit
// (pg_cont_fit_warm). Once a Newton step d = -H^-1 g is at most
// sqrt(cert_ab) * max(1, |a|, |b|) (Newton's convergence is quadratic, so the
// error after it is of order |d|^2), the step is taken and the iteration
// ends; the final pass, which evaluates chi2 at the new point anyway, also
// sums the gradient g' there and certifies the point: the remaining step
// H^-1 g' (with the last Hessian) at most cert_ab * max(1, |a|, |b|) and half
// the Newton decrement, g'.H^-1 g' / 2 (chi2's excess over the minimum of its
// quadratic model), at most cert_chi2 * max(|chi2|, ndata). There is no FP64
// finish; a forest not certified within max_iter iterations gets status 1
// (the caller re-fits it with the plain fit).
__global__ void __launch_bounds__(kContBlock, 4) cont_fit_mixed_kernel(
    const __grid_constant__ pg_spectra sp, const __grid_constant__ pg_cont_model m,
    const double *__restrict__ start, const int32_t *__restrict__ index, int64_t count,
    int max_iter, double tol, const __grid_constant__ pg_cont_fit out, Scratch *scratch,
    float cert_chi2, float cert_ab) {
    extern __shared__ __align__(16) unsigned char smem[];
    const FitTables tab = load_fit_tables(m, smem + kFitSlabBytes * (kContBlock / 32));
    const int lane = threadIdx.x & 31;
    FitSlab px;
    px.a = reinterpret_cast<float4 *>(smem + kFitSlabBytes * (threadIdx.x >> 5));
    px.b = reinterpret_cast<float2 *>(px.a + kContK * 32);
    const bool const_w = m.use_constant_weight != 0;
    const float eff_tol = tol > 1e-6 ? (float)tol : 1e-6f;
    const bool evaluate_only = max_iter == 0 && start != nullptr;
    const bool certify = cert_chi2 > 0.f;
    const float inv_span = tab.inv_span;
    const int64_t num_groups = (count + kFitGroup - 1) / kFitGroup;
    // the group's per-forest scalars and results, in shared memory (not
    // registers) while the warp fits the forests one after the other
    __shared__ FitSlot s_slots[kContBlock / 32][kFitGroup];
    FitSlot *slots = s_slots[threadIdx.x >> 5];
    for (;;) {
        int64_t group = 0;
        if (lane == 0) group = atomicAdd(&scratch->work_counter, 1);
        group = __shfl_sync(0xffffffffu, group, 0);
        if (group >= num_groups) break;
        if (lane < kFitGroup) {
            FitSlot sl;
            sl.f = -1;
            sl.off = 0;
            sl.n = 0;
            sl.lm_hi = sl.lm_lo = sl.ah = sl.al = sl.bh = sl.bl = 0.f;
            sl.cs = NAN;
            sl.ce = 0.f;
            sl.nd = 0;
            sl.status = 1;
            sl.it = 0;
            sl.write = 0;
            if (group * kFitGroup + lane < count) {
                const int64_t w = group * kFitGroup + lane;
                sl.f = index ? (int64_t)index[w] : w;
                sl.off = sp.pix_offset[sl.f];
                sl.n = (int)(sp.pix_offset[sl.f + 1] - sl.off);
                const float2 lm = split_f64(m.log_lambda_rest_min + log10(1. + sp.z_qso[sl.f]));
                sl.lm_hi = lm.x;
                sl.lm_lo = lm.y;
                if (start) {
                    const float2 sa = split_f64(start[2 * sl.f]);
                    const float2 sb =
                        m.order == 0 ? make_float2(0.f, 0.f) : split_f64(start[2 * sl.f + 1]);
                    // renormalise (hi + lo) to a two-float sum
                    sl.ah = sa.x + sa.y;
                    sl.al = sa.y - (sl.ah - sa.x);
                    sl.bh = sb.x + sb.y;
                    sl.bl = sb.y - (sl.bh - sb.x);
                }
            }
            slots[lane] = sl;
        }
        __syncwarp();
        for (int j = 0; j < kFitGroup; ++j) {
            const int64_t f = slots[j].f;
            if (f < 0) break;
            const int64_t off = slots[j].off;
            const int n = slots[j].n;
            if (n > 32 * kContK) continue;  // a long forest: cont_fit64_kernel<kLongK>
            if (lane == j) slots[j].write = 1;
            if (n <= 0) continue;           // empty: the defaults (status 1, NaN)
            const float lmh = slots[j].lm_hi;
            const float lml = slots[j].lm_lo;
            const int nk = (n + 31) >> 5;
            if (j + 1 < kFitGroup && slots[j + 1].f >= 0) {
                // the group's next forest into L2 while this one is fitted
                const int64_t noff = slots[j + 1].off;
                const int nn = slots[j + 1].n < 32 * kContK ? slots[j + 1].n : 32 * kContK;
                for (int p = lane; p < nn; p += 32) {
                    prefetch_l2(sp.log_lambda + noff + p);
                    prefetch_l2(sp.flux + noff + p);
                    prefetch_l2(sp.ivar + noff + p);
                    prefetch_l2(sp.transmission_correction + noff + p);
                }
            }
            unsigned valid = 0;
            float sfi = 0.f, si = 0.f;
#pragma unroll 2
            for (int k = 0; k < nk; ++k) {
                float4 pa = make_float4(0.f, 0.f, 0.f, 1.f);
                float2 pb = make_float2(0.f, 0.f);
                const int p = lane + 32 * k;
                if (p < n) {
                    const float iv = f64_to_f32(sp.ivar[off + p]);
                    const float fl = f64_to_f32(sp.flux[off + p]);
                    sfi = fmaf(fl, iv, sfi);
                    si += iv;
                    if (iv > 0.f) {
                        const float2 ll = split_f64(sp.log_lambda[off + p]);
                        const float u = (ll.x - lmh) + (ll.y - lml);  // L - Lmin
                        pa.y = u * inv_span;
                        pa.x = fit_mean_cont(tab, u) * f64_to_f32(sp.transmission_correction[off + p]);
                        pa.z = fl;
                        if (!const_w) {
                            float eta, var_lss, fudge;
                            fit_var_funcs(tab, ll.x + ll.y, eta, var_lss, fudge);
                            pa.w = __fdividef(eta, fmaxf(iv, 1.17549435e-38f));
                            pb.x = var_lss;
                            pb.y = fudge * iv;
                        }
                        valid |= 1u << k;
                    }
                }
                px.a[k * 32 + lane] = pa;
                px.b[k * 32 + lane] = pb;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                sfi += __shfl_xor_sync(0xffffffffu, sfi, o);
                si += __shfl_xor_sync(0xffffffffu, si, o);
            }
            // starting point (utils.py:92): FP32 sums, only a start
            const float a0f = sfi / si;
            int nd = 0;
#pragma unroll 1
            for (int k = 0; k < nk; ++k) {
                if ((valid >> k) & 1u) {
                    const float4 pa = px.a[k * 32 + lane];
                    const float2 pb = px.b[k * 32 + lane];
                    const float c = a0f * pa.x;
                    const float c2 = c * c;
                    nd += fmaf(fmaf(pb.y, c2, pb.x), c2, pa.w) > 0.f ? 1 : 0;
                }
            }
            nd = __reduce_add_sync(0xffffffffu, nd);
            float ah = a0f, al = 0.f, bh = 0.f, bl = 0.f;
            if (start) {
                ah = slots[j].ah;
                al = slots[j].al;
                bh = slots[j].bh;
                bl = slots[j].bl;
            }
            float s[6];
            bool have_val = false;
            fit_terms(px, lane, nk, ah, bh, const_w, !evaluate_only, s);
            have_val = !evaluate_only;
            int it = 0;
            bool converged = evaluate_only;
            for (; it < max_iter; ++it) {
                // Newton step from the exact-product 2x2 solve
                float da, db;
                bool newton = true;  // d = -H^-1 g (not the gradient fallback)
                if (m.order == 0) {
                    newton = s[3] > 0.f;
                    da = newton ? -s[1] / s[3] : -s[1];
                    db = 0.f;
                } else {
                    const float det = diff_prod(s[3], s[5], s[4], s[4]);
                    da = db = 0.f;
                    if (det > 0.f && s[3] > 0.f) {
                        da = -diff_prod(s[5], s[1], s[4], s[2]) / det;
                        db = -diff_prod(s[3], s[2], s[4], s[1]) / det;
                    }
                    if ((da == 0.f && db == 0.f) || da * s[1] + db * s[2] >= 0.f) {
                        // singular Hessian or not a descent direction: gradient step
                        const float scale = fmaxf(fabsf(s[3]), fabsf(s[5]));
                        da = -s[1] / (scale > 0.f ? scale : 1.f);
                        db = -s[2] / (scale > 0.f ? scale : 1.f);
                        newton = false;
                    }
                }
                const float ref = fmaxf(1.f, fmaxf(fabsf(ah), fabsf(bh)));
                float t = 1.f;
                // a Newton step small enough that the point after it is within
                // cert_ab: take it; the final pass certifies the new point
                if (certify && newton && fabsf(da) <= sqrtf(cert_ab) * ref &&
                    fabsf(db) <= sqrtf(cert_ab) * ref) {
                    float hi = ah + da, bb = hi - ah;
                    al += (ah - (hi - bb)) + (da - bb);
                    ah = hi;
                    hi = bh + db;
                    bb = hi - bh;
                    bl += (bh - (hi - bb)) + (db - bb);
                    bh = hi;
                    converged = true;
                    ++it;
                    break;
                }
                float trial[6];
                if (fabsf(da) < 1e-3f * ref && fabsf(db) < 1e-3f * ref) {
                    fit_terms(px, lane, nk, ah + da, bh + db, const_w, false, trial);
                    have_val = false;
                } else {
                    if (!have_val) fit_terms(px, lane, nk, ah, bh, const_w, true, s);
                    const float slope_dir = da * s[1] + db * s[2];
                    bool accepted = false;
                    for (int ls = 0; ls < 40; ++ls) {
                        fit_terms(px, lane, nk, ah + t * da, bh + t * db, const_w, true, trial);
                        if (isfinite(trial[0]) && trial[0] <= s[0] + 1e-4f * t * slope_dir) {
                            accepted = true;
                            break;
                        }
                        t *= 0.5f;
                    }
                    if (!accepted) break;
                    have_val = true;
                }
                {
                    // (ah, al) += t da exactly to FP32-pair precision (TwoSum)
                    const float sa = t * da, sb = t * db;
                    float hi = ah + sa, bb = hi - ah;
                    al += (ah - (hi - bb)) + (sa - bb);
                    ah = hi;
                    hi = bh + sb;
                    bb = hi - bh;
                    bl += (bh - (hi - bb)) + (sb - bb);
                    bh = hi;
                }
#pragma unroll
                for (int k = 0; k < 6; ++k) s[k] = trial[k];
                const float ref2 = fmaxf(1.f, fmaxf(fabsf(ah), fabsf(bh)));
                if (!certify && fabsf(t * da) < eff_tol * ref2 && fabsf(t * db) < eff_tol * ref2) {
                    converged = true;
                    ++it;
                    break;
                }
            }
            // chi2 at the solution (compensated FP32 sums, lanes and warp),
            // the scale of the gradient's FP32 rounding (the per-pixel
            // roundings are independent, so it grows as the root of the sum
            // of squares of the per-pixel gradient terms), the gradient for
            // the certificate, and the continuum
            float cs = 0.f, ce = 0.f, ga_abs = 0.f, gb_abs = 0.f, ga_s = 0.f, gb_s = 0.f;
            bool negative = false, all_zero = true;
            const float af = ah, bf = bh;
#pragma unroll 1
            for (int k = 0; k < nk; ++k) {
                const int p = lane + 32 * k;
                if (p >= n) continue;
                float cont;
                if ((valid >> k) & 1u) {
                    const float4 pa = px.a[k * 32 + lane];
                    const float2 pb = px.b[k * 32 + lane];
                    const float c = pa.x * fmaf(bf, pa.y, af);
                    cont = c;
                    const float c2 = c * c;
                    const float t1 = fmaf(pb.y, c2, pb.x);
                    const float d = fmaf(t1, c2, pa.w);
                    const float r = pa.z - c;
                    const float id = 1.f / d;
                    const float rid = r * id;
                    const float dd = 2.f * c * fmaf(pb.y, c2, t1);
                    const float g = fabsf(2.f * rid) + rid * rid * fabsf(dd) + fabsf(dd * id);
                    const float jb = pa.y * pa.x;
                    ga_abs += (g * pa.x) * (g * pa.x);
                    gb_abs += (g * jb) * (g * jb);
                    if (certify) {
                        const float gs = fmaf(-rid, fmaf(rid, dd, 2.f), dd * id);
                        ga_s = fmaf(gs, pa.x, ga_s);
                        gb_s = fmaf(gs, jb, gb_s);
                    }
                    const float term = fmaf(r, rid, const_w ? 0.f : logf(d));
                    const float ns = cs + term;
                    const float bb = ns - cs;
                    ce += (cs - (ns - bb)) + (term - bb);
                    cs = ns;
                } else {
                    // masked pixel: the continuum only
                    const float2 ll = split_f64(sp.log_lambda[off + p]);
                    const float u = (ll.x - lmh) + (ll.y - lml);
                    const float mc = fit_mean_cont(tab, u) *
                                     f64_to_f32(sp.transmission_correction[off + p]);
                    cont = mc * fmaf(bf, u * inv_span, af);
                }
                if (out.continuum) out.continuum[off + p] = f32_to_f64(cont);
                negative |= cont < 0.f;
                all_zero &= cont == 0.f;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float os = __shfl_xor_sync(0xffffffffu, cs, o);
                const float oe = __shfl_xor_sync(0xffffffffu, ce, o);
                const float ns = cs + os;
                const float bb = ns - cs;
                ce += oe + ((cs - (ns - bb)) + (os - bb));
                cs = ns;
                ga_abs += __shfl_xor_sync(0xffffffffu, ga_abs, o);
                gb_abs += __shfl_xor_sync(0xffffffffu, gb_abs, o);
                if (certify) {
                    ga_s += __shfl_xor_sync(0xffffffffu, ga_s, o);
                    gb_s += __shfl_xor_sync(0xffffffffu, gb_s, o);
                }
            }
            negative = __any_sync(0xffffffffu, negative);
            all_zero = __all_sync(0xffffffffu, all_zero);
            const float ref = fmaxf(1.f, fmaxf(fabsf(ah), fabsf(bh)));
            if (certify) {
                // certificate at the accepted point, with the last Hessian
                bool cert = false;
                if (converged) {
                    float ra = 0.f, rb = 0.f;
                    bool ok_h;
                    if (m.order == 0) {
                        ok_h = s[3] > 0.f;
                        ra = ok_h ? -ga_s / s[3] : 0.f;
                    } else {
                        const float det = diff_prod(s[3], s[5], s[4], s[4]);
                        ok_h = det > 0.f && s[3] > 0.f;
                        if (ok_h) {
                            ra = -diff_prod(s[5], ga_s, s[4], gb_s) / det;
                            rb = -diff_prod(s[3], gb_s, s[4], ga_s) / det;
                        }
                    }
                    const float half_dec = -0.5f * (ra * ga_s + rb * gb_s);
                    cert = ok_h && fabsf(ra) <= cert_ab * ref && fabsf(rb) <= cert_ab * ref &&
                           half_dec <= cert_chi2 * fmaxf(fabsf(cs + ce), (float)nd);
                }
                converged = cert;
            }
            // estimate of the optimum's shift by that rounding, |H^-1| (8 u
            // rms(g)): large when the data barely separate a from b (a forest
            // covering a short stretch of the rest-frame window)
            bool refine = false;
            if (converged && !evaluate_only && !certify) {
                const float ua = 8.f * 5.96e-8f * sqrtf(ga_abs);
                const float ub = 8.f * 5.96e-8f * sqrtf(gb_abs);
                float ea, eb;
                if (m.order == 0) {
                    ea = s[3] > 0.f ? ua / s[3] : INFINITY;
                    eb = 0.f;
                } else {
                    const float det = diff_prod(s[3], s[5], s[4], s[4]);
                    ea = det > 0.f ? (fabsf(s[5]) * ua + fabsf(s[4]) * ub) / det : INFINITY;
                    eb = det > 0.f ? (fabsf(s[4]) * ua + fabsf(s[3]) * ub) / det : INFINITY;
                }
                refine = !(ea <= 2e-6f * ref && eb <= 2e-6f * ref);
            }
            if (lane == j) {
                int status = converged ? (refine ? 4 : 0) : 1;
                if (negative) status = 2;
                if (all_zero) status = 3;
                FitSlot &sl = slots[j];
                sl.status = status;
                sl.ah = ah; sl.al = al; sl.bh = bh; sl.bl = bl; sl.cs = cs; sl.ce = ce;
                sl.nd = nd;
                sl.it = it;
            }
        }
        __syncwarp();
        if (lane < kFitGroup && slots[lane].write) {
            const FitSlot sl = slots[lane];
            const bool keep = sl.status == 0 || sl.status == 4;
            out.zero_point[sl.f] = keep ? f32_to_f64(sl.ah) + f32_to_f64(sl.al) : NAN;
            out.slope[sl.f] = keep ? f32_to_f64(sl.bh) + f32_to_f64(sl.bl) : NAN;
            out.chi2[sl.f] = keep ? f32_to_f64(sl.cs) + f32_to_f64(sl.ce) : NAN;
            out.ndata[sl.f] = sl.nd;
            out.status[sl.f] = sl.status;
            out.iterations[sl.f] = sl.it;
        }
        __syncwarp();
    }
}

// find_bins_log / find_bins_lin (delta_extraction/utils.py:139-186): the
// nearest node of an evenly spaced grid in log10(lambda) (grid0, step in
// log10 Angstrom) or in lambda (grid0, step in Angstrom; the value's lambda is
// 10**x). The int conversion truncates toward zero, as astype(int64) does.
__device__ __forceinline__ int64_t find_bin(double x, double grid0, double step, int lin) {
    if (lin) return (int64_t)((pow(10.0, x) - grid0) / step + 0.5);
    return (int64_t)((x - grid0) / step + 0.5);
}

// eta, var_lss and fudge at v in FP64 from the model's coefficient arrays.
__device__ void var_funcs_f64(const pg_cont_model &m, double v, double &eta, double &vlss,
                              double &fudge) {
    const int mi = m.num_var_intervals, i = ppoly_piece(m.var_breaks, mi, v);
    const double dx = v - m.var_breaks[i];
    eta = ppoly_at(m.eta_coef, mi, i, dx);
    vlss = ppoly_at(m.var_lss_coef, mi, i, dx);
    fudge = ppoly_at(m.fudge_coef, mi, i, dx);
}

// ---- two-float (double-float) arithmetic -----------------------------------
// Values as unevaluated sums hi + lo of two floats (about 48 significant
// bits): the FP32 pipe stands in for the narrow FP64 pipe where FP32 alone
// would lose the reference's FP64 accuracy.
struct dfl {
    float hi, lo;
};

__device__ __forceinline__ dfl dfl_fast(float a, float b) {  // |a| >= |b|
    const float s = a + b;
    return {s, b - (s - a)};
}

__device__ __forceinline__ dfl dfl_of(double v) {
    const float2 p = split_f64(v);
    return dfl_fast(p.x, p.y);
}

__device__ __forceinline__ dfl dfl_two_sum(float a, float b) {
    const float s = a + b;
    const float bb = s - a;
    return {s, (a - (s - bb)) + (b - bb)};
}

__device__ __forceinline__ dfl dfl_add(dfl x, dfl y) {
    dfl s = dfl_two_sum(x.hi, y.hi);
    const dfl t = dfl_two_sum(x.lo, y.lo);
    s.lo += t.hi;
    s = dfl_fast(s.hi, s.lo);
    s.lo += t.lo;
    return dfl_fast(s.hi, s.lo);
}

__device__ __forceinline__ dfl dfl_mul(dfl x, dfl y) {
    const float p = x.hi * y.hi;
    float e = fmaf(x.hi, y.hi, -p);
    e = fmaf(x.hi, y.lo, fmaf(x.lo, y.hi, e));
    return dfl_fast(p, e);
}

// x / y: a quotient estimate corrected once with the exact residual
__device__ __forceinline__ dfl dfl_div(dfl x, dfl y) {
    const float q1 = __fdividef(x.hi, y.hi);
    const float p = q1 * y.hi;
    const float pe = fmaf(q1, y.hi, -p);
    // r = x - q1 y, from the exact product p + pe (+ q1 y.lo)
    const dfl r = dfl_add(x, dfl{-p, -fmaf(q1, y.lo, pe)});
    const float q2 = __fdividef(r.hi, y.hi);
    return dfl_fast(q1, q2);
}

__device__ __forceinline__ double dfl_to_f64(dfl x) { return f32_to_f64(x.hi) + f32_to_f64(x.lo); }

// hi/lo histogram bin += x: FP32 atomic adds whose rounding error is
// recovered exactly from the value each one replaced (TwoSum against the
// returned old value) and added to the low word with the low part of x
__device__ __forceinline__ void hist_add(float *hi, float *lo, int bin, dfl x) {
    const float old = atomicAdd(&hi[bin], x.hi);
    const float s = old + x.hi;
    const float bb = s - old;
    const float err = (old - (s - bb)) + (x.hi - bb);
    atomicAdd(&lo[bin], err + x.lo);
}

// trunc(t) of a bin coordinate t evaluated in FP32 with absolute error
// below guard: certain when t is farther than guard from an integer
__device__ __forceinline__ bool bin_certain(float t, float guard, int &bin) {
    const float a = fabsf(t);
    const float fr = a - truncf(a);
    bin = __float2int_rz(t);  // toward zero, as astype(int64)
    return a < 1.0e6f && fr > guard && fr < 1.f - guard;
}

// ---- two-float finish of the mixed fit ------------------------------------
// The forests the mixed fit flagged (status 4: FP32 rounding could move their
// optimum by more than 2e-6 of max(1, |a|, |b|), a short stretch of the
// rest-frame window barely separating a from b) are finished here, in the
// same call, to FP64 accuracy without the FP64 pipe: every per-pixel input
// (x, the mean continuum, the variance functions) is formed in two-float
// arithmetic from the FP64 model, the gradient of chi2 is summed in
// two-float, and Newton steps from the mixed solution (the Hessian in FP32
// is enough for a correction step) run until the step is below 1e-11 of
// max(1, |a|, |b|). chi2 is re-evaluated with the logarithm in FP32 plus its
// first-order two-float correction.
constexpr int kRefineWarps = 4;
constexpr size_t kRefineSlabBytes = (size_t)kContK * 32 * 3 * sizeof(float4);

__host__ __device__ inline size_t refine_smem_bytes(int nmc, int m) {
    return (size_t)kRefineWarps * kRefineSlabBytes + (size_t)3 * nmc * 8 + (size_t)(m + 1) * 8 +
           (size_t)12 * m * 8 + 16;
}

// sign of x - y (two-float values)
__device__ __forceinline__ bool dfl_less(dfl x, dfl y) {
    return (x.hi - y.hi) + (x.lo - y.lo) < 0.f;
}

__device__ __forceinline__ dfl dfl_neg(dfl x) { return {-x.hi, -x.lo}; }

__device__ __forceinline__ dfl warp_sum_dfl(dfl v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const dfl w = {__shfl_xor_sync(0xffffffffu, v.hi, o), __shfl_xor_sync(0xffffffffu, v.lo, o)};
        v = dfl_add(v, w);
    }
    return v;
}

__global__ void __launch_bounds__(32 * kRefineWarps) cont_fit_refine_kernel(
    const __grid_constant__ pg_spectra sp, const __grid_constant__ pg_cont_model m,
    const int32_t *__restrict__ index, int64_t count, const __grid_constant__ pg_cont_fit out,
    Scratch *scratch) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31;
    const int nmc = m.num_mean_cont;
    const int mi = m.use_constant_weight ? 0 : m.num_var_intervals;
    const bool const_w = mi == 0;
    float4 *slab = reinterpret_cast<float4 *>(smem + kRefineSlabBytes * (threadIdx.x >> 5));
    dfl *node = reinterpret_cast<dfl *>(smem + kRefineSlabBytes * kRefineWarps);  // off, y, slope
    dfl *brk = node + 3 * nmc;
    dfl *coef = brk + (mi + 1);  // [i][12]: eta, var_lss, fudge (c3 c2 c1 c0)
    const double rest_min = m.log_lambda_rest_min;
    for (int i = threadIdx.x; i < nmc; i += blockDim.x) {
        const double x = m.mean_cont_x[i], y = m.mean_cont_y[i];
        node[3 * i] = dfl_of(x - rest_min);
        node[3 * i + 1] = dfl_of(y);
        node[3 * i + 2] = dfl_of(i + 1 < nmc ? (m.mean_cont_y[i + 1] - y) / (m.mean_cont_x[i + 1] - x)
                                             : 0.);
    }
    for (int i = threadIdx.x; i <= mi; i += blockDim.x) brk[i] = dfl_of(m.var_breaks[i]);
    for (int i = threadIdx.x; i < mi; i += blockDim.x) {
        for (int k = 0; k < 4; ++k) {
            coef[12 * i + k] = dfl_of(m.eta_coef[k * mi + i]);
            coef[12 * i + 4 + k] = dfl_of(m.var_lss_coef[k * mi + i]);
            coef[12 * i + 8 + k] = dfl_of(m.fudge_coef[k * mi + i]);
        }
    }
    __syncthreads();
    const dfl inv_span = dfl_of(1.0 / (m.log_lambda_rest_max - m.log_lambda_rest_min));
    const int64_t warp_global = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t base = warp_global * 32; base < count; base += nwarps * 32) {
        int64_t lane_f = -1;
        bool flagged = false;
        double lane_lmin = 0.;
        if (base + lane < count) {
            lane_f = index ? (int64_t)index[base + lane] : base + lane;
            flagged = out.status[lane_f] == 4;
            if (flagged) lane_lmin = rest_min + log10(1. + sp.z_qso[lane_f]);
        }
        unsigned todo = __ballot_sync(0xffffffffu, flagged);
        while (todo) {
            const int src = __ffs(todo) - 1;
            todo &= todo - 1;
            const int64_t f = __shfl_sync(0xffffffffu, lane_f, src);
            const dfl lmin = dfl_of(__shfl_sync(0xffffffffu, lane_lmin, src));
            const int64_t off = sp.pix_offset[f];
            const int n = (int)(sp.pix_offset[f + 1] - off);
            const int nk = (n + 31) >> 5;
            // two-float pixel terms: slab[3 (k 32 + lane) + {0, 1, 2}] =
            // (mc, x), (f, q), (vl, fi), each as hi, lo
            unsigned valid = 0;
            for (int k = 0; k < nk; ++k) {
                const int p = lane + 32 * k;
                dfl mc = {0.f, 0.f}, x = {0.f, 0.f}, fl = {0.f, 0.f}, q = {1.f, 0.f};
                dfl vl = {0.f, 0.f}, fi = {0.f, 0.f};
                if (p < n) {
                    const dfl L = dfl_of(sp.log_lambda[off + p]);
                    const dfl u = dfl_add(L, dfl_neg(lmin));  // L - Lmin
                    x = dfl_mul(u, inv_span);
                    int lo = 0, hi = nmc;
                    while (lo < hi) {
                        const int mid = (lo + hi) >> 1;
                        if (dfl_less(node[3 * mid], u)) lo = mid + 1;
                        else hi = mid;
                    }
                    const int i = lo < 1 ? 0 : (lo > nmc - 1 ? nmc - 2 : lo - 1);
                    mc = dfl_add(node[3 * i + 1],
                                 dfl_mul(node[3 * i + 2], dfl_add(u, dfl_neg(node[3 * i]))));
                    mc = dfl_mul(mc, dfl_of(sp.transmission_correction[off + p]));
                    const dfl iv = dfl_of(sp.ivar[off + p]);
                    if (iv.hi > 0.f) {
                        fl = dfl_of(sp.flux[off + p]);
                        if (!const_w) {
                            int a = 0, b = mi + 1;
                            while (a < b) {
                                const int mid = (a + b) >> 1;
                                if (!dfl_less(L, brk[mid])) a = mid + 1;
                                else b = mid;
                            }
                            int j = a - 1;
                            j = j < 0 ? 0 : (j > mi - 1 ? mi - 1 : j);
                            const dfl dx = dfl_add(L, dfl_neg(brk[j]));
                            dfl v3[3];
#pragma unroll
                            for (int g = 0; g < 3; ++g) {
                                const dfl *c = coef + 12 * j + 4 * g;
                                dfl acc = c[0];
                                acc = dfl_add(dfl_mul(acc, dx), c[1]);
                                acc = dfl_add(dfl_mul(acc, dx), c[2]);
                                v3[g] = dfl_add(dfl_mul(acc, dx), c[3]);
                            }
                            q = dfl_div(v3[0], iv);
                            vl = v3[1];
                            fi = dfl_mul(v3[2], iv);
                        }
                        valid |= 1u << k;
                    }
                }
                float4 *e = slab + 3 * (k * 32 + lane);
                e[0] = make_float4(mc.hi, mc.lo, x.hi, x.lo);
                e[1] = make_float4(fl.hi, fl.lo, q.hi, q.lo);
                e[2] = make_float4(vl.hi, vl.lo, fi.hi, fi.lo);
            }
            dfl a = dfl_of(out.zero_point[f]);
            dfl b = m.order == 0 ? dfl{0.f, 0.f} : dfl_of(out.slope[f]);
            int it = 0;
            bool converged = false;
            float h3 = 0.f, h4 = 0.f, h5 = 0.f;
            for (; it < 10; ++it) {
                // gradient (two-float) and Hessian (FP32) at (a, b)
                dfl ga = {0.f, 0.f}, gb = {0.f, 0.f};
                float haa = 0.f, hab = 0.f, hbb = 0.f;
                for (int k = 0; k < nk; ++k) {
                    if (!((valid >> k) & 1u)) continue;
                    const float4 *e = slab + 3 * (k * 32 + lane);
                    const float4 e0 = e[0], e1 = e[1], e2 = e[2];
                    const dfl mc = {e0.x, e0.y}, x = {e0.z, e0.w}, fl = {e1.x, e1.y};
                    const dfl q = {e1.z, e1.w}, vl = {e2.x, e2.y}, fi = {e2.z, e2.w};
                    const dfl c = dfl_mul(mc, dfl_add(a, dfl_mul(b, x)));
                    const dfl c2 = dfl_mul(c, c);
                    const dfl fc2 = dfl_mul(fi, c2);
                    const dfl t1 = dfl_add(vl, fc2);
                    const dfl d = dfl_add(q, dfl_mul(t1, c2));
                    const dfl hd = dfl_mul(c, dfl_add(t1, fc2));
                    const dfl r = dfl_add(fl, dfl_neg(c));
                    const dfl id = dfl_div(dfl{1.f, 0.f}, d);
                    const dfl rid = dfl_mul(r, id);
                    const dfl e_ = dfl_mul(hd, id);
                    const dfl w1 = dfl_add(dfl{1.f, 0.f}, dfl_mul(rid, hd));
                    const dfl g = dfl_add(e_, dfl_neg(dfl_mul(rid, w1)));
                    const dfl gj = dfl_mul(g, mc);
                    ga = dfl_add(ga, gj);
                    gb = dfl_add(gb, dfl_mul(gj, x));
                    // Hessian from the leading parts
                    const float h2 = fmaf(5.f * fi.hi, c2.hi, t1.hi);
                    const float hh = fmaf(h2, fmaf(-rid.hi, rid.hi, id.hi), id.hi) +
                                     e_.hi * fmaf(4.f * rid.hi, w1.hi, -2.f * e_.hi);
                    const float hj = hh * mc.hi * mc.hi;
                    haa += hj;
                    hab = fmaf(hj, x.hi, hab);
                    hbb = fmaf(hj * x.hi, x.hi, hbb);
                }
                ga = warp_sum_dfl(ga);
                gb = warp_sum_dfl(gb);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    haa += __shfl_xor_sync(0xffffffffu, haa, o);
                    hab += __shfl_xor_sync(0xffffffffu, hab, o);
                    hbb += __shfl_xor_sync(0xffffffffu, hbb, o);
                }
                // half-derivatives: the factors 2 cancel in the Newton step
                h3 = 2.f * haa;
                h4 = 2.f * hab;
                h5 = 2.f * hbb;
                const float g1 = 2.f * (ga.hi + ga.lo), g2 = 2.f * (gb.hi + gb.lo);
                float da, db;
                if (m.order == 0) {
                    if (!(h3 > 0.f)) break;
                    da = -g1 / h3;
                    db = 0.f;
                } else {
                    const float det = diff_prod(h3, h5, h4, h4);
                    if (!(det > 0.f && h3 > 0.f)) break;
                    da = -diff_prod(h5, g1, h4, g2) / det;
                    db = -diff_prod(h3, g2, h4, g1) / det;
                }
                if (!isfinite(da) || !isfinite(db)) break;
                a = dfl_add(a, dfl{da, 0.f});
                b = dfl_add(b, dfl{db, 0.f});
                const float ref = fmaxf(1.f, fmaxf(fabsf(a.hi), fabsf(b.hi)));
                if (fabsf(da) <= 1e-11f * ref && fabsf(db) <= 1e-11f * ref) {
                    converged = true;
                    ++it;
                    break;
                }
            }
            // chi2 and the continuum at the solution
            dfl chi = {0.f, 0.f};
            bool negative = false, all_zero = true;
            for (int k = 0; k < nk; ++k) {
                const int p = lane + 32 * k;
                if (p >= n) continue;
                const float4 *e = slab + 3 * (k * 32 + lane);
                const float4 e0 = e[0];
                const dfl mc = {e0.x, e0.y}, x = {e0.z, e0.w};
                const dfl c = dfl_mul(mc, dfl_add(a, dfl_mul(b, x)));
                if ((valid >> k) & 1u) {
                    const float4 e1 = e[1], e2 = e[2];
                    const dfl fl = {e1.x, e1.y}, q = {e1.z, e1.w};
                    const dfl vl = {e2.x, e2.y}, fi = {e2.z, e2.w};
                    const dfl c2 = dfl_mul(c, c);
                    const dfl d = dfl_add(q, dfl_mul(dfl_add(vl, dfl_mul(fi, c2)), c2));
                    const dfl r = dfl_add(fl, dfl_neg(c));
                    const dfl term = dfl_div(dfl_mul(r, r), d);
                    chi = dfl_add(chi, term);
                    if (!const_w) chi = dfl_add(chi, dfl_fast(logf(d.hi), d.lo / d.hi));
                }
                if (out.continuum) out.continuum[off + p] = dfl_to_f64(c);
                negative |= c.hi < 0.f;
                all_zero &= c.hi == 0.f;
            }
            chi = warp_sum_dfl(chi);
            negative = __any_sync(0xffffffffu, negative);
            all_zero = __all_sync(0xffffffffu, all_zero);
            if (lane == 0) {
                int status = converged ? 0 : 1;
                if (negative) status = 2;
                if (all_zero) status = 3;
                const bool keep = status == 0;
                out.zero_point[f] = keep ? dfl_to_f64(a) : NAN;
                out.slope[f] = keep ? dfl_to_f64(b) : NAN;
                out.chi2[f] = keep ? dfl_to_f64(chi) : NAN;
                out.status[f] = status;
                out.iterations[f] += it;
                atomicAdd(&scratch->work_items, 1ull);
            }
        }
    }
}

// Histograms of one Dr16 iteration. Persistent blocks (one warp per forest,
// pixels across lanes, forests drawn kStackGroup at a time from the work
// counter) accumulate the rest-frame mean continuum, the observed-frame stack
// and the variance statistics in shared memory and add them to the global
// FP64 sums once at the end: 400k forests add to a few thousand bins.
//
// GB300's FP64 pipe is 1/64 of its FP32 pipe, so the per-pixel arithmetic is
// two-float: the FP64 inputs are split on the integer pipe, the weights,
// flux ratios and delta moments are formed with FP32 error-free
// transformations (relative error about 1e-13, against the 1e-16 of the
// reference's FP64), and the histograms are hi/lo pairs of FP32 words. Bin
// indices are evaluated in FP32 and used where they are certain (farther
// than a guard from a bin edge); the few pixels within the guard take the
// reference's FP64 formula. The variance functions are tabulated (FP64,
// stored as two floats) on the observed-frame grid and read for pixels on a
// grid node (all of them for forests rebinned to the grid); others evaluate
// them in FP64.
//
// EXACT: the histograms are 128-bit fixed-point numbers (four 32-bit words, the
// last place 2^-kFixScale) instead of hi/lo pairs, in shared memory and across
// the blocks, so that a sum does not depend on the order of its terms: the
// same inputs give the same bits. With pairs the model of the next iteration
// moved by its last bits from run to run, and the FP32 decisions of the mixed
// fit on it moved single forests by up to 1e-6. Two more numbers of a bin in
// global memory, with other last places, take the terms of 2^kFineTop and more
// and what terms below 2^kFineLow have under the first one's last place, so that
// every sum keeps the 2^-50 of its terms; terms of 2^kCoarseTop and more, below
// 2^-78, or none go straight to the FP64 result. Calls whose words do not fit in shared memory keep the pairs. 1,024
// threads (a block an SM; 512 leave the chains of word adds less to overlap
// with). Five passes over 40,000 forests of 160 pixels: 1.45 ms in pairs, 1.57 ms
// exact (1.60 where the blocks end on carries in global memory, 1.95 in blocks of 512).
constexpr int kStackBlock = 512;
constexpr int kStackGroup = 8;
// 2^25 terms at the top of each range stay below 2^(127 - scale)
constexpr int kFixScale = 88, kFineLow = -39, kFineTop = 14;
constexpr int kCoarseScale = 56, kCoarseTop = 46;
constexpr int kSmallScale = 168;  // parts below 2^-kFixScale
constexpr int kStackNumbers = 3;  // of a cell in global memory

struct StackSlot {
    int64_t off;
    int n, skip;
    double zp1;
    float zr_hi, zr_lo;  // log10(1 + z) + rest grid start (log grid) or log10(1 + z) (linear)
};

// The size limit of a call (all histograms as hi/lo pairs).
__host__ __device__ inline size_t stack_smem_bytes(const pg_cont_stacks &st, bool table) {
    const size_t nvar = (size_t)st.var_lambda_bins * kVarBins;
    return (size_t)8 * (2 * st.rest_bins + 2 * st.obs_bins + 3 * nvar) + (size_t)8 * nvar +
           (table ? (size_t)32 * st.obs_bins : 0) + 64;
}

// The wanted histograms as one array of cells, a word of a cell per plane (hi
// and lo, or four words); then the counts of the variance bins.
struct StackCells {
    int mc_num, mc_w, s_num, s_w, v_mean, v_d2, v_d4, total, nvar;
};

__host__ __device__ inline StackCells stack_cells(const pg_cont_stacks &st) {
    StackCells c;
    const int r = st.mean_cont_num ? st.rest_bins : 0, o = st.stack_num ? st.obs_bins : 0;
    c.nvar = st.var_mean ? st.var_lambda_bins * kVarBins : 0;
    c.mc_num = 0;
    c.mc_w = r;
    c.s_num = 2 * r;
    c.s_w = c.s_num + o;
    c.v_mean = c.s_num + 2 * o;
    c.v_d2 = c.v_mean + c.nvar;
    c.v_d4 = c.v_d2 + c.nvar;
    c.total = c.v_d4 + c.nvar;
    return c;
}

__host__ __device__ inline size_t stack_bytes(const pg_cont_stacks &st, bool exact, bool table) {
    const StackCells c = stack_cells(st);
    return (size_t)(exact ? 16 : 8) * c.total + (size_t)8 * c.nvar +
           (table ? (size_t)32 * st.obs_bins : 0) + 64;
}

// Adds the N two's complement numbers word[n][0..3] to the four words at
// h[n], h[n] + stride, ...: the carry out of a word is seen by the add that
// causes it. Word by word, so that the N round trips overlap.
template <int N>
__device__ __forceinline__ void fix_add_words(uint32_t *const h[N], int stride,
                                              const uint32_t word[N][4]) {
    uint32_t carry[N];
#pragma unroll
    for (int n = 0; n < N; ++n) carry[n] = 0u;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        uint32_t x[N], old[N];
#pragma unroll
        for (int n = 0; n < N; ++n) {
            x[n] = word[n][k] + carry[n];
            carry[n] = x[n] < carry[n] ? 1u : 0u;  // word + carry was 2^32: nothing to add
            if (x[n]) old[n] = atomicAdd(h[n] + k * stride, x[n]);
        }
#pragma unroll
        for (int n = 0; n < N; ++n)
            if (x[n]) carry[n] |= old[n] + x[n] < x[n] ? 1u : 0u;
    }
}

// Adds a number to one in global memory: three 64-bit counters (at sum, sum +
// stride, ...) take word 0, word 1 and the upper half, so that no carry is waited
// for (up to 2^32 numbers).
__device__ __forceinline__ void fix_add_global(unsigned long long *sum, int stride,
                                               const uint32_t word[4]) {
    const unsigned long long upper = (unsigned long long)word[3] << 32 | word[2];
    if (word[0]) atomicAdd(sum, (unsigned long long)word[0]);
    if (word[1]) atomicAdd(sum + stride, (unsigned long long)word[1]);
    if (upper) atomicAdd(sum + 2 * stride, upper);
}

// t 2^p as four words, |t| < 2^51, 0 <= p < 64 (WIDE: 96).
template <bool WIDE>
__device__ __forceinline__ void fix_words(long long t, int p, uint32_t word[4]) {
    const uint32_t lo = (uint32_t)t, hi = (uint32_t)((unsigned long long)t >> 32);
    const uint32_t sign = (uint32_t)((int)hi >> 31);
    const uint32_t a = lo << (p & 31);  // the shifts go by the low five bits of p
    const uint32_t b = __funnelshift_l(lo, hi, p), c = __funnelshift_l(hi, sign, p);
    const bool up = p >= 32, upper = WIDE && p >= 64;
    word[0] = up ? 0u : a;
    word[1] = upper ? 0u : (up ? a : b);
    word[2] = upper ? a : (up ? b : c);
    word[3] = upper ? b : (up ? c : sign);
}

// v = t 2^(e - 176) to 2^-50 of it, the last place of v.hi at bit 26 of t (e:
// exponent of v.hi, 49 to 254).
__device__ __forceinline__ long long fix_digits(dfl v, int e) {
    const uint32_t u = __float_as_uint(v.hi);
    const int m = (int)((u & 0x7FFFFFu) | 0x800000u);
    const float lo = v.lo * __uint_as_float((uint32_t)(303 - e) << 23);
    return (long long)((int)u < 0 ? -m : m) * (1 << 26) + __float2int_rn(lo);
}

// The number in three counters, in units of 2^-scale.
__device__ __forceinline__ double fix_value(const unsigned long long sum[3], int scale) {
    const unsigned long long s1 = sum[1] + (sum[0] >> 32);
    unsigned long long hi = sum[2] + (s1 >> 32);
    unsigned long long lo = (s1 << 32) | (sum[0] & 0xFFFFFFFFull);
    const bool negative = (long long)hi < 0;
    if (negative) {
        lo = 0ull - lo;
        hi = ~hi + (lo == 0ull ? 1ull : 0ull);
    }
    const double v = ldexp((double)hi, 64 - scale) + ldexp((double)lo, -scale);
    return negative ? -v : v;
}

// The terms that the fine number alone does not hold: of 2^kFineTop or more to
// the bin's coarse number; below 2^kFineLow the part in units of 2^-kFixScale to
// the fine number (of the block, at fine) and what is left of it to the small
// number; infinities, NaN and what no number holds to the FP64 result.
__device__ __noinline__ void stack_add_rare(uint32_t *fine, unsigned long long *work, int nc,
                                            int cell, double *dst, dfl v) {
    const int e = (int)((__float_as_uint(v.hi) >> 23) & 0xFFu);
    uint32_t word[1][4];
    if (e >= 127 + kCoarseTop || e < 127 - 78) {
        atomicAdd(dst, (double)v.hi + (double)v.lo);
        return;
    }
    const long long t = fix_digits(v, e);
    if (e >= 127 + kFineTop) {
        fix_words<false>(t, e - 176 + kCoarseScale, word[0]);
        fix_add_global(work + 3 * nc + cell, nc, word[0]);
        return;
    }
    const int below = 176 - kFixScale - e;  // bits of t below the fine number's last place
    const long long whole = t >> below;
    uint32_t *at_fine[1] = {fine};
    fix_words<false>(whole, 0, word[0]);
    fix_add_words<1>(at_fine, nc, word);
    fix_words<true>(t - whole * (1LL << below), e - 176 + kSmallScale, word[0]);
    fix_add_global(work + 6 * nc + cell, nc, word[0]);
}

// exact_work (EXACT): kStackNumbers x 3 counters of every cell, zeroed: the
// blocks' sums, the terms of 2^kFineTop and more, the parts below 2^-kFixScale.
template <bool EXACT, int BLOCK>
__global__ void __launch_bounds__(BLOCK) cont_stacks_kernel(
    const __grid_constant__ pg_spectra sp, const __grid_constant__ pg_cont_model m,
    const __grid_constant__ pg_cont_fit fit, const __grid_constant__ pg_cont_stacks st,
    Scratch *scratch, int use_table, unsigned long long *exact_work) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ uint32_t seen[BLOCK / 32][64];  // per-warp bitmap of var bins (<= 2048)
    __shared__ StackSlot s_slots[BLOCK / 32][kStackGroup];
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    const StackCells cells = stack_cells(st);
    const int nvar = cells.nvar, nc = cells.total;
    const int mi = m.use_constant_weight ? 0 : m.num_var_intervals;
    const int R = st.rest_bins, O = st.obs_bins;
    // layout: table (float4 x 2 per obs bin), then the histograms, then counts
    float4 *table = reinterpret_cast<float4 *>(smem_raw);
    uint32_t *hist =
        reinterpret_cast<uint32_t *>(smem_raw + (use_table ? (size_t)32 * O : 0));
    constexpr int kPlanes = EXACT ? 4 : 2;
    uint32_t *v_np = hist + kPlanes * nc, *v_nq = v_np + nvar;
    const int nwords = kPlanes * nc + 2 * nvar;
    for (int k = threadIdx.x; k < nwords; k += blockDim.x) hist[k] = 0u;
    // N terms v to the cells, whose FP64 results are at dst
    auto add = [&](auto count, const int *cell, double *const *dst, const dfl *v) {
        constexpr int N = decltype(count)::value;
        if (!EXACT) {
            float *h = reinterpret_cast<float *>(hist);
#pragma unroll
            for (int n = 0; n < N; ++n) hist_add(h, h + nc, cell[n], v[n]);
            return;
        }
        uint32_t *at[N], word[N][4];
#pragma unroll
        for (int n = 0; n < N; ++n) {
            const int e = (int)((__float_as_uint(v[n].hi) >> 23) & 0xFFu);
            const bool fine = e >= 127 + kFineLow && e < 127 + kFineTop;
            at[n] = hist + cell[n];
            fix_words<false>(fine ? fix_digits(v[n], e) : 0, fine ? e - 176 + kFixScale : 0,
                             word[n]);
            if (!fine && v[n].hi != 0.f)
                stack_add_rare(hist + cell[n], exact_work, nc, cell[n], dst[n], v[n]);
        }
        fix_add_words<N>(at, nc, word);
    };
    if (use_table) {
        // variance functions on the observed-frame grid nodes
        for (int j = threadIdx.x; j < O; j += blockDim.x) {
            const double g = st.obs_grid0 + j * st.obs_step;
            const double node = st.wave_lin ? log10(g) : g;
            double eta, vlss, fudge;
            var_funcs_f64(m, node, eta, vlss, fudge);
            const dfl n = dfl_of(node), e = dfl_of(eta), v = dfl_of(vlss), f = dfl_of(fudge);
            table[2 * j] = make_float4(n.hi, n.lo, e.hi, e.lo);
            table[2 * j + 1] = make_float4(v.hi, v.lo, f.hi, f.lo);
        }
    }
    __syncthreads();
    const bool do_mc = st.mean_cont_num != nullptr;
    const bool do_stack = st.stack_num != nullptr;
    const bool do_var = st.var_mean != nullptr && nvar <= 2048;
    const bool lin = st.wave_lin != 0;
    const double mod64 = m.var_lss_mod;
    const dfl mod = dfl_of(mod64);
    const dfl obs0 = dfl_of(lin ? st.obs_grid0 : st.obs_grid0);
    const dfl var0 = dfl_of(st.var_grid0);
    const float inv_obs = (float)(1.0 / st.obs_step), inv_rest = (float)(1.0 / st.rest_step);
    const float inv_var = (float)(1.0 / st.var_step);
    const float guard = lin ? 5e-3f : 1e-3f;
    constexpr float kLn10 = 2.302585093f;
    const int64_t num_groups = (sp.num + kStackGroup - 1) / kStackGroup;
    StackSlot *slots = s_slots[wib];
    for (;;) {
        int64_t group = 0;
        if (lane == 0) group = atomicAdd(&scratch->work_counter, 1);
        group = __shfl_sync(0xffffffffu, group, 0);
        if (group >= num_groups) break;
        if (lane < kStackGroup) {
            StackSlot sl;
            const int64_t f = group * kStackGroup + lane;
            sl.skip = 1;
            sl.off = 0;
            sl.n = 0;
            sl.zp1 = 0.;
            sl.zr_hi = sl.zr_lo = 0.f;
            if (f < sp.num && fit.status[f] == 0) {
                sl.skip = 0;
                sl.off = sp.pix_offset[f];
                sl.n = (int)(sp.pix_offset[f + 1] - sl.off);
                sl.zp1 = log10(1 + sp.z_qso[f]);
                const dfl zr = dfl_of(lin ? sl.zp1 : sl.zp1 + st.rest_grid0);
                sl.zr_hi = zr.hi;
                sl.zr_lo = zr.lo;
            }
            slots[lane] = sl;
        }
        __syncwarp();
        for (int jf = 0; jf < kStackGroup; ++jf) {
            if (slots[jf].skip) continue;
            const int64_t off = slots[jf].off;
            const int n = slots[jf].n;
            const double zp1 = slots[jf].zp1;
            const dfl zr = {slots[jf].zr_hi, slots[jf].zr_lo};
            if (do_var) {
                for (int k = lane; k < 64; k += 32) seen[wib][k] = 0u;
                __syncwarp();
            }
            for (int p = lane; p < n; p += 32) {
                const double ll = sp.log_lambda[off + p];
                const double iv64 = sp.ivar[off + p];
                const dfl L = dfl_of(ll), F = dfl_of(sp.flux[off + p]);
                const dfl C = dfl_of(fit.continuum[off + p]);
                const dfl IV = dfl_of(iv64);
                const bool has_iv = IV.hi > 0.f;
                // observed-frame bin (stack, variance-function table)
                int jobs = -1;
                if (do_stack || use_table) {
                    float t;
                    if (lin) {
                        const float lam = exp10f(L.hi) * fmaf(L.lo, kLn10, 1.f);
                        t = fmaf(lam - (float)st.obs_grid0, inv_obs, 0.5f);
                    } else {
                        t = fmaf((L.hi - obs0.hi) + (L.lo - obs0.lo), inv_obs, 0.5f);
                    }
                    if (!bin_certain(t, guard, jobs))
                        jobs = (int)find_bin(ll, st.obs_grid0, st.obs_step, st.wave_lin);
                }
                // X = ivar C^2 and var_pipe = 1 / X
                dfl X = {0.f, 0.f}, vp = {0.f, 0.f}, Q = {0.f, 0.f};
                if (has_iv) {
                    X = dfl_mul(IV, dfl_mul(C, C));
                    vp = dfl_div(dfl{1.f, 0.f}, X);
                    Q = dfl_div(F, C);
                }
                if (do_mc || do_stack) {
                    // compute_forest_weights (dr16_expected_flux.py:466-488)
                    dfl w = {0.f, 0.f};
                    if (has_iv) {
                        dfl eta = {0.f, 0.f}, vlss = {1.f, 0.f}, fudge = {0.f, 0.f};
                        if (mi > 0) {
                            bool done = false;
                            if (use_table && jobs >= 0 && jobs < O) {
                                const float4 t0 = table[2 * jobs];
                                if (fabsf((L.hi - t0.x) + (L.lo - t0.y)) <= 1e-12f) {
                                    const float4 t1 = table[2 * jobs + 1];
                                    eta = dfl{t0.z, t0.w};
                                    vlss = dfl{t1.x, t1.y};
                                    fudge = dfl{t1.z, t1.w};
                                    done = true;
                                }
                            }
                            if (!done) {
                                double e, v, f;
                                var_funcs_f64(m, ll, e, v, f);
                                eta = dfl_of(e);
                                vlss = dfl_of(v);
                                fudge = dfl_of(f);
                            }
                        }
                        const dfl den = dfl_add(dfl_add(dfl_mul(eta, vp), dfl_mul(mod, vlss)),
                                                dfl_mul(fudge, X));
                        w = dfl_div(dfl{1.f, 0.f}, den);
                    }
                    if (do_mc) {
                        // _compute_mean_cont: (f / (C + 1e-16)) * w binned in the rest frame
                        float t;
                        if (lin) {
                            const dfl x = dfl_add(L, dfl{-zr.hi, -zr.lo});
                            const float lam = exp10f(x.hi) * fmaf(x.lo, kLn10, 1.f);
                            t = fmaf(lam - (float)st.rest_grid0, inv_rest, 0.5f);
                        } else {
                            t = fmaf((L.hi - zr.hi) + (L.lo - zr.lo), inv_rest, 0.5f);
                        }
                        int bin;
                        if (!bin_certain(t, guard, bin))
                            bin = (int)find_bin(ll - zp1, st.rest_grid0, st.rest_step, st.wave_lin);
                        if (bin >= 0 && bin < R) {
                            if (has_iv) {
                                dfl ratio = Q;
                                if (!(fabsf(C.hi) > 1e-4f)) {
                                    // the 1e-16 offset matters: the reference's formula
                                    const double c64 = fit.continuum[off + p];
                                    ratio = dfl_of(sp.flux[off + p] / (c64 + 1e-16));
                                }
                                const int cell[] = {cells.mc_num + bin, cells.mc_w + bin};
                                double *const dst[] = {st.mean_cont_num + bin,
                                                       st.mean_cont_weight + bin};
                                const dfl v[] = {dfl_mul(ratio, w), w};
                                add(std::integral_constant<int, 2>{}, cell, dst, v);
                            }
                        } else {
                            report_error(scratch, PG_ERR_BIN_RANGE, bin);
                        }
                    }
                    if (do_stack) {
                        // compute_delta_stack: delta = f / C where ivar > 0
                        if (jobs >= 0 && jobs < O) {
                            if (has_iv) {
                                const int cell[] = {cells.s_num + jobs, cells.s_w + jobs};
                                double *const dst[] = {st.stack_num + jobs, st.stack_weight + jobs};
                                const dfl v[] = {dfl_mul(Q, w), w};
                                add(std::integral_constant<int, 2>{}, cell, dst, v);
                            }
                        } else {
                            report_error(scratch, PG_ERR_BIN_RANGE, jobs);
                        }
                    }
                }
                if (do_var && has_iv) {
                    // LeastsSquaresVarStats.initialize_delta_arrays
                    // (least_squares_var_stats.py:134-184)
                    constexpr float kMin = (float)kVarPipeMin, kMax = (float)kVarPipeMax;
                    const float lv = log10f(vp.hi) + vp.lo / (vp.hi * kLn10);
                    bool in_range;
                    int vbin = 0;
                    const float tv = (lv - kMin) * (float)(kVarBins / (kVarPipeMax - kVarPipeMin));
                    if (fabsf(lv - kMin) > 1e-4f && fabsf(lv - kMax) > 1e-4f &&
                        bin_certain(tv, 1e-3f, vbin)) {
                        in_range = lv > kMin && lv < kMax;
                    } else {
                        const double c64 = fit.continuum[off + p];
                        const double lv64 = log10(1 / iv64 / (c64 * c64));
                        in_range = lv64 > kVarPipeMin && lv64 < kVarPipeMax;
                        vbin = (int)((lv64 - kVarPipeMin) / (kVarPipeMax - kVarPipeMin) * kVarBins);
                    }
                    if (in_range) {
                        float t;
                        if (lin) {
                            const float lam = exp10f(L.hi) * fmaf(L.lo, kLn10, 1.f);
                            t = fmaf(lam - (float)st.var_grid0, inv_var, 0.5f);
                        } else {
                            t = fmaf((L.hi - var0.hi) + (L.lo - var0.lo), inv_var, 0.5f);
                        }
                        int lbin;
                        if (!bin_certain(t, guard, lbin))
                            lbin = (int)find_bin(ll, st.var_grid0, st.var_step, st.wave_lin);
                        const int64_t bin = vbin + (int64_t)kVarBins * lbin;
                        if (lbin >= 0 && bin >= 0 && bin < nvar) {
                            const dfl delta = dfl_add(Q, dfl{-1.f, 0.f});
                            const dfl d2 = dfl_mul(delta, delta);
                            const int k = (int)bin;
                            const int cell[] = {cells.v_mean + k, cells.v_d2 + k, cells.v_d4 + k};
                            double *const dst[] = {st.var_mean + k, st.var_delta2 + k,
                                                   st.var_delta4 + k};
                            const dfl v[] = {delta, d2, dfl_mul(d2, d2)};
                            add(std::integral_constant<int, 3>{}, cell, dst, v);
                            atomicAdd(&v_np[bin], 1u);
                            atomicOr(&seen[wib][bin >> 5], 1u << (bin & 31));
                        } else {
                            report_error(scratch, PG_ERR_BIN_RANGE, (int32_t)bin);
                        }
                    }
                }
            }
            if (do_var) {
                __syncwarp();
                for (int k = lane; k < 64; k += 32) {
                    uint32_t bits = seen[wib][k];
                    while (bits) {
                        const int bit = __ffs(bits) - 1;
                        bits &= bits - 1;
                        atomicAdd(&v_nq[k * 32 + bit], 1u);
                    }
                }
                __syncwarp();
            }
        }
        __syncwarp();
    }
    __syncthreads();
    auto flush_count = [&](double *dst, const uint32_t *c, int count) {
        for (int k = threadIdx.x; k < count; k += blockDim.x)
            if (c[k]) atomicAdd(&dst[k], (double)c[k]);
    };
    if (do_var) {
        flush_count(st.var_npix, v_np, nvar);
        flush_count(st.var_nqso, v_nq, nvar);
    }
    if (EXACT) {
        for (int k = threadIdx.x; k < nc; k += blockDim.x) {
            const uint32_t word[4] = {hist[k], hist[nc + k], hist[2 * nc + k], hist[3 * nc + k]};
            fix_add_global(exact_work + k, nc, word);
        }
        return;
    }
    // one FP64 add per nonzero bin and block
    const float *h = reinterpret_cast<const float *>(hist), *l = h + nc;
    auto flush = [&](double *dst, int from, int count) {
        for (int k = threadIdx.x; k < count; k += blockDim.x) {
            const float hk = h[from + k], lk = l[from + k];
            if (hk != 0.f || lk != 0.f) atomicAdd(&dst[k], (double)hk + (double)lk);
        }
    };
    flush(st.mean_cont_num, cells.mc_num, cells.mc_w - cells.mc_num);
    flush(st.mean_cont_weight, cells.mc_w, cells.s_num - cells.mc_w);
    flush(st.stack_num, cells.s_num, cells.s_w - cells.s_num);
    flush(st.stack_weight, cells.s_w, cells.v_mean - cells.s_w);
    flush(st.var_mean, cells.v_mean, nvar);
    flush(st.var_delta2, cells.v_d2, nvar);
    flush(st.var_delta4, cells.v_d4, nvar);
}

// The fixed-point sums of all blocks, added to the FP64 results.
__global__ void cont_stacks_finish_kernel(const __grid_constant__ pg_cont_stacks st,
                                          const unsigned long long *exact_work) {
    const StackCells c = stack_cells(st);
    const int k = blockIdx.x * blockDim.x + threadIdx.x, nc = c.total;
    if (k >= nc) return;
    double *dst;
    int from;
    if (k < c.mc_w) { dst = st.mean_cont_num; from = c.mc_num; }
    else if (k < c.s_num) { dst = st.mean_cont_weight; from = c.mc_w; }
    else if (k < c.s_w) { dst = st.stack_num; from = c.s_num; }
    else if (k < c.v_mean) { dst = st.stack_weight; from = c.s_w; }
    else if (k < c.v_d2) { dst = st.var_mean; from = c.v_mean; }
    else if (k < c.v_d4) { dst = st.var_delta2; from = c.v_d2; }
    else { dst = st.var_delta4; from = c.v_d4; }
    unsigned long long sum[kStackNumbers][3];
#pragma unroll
    for (int w = 0; w < kStackNumbers * 3; ++w) sum[w / 3][w % 3] = exact_work[w * nc + k];
    dst[k - from] += fix_value(sum[0], kFixScale) + fix_value(sum[1], kCoarseScale) +
                     fix_value(sum[2], kSmallScale);
}

// Deltas and weights (populate_los_ids, extract_deltas). Bound: the FP64 pipe.
// The table searches (nearest stack point, variance interval) compare keys
// that order like the doubles, on the integer pipe, against tables in shared
// memory (the stack's midpoints formed once per CTA), with one interval search
// for the three functions, and three divisions a pixel are left of five: about
// 60 FP64 operations instead of 125. 40,000 forests (6.4 million pixels):
// 1.47 ms, 0.72 ms now.
struct DeltaSmem {
    size_t mid, stack_y, brk, total;
};

__host__ __device__ inline DeltaSmem delta_smem(int num_stack, int intervals) {
    DeltaSmem l;
    l.mid = 0;
    l.stack_y = l.mid + (size_t)num_stack * 8;
    l.brk = l.stack_y + (size_t)num_stack * 8;
    l.total = l.brk + (size_t)(intervals + 1) * 8;
    return l;
}

// number of leading keys below v (OR_EQUAL: not above v)
template <bool OR_EQUAL>
__device__ __forceinline__ int count_keys(const unsigned long long *key, int n,
                                          unsigned long long v) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (OR_EQUAL ? key[mid] <= v : key[mid] < v) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// TABLES: the tables fit in shared memory; else (a stack of more than some
// 14,000 points) the searches read the model's arrays.
template <bool TABLES>
__global__ void __launch_bounds__(kContBlock) cont_deltas_kernel(
    const __grid_constant__ pg_spectra sp, const __grid_constant__ pg_cont_model m,
    const __grid_constant__ pg_cont_fit fit, double *__restrict__ delta,
    double *__restrict__ weights) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int ns = m.stack_x ? m.num_stack : 0;
    const int mi = m.use_constant_weight ? 0 : m.num_var_intervals;
    const DeltaSmem L = delta_smem(ns, mi);
    unsigned long long *mid = reinterpret_cast<unsigned long long *>(smem + L.mid);
    double *stack_y = reinterpret_cast<double *>(smem + L.stack_y);
    unsigned long long *brk = reinterpret_cast<unsigned long long *>(smem + L.brk);
    // scipy interp1d(kind="nearest"): x_bds[i] = (x[i] + x[i + 1]) / 2,
    // index = searchsorted(x_bds, v, "left")
    for (int k = threadIdx.x; TABLES && k < ns; k += blockDim.x) {
        if (k + 1 < ns) mid[k] = order_key((m.stack_x[k] + m.stack_x[k + 1]) / 2.0);
        stack_y[k] = m.stack_y[k];
    }
    if (TABLES && mi > 0)
        for (int k = threadIdx.x; k <= mi; k += blockDim.x) brk[k] = order_key(m.var_breaks[k]);
    __syncthreads();
    auto stack_at = [&](unsigned long long v) {
        if (TABLES) return stack_y[count_keys<false>(mid, ns - 1, v)];
        int lo = 0, hi = ns - 1;
        while (lo < hi) {
            const int i = (lo + hi) >> 1;
            if (order_key((m.stack_x[i] + m.stack_x[i + 1]) / 2.0) < v) lo = i + 1;
            else hi = i;
        }
        return m.stack_y[lo];
    };
    const int lane = threadIdx.x & 31;
    const int64_t warp_global = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t f = warp_global; f < sp.num; f += nwarps) {
        const int64_t off = sp.pix_offset[f];
        const int64_t n = sp.pix_offset[f + 1] - off;
        const bool ok = fit.status[f] == 0;
        for (int64_t p = lane; p < n; p += 32) {
            double w = 0., d = 0.;
            if (ok) {
                const double ll = sp.log_lambda[off + p], iv = sp.ivar[off + p];
                const unsigned long long key = order_key(ll);
                double expected = fit.continuum[off + p];
                if (ns > 0) expected *= stack_at(key);
                // compute_forest_weights (dr16_expected_flux.py:466-488) with
                // 1 / var_pipe = ivar expected^2
                if (iv > 0) {
                    double eta = 0., vlss = 1., fudge = 0.;
                    if (mi > 0) {
                        int i = TABLES ? count_keys<true>(brk, mi + 1, key) - 1
                                       : ppoly_piece(m.var_breaks, mi, ll);
                        i = i < 0 ? 0 : (i > mi - 1 ? mi - 1 : i);
                        const double dx = ll - m.var_breaks[i];
                        eta = ppoly_at(m.eta_coef, mi, i, dx);
                        vlss = ppoly_at(m.var_lss_coef, mi, i, dx);
                        fudge = ppoly_at(m.fudge_coef, mi, i, dx);
                    }
                    const double inv_pipe = iv * (expected * expected);
                    w = 1.0 / (eta * (1.0 / inv_pipe) + m.var_lss_mod * vlss + fudge * inv_pipe);
                }
                if (w > 0) d = sp.flux[off + p] / expected - 1;
            }
            delta[off + p] = d;
            weights[off + p] = w;
        }
    }
}

// Warm-start network inputs (see pg_mlp_features in include/picca_gb300.h),
// a warp per forest with forest_feature_sums. A CTA has a range of forests;
// its threads fetch the offsets and redshifts and form log10(1 + z) (FP64) of
// up to kFeatBlock of them together. Before, a
// warp took eight forests of five dependent loads each in a row: 209 us
// for 50,021 forests, 111 us now, at 2.3 TB/s bound by issue (1,700 instructions a
// forest: conversions, the segmented scan, IEEE roots and quotients).
constexpr int kFeatBlock = 512;

__global__ void __launch_bounds__(kFeatBlock) mlp_features_kernel(
    const __grid_constant__ pg_spectra sp, const __grid_constant__ pg_cont_model m, int64_t each,
    __nv_bfloat16 *__restrict__ feat, int stride, double *__restrict__ a0_out) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ float sums[kFeatBlock / 32][2][kFeatBins];
    __shared__ int64_t s_off[kFeatBlock];
    __shared__ int s_n[kFeatBlock];
    __shared__ double s_z[kFeatBlock];
    __shared__ float2 s_lm[kFeatBlock];
    const FitTables tab = load_fit_tables(m, smem);
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    const float bins_per_span = kFeatBins * tab.inv_span;
    const int64_t last = min(sp.num, (blockIdx.x + (int64_t)1) * each);
    for (int64_t first = blockIdx.x * each; first < last; first += kFeatBlock) {
        const int here = (int)min((int64_t)kFeatBlock, last - first);
        __syncthreads();
        if (threadIdx.x < here) {
            const int64_t f = first + threadIdx.x;
            const int64_t off = sp.pix_offset[f];
            s_off[threadIdx.x] = off;
            s_n[threadIdx.x] = (int)(sp.pix_offset[f + 1] - off);
            s_z[threadIdx.x] = sp.z_qso[f];
            s_lm[threadIdx.x] = forest_lmin(sp, m, f);
        }
        __syncthreads();
        for (int j = wib; j < here; j += kFeatBlock / 32) {
            const int64_t f = first + j;
            const FeatScalars fs = forest_feature_sums(sp, tab, s_off[j], s_n[j], s_z[j], s_lm[j].x,
                                                       s_lm[j].y, bins_per_span, sums[wib], lane);
            __nv_bfloat16 *row = feat + f * (int64_t)stride;
            for (int k = lane; k < stride; k += 32)
                row[k] = __float2bfloat16(forest_feature(sums[wib], fs, k));
            if (lane == 0) a0_out[f] = f32_to_f64(fs.a0);
            __syncwarp();
        }
    }
}

unsigned blocks_for(int64_t num, int num_sms) {
    const int64_t warps = (num + 0) > 0 ? num : 1;
    int64_t blocks = (warps * 32 + kContBlock - 1) / kContBlock;
    const int64_t cap = (int64_t)num_sms * 16;
    if (blocks > cap) blocks = cap;
    return (unsigned)(blocks < 1 ? 1 : blocks);
}

}  // namespace

int launch_cont_fit(const pg_spectra &sp, const pg_cont_model &m, const double *start,
                    const int32_t *index, int64_t count, int max_iter, double tol, int mode,
                    const pg_cont_fit &out, Scratch *scratch, int num_sms, cudaStream_t stream,
                    float cert_chi2, float cert_ab) {
    if (count <= 0) return PG_OK;
    if (mode == PG_FIT_MIXED) {
        const size_t smem = kFitSlabBytes * (kContBlock / 32) +
                            fit_smem_bytes(m.num_mean_cont, m.num_var_intervals);
        if (smem > 200 * 1024) return PG_ERR_UNSUPPORTED;
        cudaError_t err = cudaFuncSetAttribute(
            cont_fit_mixed_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (err != cudaSuccess) return check_cuda(err);
        // persistent blocks drawing groups of forests from the work counter
        int per_sm = 0;
        err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, cont_fit_mixed_kernel,
                                                            kContBlock, smem);
        if (err != cudaSuccess) return check_cuda(err);
        const int64_t groups = (count + kFitGroup - 1) / kFitGroup;
        int64_t mixed_blocks = (groups + kContBlock / 32 - 1) / (kContBlock / 32);
        const int64_t resident = (int64_t)num_sms * (per_sm > 0 ? per_sm : 1);
        if (mixed_blocks > resident) mixed_blocks = resident;
        cont_fit_mixed_kernel<<<(unsigned)mixed_blocks, kContBlock, smem, stream>>>(
            sp, m, start, index, count, max_iter, tol, out, scratch, cert_chi2, cert_ab);
    } else {
        const int rc = launch_fit64<kContK>(sp, m, start, index, count, max_iter, tol, out,
                                            &scratch->work_counter, scratch, num_sms, stream);
        if (rc) return rc;
    }
    cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) return check_cuda(err);
    // forests longer than those hold (the linear grid), in FP64; the long form
    // has no certificate: under it the warm-started fit of a long forest runs
    // to convergence with the plain fit's iteration limit
    const int rc = launch_fit64<kLongK>(sp, m, start, index, count,
                                        cert_chi2 > 0.f && max_iter < 100 ? 100 : max_iter,
                                        cert_chi2 > 0.f ? 1e-10 : tol, out, &scratch->long_counter, scratch,
                                        num_sms, stream);
    if (rc) return rc;
    if (mode == PG_FIT_MIXED && max_iter > 0 && !(cert_chi2 > 0.f)) {
        // the two-float finish of the forests flagged status 4, same stream
        const size_t rsmem = refine_smem_bytes(m.num_mean_cont, m.num_var_intervals);
        if (rsmem > 200 * 1024) return PG_ERR_UNSUPPORTED;
        err = cudaFuncSetAttribute(cont_fit_refine_kernel,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rsmem);
        if (err != cudaSuccess) return check_cuda(err);
        // every SM filled: the flagged forests are scattered over the list
        int per_sm = 0;
        err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, cont_fit_refine_kernel,
                                                            32 * kRefineWarps, rsmem);
        if (err != cudaSuccess) return check_cuda(err);
        int64_t rblocks = (int64_t)num_sms * (per_sm > 0 ? per_sm : 1);
        const int64_t need = (count + 32 * kRefineWarps - 1) / (32 * kRefineWarps);
        if (rblocks > need) rblocks = need;
        cont_fit_refine_kernel<<<(unsigned)rblocks, 32 * kRefineWarps, rsmem, stream>>>(
            sp, m, index, count, out, scratch);
        err = cudaGetLastError();
    }
    return check_cuda(err);
}

constexpr size_t kStackLimit = 200 * 1024;  // shared memory of a block

// Blocks of BLOCK threads as many as are resident; the variance-function table
// where it fits beside the histograms.
template <bool EXACT, int BLOCK>
static int launch_stacks(const pg_spectra &sp, const pg_cont_model &m, const pg_cont_fit &fit,
                         const pg_cont_stacks &st, bool use_table,
                         unsigned long long *exact_work, Scratch *scratch, int num_sms,
                         cudaStream_t stream) {
    const auto kernel = cont_stacks_kernel<EXACT, BLOCK>;
    const size_t smem = stack_bytes(st, EXACT, use_table);
    cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)kStackLimit);
    if (err != cudaSuccess) return check_cuda(err);
    int per_sm = 0;
    err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, BLOCK, smem);
    if (err != cudaSuccess) return check_cuda(err);
    // few forests: a group of them a block, spread over the SMs (1,000 of the log
    // grid 0.45 ms in full blocks, 0.32 ms)
    int64_t blocks = (sp.num + kStackGroup - 1) / kStackGroup;
    const int64_t resident = (int64_t)num_sms * (per_sm > 0 ? per_sm : 1);
    if (blocks > resident) blocks = resident;
    kernel<<<(unsigned)(blocks < 1 ? 1 : blocks), BLOCK, smem, stream>>>(
        sp, m, fit, st, scratch, use_table, exact_work);
    return check_cuda(cudaGetLastError());
}

// a cell has 16 bytes of shared memory and kStackWork of the work (a plan with
// over 1 MB, as four counters a number would need, takes 0.07 ms more to make)
constexpr size_t kStackWork = 24 * kStackNumbers;
size_t cont_exact_bytes() { return kStackLimit / 16 * kStackWork; }

int launch_cont_stacks(const pg_spectra &sp, const pg_cont_model &m, const pg_cont_fit &fit,
                       const pg_cont_stacks &st, unsigned long long *exact_work,
                       size_t exact_bytes, Scratch *scratch, int num_sms,
                       cudaStream_t stream) {
    if (sp.num <= 0) return PG_OK;
    if (st.var_mean && st.var_lambda_bins * kVarBins > 2048) return PG_ERR_UNSUPPORTED;
    constexpr size_t limit = kStackLimit;
    const bool want_table = !m.use_constant_weight && (st.mean_cont_num || st.stack_num);
    const bool pair_table = want_table && stack_smem_bytes(st, true) <= limit;
    if (stack_smem_bytes(st, pair_table) > limit) return PG_ERR_UNSUPPORTED;
    const StackCells cells = stack_cells(st);
    const size_t work = (size_t)cells.total * kStackWork;
    if (stack_bytes(st, true, false) > limit || work > exact_bytes)
        return launch_stacks<false, kStackBlock>(sp, m, fit, st, pair_table, nullptr, scratch,
                                                 num_sms, stream);
    const bool table = want_table && stack_bytes(st, true, true) <= limit;
    if (pair_table && !table && st.stack_num && (st.mean_cont_num || st.var_mean)) {
        // the table beside one part of the histograms at a time (6,000 forests,
        // 2,400 bins of the linear grid: 4.2 ms in one pass without it, 2.1 ms)
        pg_cont_stacks one = st, two = st;
        one.stack_num = one.stack_weight = nullptr;
        two.mean_cont_num = two.mean_cont_weight = two.var_mean = nullptr;
        int rc = launch_cont_stacks(sp, m, fit, one, exact_work, exact_bytes, scratch, num_sms,
                                    stream);
        if (rc) return rc;
        rc = check_cuda(cudaMemsetAsync(&scratch->work_counter, 0, sizeof(scratch->work_counter),
                                        stream));
        return rc ? rc
                  : launch_cont_stacks(sp, m, fit, two, exact_work, exact_bytes, scratch, num_sms,
                                       stream);
    }
    cudaError_t err = cudaMemsetAsync(exact_work, 0, work, stream);
    if (err != cudaSuccess) return check_cuda(err);
    const int rc = launch_stacks<true, 2 * kStackBlock>(sp, m, fit, st, table, exact_work,
                                                        scratch, num_sms, stream);
    if (rc) return rc;
    if (cells.total > 0)
        cont_stacks_finish_kernel<<<(cells.total + 255) / 256, 256, 0, stream>>>(st, exact_work);
    return check_cuda(cudaGetLastError());
}

int launch_mlp_features(const pg_spectra &sp, const pg_cont_model &m, uint16_t *features,
                        int stride, double *a0, int num_sms, cudaStream_t stream) {
    if (sp.num <= 0) return PG_OK;
    const size_t smem = fit_smem_bytes(m.num_mean_cont, m.num_var_intervals);
    if (smem > 200 * 1024) return PG_ERR_UNSUPPORTED;
    cudaError_t err = cudaFuncSetAttribute(
        mlp_features_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) return check_cuda(err);
    int per_sm = 0;
    err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, mlp_features_kernel, kFeatBlock,
                                                        smem);
    if (err != cudaSuccess) return check_cuda(err);
    // one resident wave of CTAs, as many forests for each of their warps
    constexpr int64_t warps = kFeatBlock / 32;
    const int64_t resident = (int64_t)num_sms * (per_sm > 0 ? per_sm : 1) * warps;
    const int64_t each = (sp.num + resident - 1) / resident * warps;
    const int64_t blocks = (sp.num + each - 1) / each;
    mlp_features_kernel<<<(unsigned)blocks, kFeatBlock, smem, stream>>>(
        sp, m, each, reinterpret_cast<__nv_bfloat16 *>(features), stride, a0);
    return check_cuda(cudaGetLastError());
}

int launch_cont_deltas(const pg_spectra &sp, const pg_cont_model &m, const pg_cont_fit &fit,
                       double *delta, double *weights, int num_sms, cudaStream_t stream) {
    if (sp.num <= 0) return PG_OK;
    const size_t smem = delta_smem(m.stack_x ? m.num_stack : 0,
                                   m.use_constant_weight ? 0 : m.num_var_intervals).total;
    unsigned blocks = blocks_for(sp.num, num_sms);
    if (blocks > (unsigned)num_sms * 8) blocks = (unsigned)num_sms * 8;
    if (smem > kMaxDynSmem) {
        cont_deltas_kernel<false><<<blocks, kContBlock, 0, stream>>>(sp, m, fit, delta, weights);
        return check_cuda(cudaGetLastError());
    }
    cudaError_t err = cudaFuncSetAttribute(cont_deltas_kernel<true>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)kMaxDynSmem);
    if (err != cudaSuccess) return check_cuda(err);
    cont_deltas_kernel<true><<<blocks, kContBlock, smem, stream>>>(sp, m, fit, delta, weights);
    return check_cuda(cudaGetLastError());
}

}  // namespace pg
