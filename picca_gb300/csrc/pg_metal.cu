// Metal distortion matrices: cf.compute_metal_dmat (py/picca/cf.py:890-1218)
// and, with the quasars as one-pixel forests, xcf.compute_metal_dmat
// (py/picca/xcf.py:677-800).
//
// For every kept forest pair the reference bins all pixel pairs twice: with
// the tracer's distances (data bin, r_par / r_trans of the delta files) and
// with the distances the two pixels would have if they were absorbers abs1 /
// abs2 (model bin), and adds w1 w2 to the data-bin weights and
// w1 w2 zevol to the (data bin, model bin) cell and the model bin's
// effective r_par / r_trans / z / weight (numpy bincounts). Pixels whose
// absorber redshift is not below the quasar redshift are dropped; the caller
// encodes that as a zero weight in the absorber arrays.
//
// metal_runs_kernel (the correlation of delta fields): a CTA per kept forest
// pair. Both forests are staged, the pixel pairs are swept along diagonals (a
// lane per diagonal, warps take groups of 32), and both bins are decided in
// FP32 with the guard bands of pg_pairs_common.cuh (pairs near an edge of
// either are queued and decided with the reference's FP64 expressions).
// Consecutive pairs of a diagonal share (data bin, model bin) for about ten
// steps: they are summed in FP64 registers as a run and the runs applied 32 at
// a time. Bound: the FP64 pipe (16 cycles a warp operation and SM), ten
// operations a pair. The kernel below it formed the bins in FP64 (about 45
// operations) and walked forest 2 for a fixed pixel, where runs are two pixels
// long: LYA x SiIII(1207), both passes, 6,200 pairs of 500 forests 43.4 ms, and
// 3.2 ms here.
//
// metal_dmat_kernel (delta x quasar: one-pixel second forests, which have no
// diagonals; and forests too long to stage): a thread per pixel of forest 1
// walks the pixels of forest 2, sums runs and adds each with global atomics,
// FP64 in the reference's expressions; the bin quotients are estimated with
// reciprocals and formed exactly next to a bin edge.
#include <algorithm>

#include "pg_internal.cuh"
#include "pg_pairs_common.cuh"

namespace pg {
namespace {

constexpr int kMdBlock = 256;

struct MetalConst {
    Binning b;
    int32_t nmp, nmt, nm;
    double inv_range, inv_rtmax;
    double inv_zevol_den;  // 1 / (1 + z_ref)^(alpha1 + alpha2 - 2)
    int32_t xcf;           // delta x quasar rules (py/picca/xcf.py:735-770)
};

__device__ __forceinline__ double md_floor(double est, double num, double den, int32_t n) {
    const double y = __dmul_rn(est, (double)n);
    const double f = floor(y);
    if (__dsub_rn(y, f) > 1e-9 && __dsub_rn(__dadd_rn(f, 1.), y) > 1e-9) return f;
    return floor(__dmul_rn(num / den, (double)n));
}

__global__ void __launch_bounds__(kMdBlock)
    metal_dmat_kernel(MetalConst c, pg_forest_set s1, pg_forest_set s2, pg_metal_pixels a1,
                      pg_metal_pixels a2, const int32_t *pair_first,
                      const int32_t *pair_second, const double *pair_angle, int64_t num_pairs,
                      pg_dmat_sums out, Scratch *scratch) {
    __shared__ int s_item;
    const int tid = threadIdx.x;
    const int nm = c.nm;
    for (;;) {
        if (tid == 0) s_item = atomicAdd(&scratch->work_counter, 1);
        __syncthreads();
        const int64_t q = s_item;
        __syncthreads();
        if (q >= num_pairs) break;
        const int f = pair_first[q], g = pair_second[q];
        const double ang = pair_angle ? pair_angle[q]
                                      : angle_between(s1.x_cart[f], s1.y_cart[f], s1.z_cart[f],
                                                      s1.ra[f], s1.dec[f], s1.cos_dec[f],
                                                      s2.x_cart[g], s2.y_cart[g], s2.z_cart[g],
                                                      s2.ra[g], s2.dec[g]);
        const double cc = cos(ang / 2), ss = sin(ang / 2);
        bool shp = false;
        if (c.b.remove_shp && s1.plate[f] == s2.plate[g]) {
            const int64_t fa = s1.fiberid[f], fb = s2.fiberid[g];
            shp = (fa <= 500 && fb <= 500) || (fa > 500 && fb > 500);
        }
        const int64_t o1 = s1.pix_offset[f], o2 = s2.pix_offset[g];
        const int n1 = (int)(s1.pix_offset[f + 1] - o1), n2 = (int)(s2.pix_offset[g + 1] - o2);
        if (tid == 0) atomicAdd(&scratch->work_items, 1ull);
        for (int i = tid; i < n1; i += kMdBlock) {
            const double w1 = a1.weights[o1 + i];
            if (w1 == 0.) continue;
            const double r1 = s1.r_comov[o1 + i], m1 = s1.dist_m[o1 + i];
            const double ra1 = a1.r_comov[o1 + i], ma1 = a1.dist_m[o1 + i];
            const double za1 = a1.z[o1 + i], zf1 = a1.zfac[o1 + i];
            // runs of equal data bin (weights) and of equal (data, model) bin
            int32_t run_b = -1;
            double k_w = 0.;
            int64_t run = -1;
            int32_t run_m = 0;
            double k_wz = 0., k_rp = 0., k_rt = 0., k_z = 0.;
            auto flush = [&]() {
                atomicAdd(&out.dmat[run], k_wz);
                atomicAdd(&out.r_par_eff[run_m], k_rp);
                atomicAdd(&out.r_trans_eff[run_m], k_rt);
                atomicAdd(&out.z_eff[run_m], k_z);
                atomicAdd(&out.weight_eff[run_m], k_wz);
            };
            for (int j = 0; j < n2; ++j) {
                const double w2 = a2.weights[o2 + j];
                if (w2 == 0.) continue;
                // data bin with the tracer's distances (cf.py:995-1021)
                double rp = __dmul_rn(__dsub_rn(r1, s2.r_comov[o2 + j]), cc);
                if (!c.b.x_correlation) rp = fabs(rp);
                const double rt = __dmul_rn(__dadd_rn(m1, s2.dist_m[o2 + j]), ss);
                if (shp && fabs(rp) < c.b.half_plate_cut) continue;  // weight set to 0
                // the cross tests the distances (strict), the auto its bin indices
                if (c.xcf && !(rp > c.b.r_par_min && rp < c.b.r_par_max &&
                               rt < c.b.r_trans_max))
                    continue;
                const double xp = __dsub_rn(rp, c.b.r_par_min);
                const double bp = md_floor(__dmul_rn(xp, c.inv_range), xp, c.b.r_par_range,
                                           c.b.np);
                const double bt = md_floor(__dmul_rn(rt, c.inv_rtmax), rt, c.b.r_trans_max,
                                           c.b.nt);
                if (!(bp < c.b.np && bt < c.b.nt && bp >= 0.)) {
                    if (c.xcf) report_error(scratch, PG_ERR_BIN_RANGE, (int32_t)bp);
                    continue;
                }
                const double w12 = __dmul_rn(w1, w2);
                const int32_t b = (int32_t)bt + c.b.nt * (int32_t)bp;
                if (b != run_b) {
                    if (run_b >= 0) atomicAdd(&out.weights_dmat[run_b], k_w);
                    run_b = b;
                    k_w = 0.;
                }
                k_w += w12;
                // model bin with the absorbers' distances (cf.py:1023-1086)
                double rpa = __dmul_rn(__dsub_rn(ra1, a2.r_comov[o2 + j]), cc);
                if (!c.b.x_correlation) rpa = fabs(rpa);
                const double rta = __dmul_rn(__dadd_rn(ma1, a2.dist_m[o2 + j]), ss);
                if (c.xcf && !(rpa > c.b.r_par_min && rpa < c.b.r_par_max &&
                               rta < c.b.r_trans_max))
                    continue;
                const double xm = __dsub_rn(rpa, c.b.r_par_min);
                const double mp = md_floor(__dmul_rn(xm, c.inv_range), xm, c.b.r_par_range,
                                           c.nmp);
                const double mt = md_floor(__dmul_rn(rta, c.inv_rtmax), rta, c.b.r_trans_max,
                                           c.nmt);
                if (!(mp < c.nmp && mt < c.nmt && mp >= 0.)) {
                    if (c.xcf) report_error(scratch, PG_ERR_BIN_RANGE, (int32_t)mp);
                    continue;
                }
                const int32_t mb = (int32_t)mt + c.nmt * (int32_t)mp;
                const int64_t key = (int64_t)b * nm + mb;
                if (key != run) {
                    if (run >= 0) flush();
                    run = key;
                    run_m = mb;
                    k_wz = k_rp = k_rt = k_z = 0.;
                }
                const double zevol =
                    __dmul_rn(__dmul_rn(zf1, a2.zfac[o2 + j]), c.inv_zevol_den);
                const double wz = __dmul_rn(w12, zevol);
                k_wz += wz;
                k_rp += __dmul_rn(rpa, wz);
                k_rt += __dmul_rn(rta, wz);
                k_z += __dmul_rn(__dadd_rn(za1, a2.z[o2 + j]) / 2, wz);
            }
            if (run_b >= 0) atomicAdd(&out.weights_dmat[run_b], k_w);
            if (run >= 0) flush();
        }
    }
}

// ---------------------------------------------------------------------------
// Diagonal sweeps with FP32 decisions
// ---------------------------------------------------------------------------
constexpr int kMrWarps = 4;
constexpr int kMrRing = 64;    // runs held per warp (<= 31 + 32)
constexpr int kMrQueue = 96;   // queued pairs per warp

// A pixel as the sums need it (structure of arrays in shared memory).
struct MetalPix {
    double *w, *wz, *r, *m, *z;
};

__device__ __forceinline__ MetalPix metal_pix(void *base, int n) {
    double *d = static_cast<double *>(base);
    return {d, d + n, d + 2 * n, d + 3 * n, d + 4 * n};
}

// Byte offsets. f1 / f2: float4 (r_par and r_trans parts of the data bin, of
// the model bin) per pixel; q1 / q2: MetalPix; per warp the run ring (five
// sums, data and model bin) and the queue.
struct MrSmem {
    size_t f1, f2, q1, q2, warps, per_warp, ring, ring_bin, queue, total;
};

__host__ __device__ inline MrSmem mr_smem(int max1, int max2) {
    MrSmem l;
    l.f1 = 0;
    l.f2 = l.f1 + (size_t)max1 * 16;
    l.q1 = l.f2 + (size_t)max2 * 16;
    l.q2 = l.q1 + (size_t)max1 * 40;
    l.warps = l.q2 + (size_t)max2 * 40;
    l.ring = 0;
    l.ring_bin = l.ring + (size_t)kMrRing * 40;
    l.queue = l.ring_bin + (size_t)kMrRing * 8;
    l.per_warp = (l.queue + (size_t)kMrQueue * 4 + 15) & ~(size_t)15;
    l.total = l.warps + kMrWarps * l.per_warp;
    return l;
}

struct MetalPair {
    int64_t o1, o2;
    double cc, ss;
    bool shp;
};

// One pixel pair with the reference's expressions (cf.py:995-1086).
__device__ __forceinline__ void metal_pair_fp64(const MetalConst &c, const pg_forest_set &s1,
                                                const pg_forest_set &s2,
                                                const pg_metal_pixels &a1,
                                                const pg_metal_pixels &a2, const MetalPair &p,
                                                int i, int j, const pg_dmat_sums &out) {
    const int64_t x = p.o1 + i, y = p.o2 + j;
    double rp = __dmul_rn(__dsub_rn(s1.r_comov[x], s2.r_comov[y]), p.cc);
    if (!c.b.x_correlation) rp = fabs(rp);
    const double rt = __dmul_rn(__dadd_rn(s1.dist_m[x], s2.dist_m[y]), p.ss);
    if (p.shp && fabs(rp) < c.b.half_plate_cut) return;
    const double xp = __dsub_rn(rp, c.b.r_par_min);
    const double bp = md_floor(__dmul_rn(xp, c.inv_range), xp, c.b.r_par_range, c.b.np);
    const double bt = md_floor(__dmul_rn(rt, c.inv_rtmax), rt, c.b.r_trans_max, c.b.nt);
    if (!(bp < c.b.np && bt < c.b.nt && bp >= 0.)) return;
    const double w12 = __dmul_rn(a1.weights[x], a2.weights[y]);
    const int32_t b = (int32_t)bt + c.b.nt * (int32_t)bp;
    atomicAdd(&out.weights_dmat[b], w12);
    double rpa = __dmul_rn(__dsub_rn(a1.r_comov[x], a2.r_comov[y]), p.cc);
    if (!c.b.x_correlation) rpa = fabs(rpa);
    const double rta = __dmul_rn(__dadd_rn(a1.dist_m[x], a2.dist_m[y]), p.ss);
    const double xm = __dsub_rn(rpa, c.b.r_par_min);
    const double mp = md_floor(__dmul_rn(xm, c.inv_range), xm, c.b.r_par_range, c.nmp);
    const double mt = md_floor(__dmul_rn(rta, c.inv_rtmax), rta, c.b.r_trans_max, c.nmt);
    if (!(mp < c.nmp && mt < c.nmt && mp >= 0.)) return;
    const int32_t mb = (int32_t)mt + c.nmt * (int32_t)mp;
    const double wz = __dmul_rn(
        w12, __dmul_rn(__dmul_rn(a1.zfac[x], a2.zfac[y]), c.inv_zevol_den));
    atomicAdd(&out.dmat[(int64_t)b * c.nm + mb], wz);
    atomicAdd(&out.r_par_eff[mb], __dmul_rn(rpa, wz));
    atomicAdd(&out.r_trans_eff[mb], __dmul_rn(rta, wz));
    atomicAdd(&out.z_eff[mb], __dmul_rn(__dadd_rn(a1.z[x], a2.z[y]) / 2, wz));
    atomicAdd(&out.weight_eff[mb], wz);
}

__device__ __noinline__ void metal_drain(const MetalConst &c, const pg_forest_set &s1,
                                         const pg_forest_set &s2, const pg_metal_pixels &a1,
                                         const pg_metal_pixels &a2, const MetalPair &p,
                                         const uint32_t *queue, int count,
                                         const pg_dmat_sums &out) {
    __syncwarp();
    for (int e = threadIdx.x & 31; e < count; e += 32)
        metal_pair_fp64(c, s1, s2, a1, a2, p, (int)(queue[e] >> 16), (int)(queue[e] & 0xFFFF),
                        out);
    __syncwarp();
}

// Adds n (<= 32) runs of the ring, from position head.
__device__ __forceinline__ void metal_apply(const MetalConst &c, const double *ring,
                                            const int2 *ring_bin, int head, int n,
                                            const MetalPair &p, const pg_dmat_sums &out) {
    __syncwarp();
    const int lane = threadIdx.x & 31;
    if (lane < n) {
        const int e = (head + lane) & (kMrRing - 1);
        const int2 bin = ring_bin[e];
        atomicAdd(&out.weights_dmat[bin.x], ring[e]);
        if (bin.y >= 0) {
            const double wz = ring[kMrRing + e];
            atomicAdd(&out.dmat[(int64_t)bin.x * c.nm + bin.y], wz);
            atomicAdd(&out.weight_eff[bin.y], wz);
            atomicAdd(&out.r_par_eff[bin.y], __dmul_rn(ring[2 * kMrRing + e], p.cc));
            atomicAdd(&out.r_trans_eff[bin.y], __dmul_rn(ring[3 * kMrRing + e], p.ss));
            atomicAdd(&out.z_eff[bin.y], __dmul_rn(ring[4 * kMrRing + e], 0.5));
        }
    }
    __syncwarp();
}

// Stages n pixels: f = the FP32 parts (sign * cp * (r - ref), st * d + off,
// the same with the absorber's distances), q = the FP64 terms. A pixel
// without weight is marked by an r_par part of the model bin at kFar. Returns
// whether the tracer's distances are non-decreasing (this thread's pixels)
// and raises the largest |r - ref| of both.
template <bool SECOND>
__device__ __forceinline__ bool stage_metal(const pg_forest_set &s, const pg_metal_pixels &a,
                                            int64_t o, int n, double ref, double ref_a, float cp,
                                            float st, float cpm, float stm, double wz_scale,
                                            float4 *f, const MetalPix &q, unsigned *max_rho) {
    bool ordered = true;
    float top = 0.f, top_a = 0.f;
    for (int i = threadIdx.x; i < n; i += kMrWarps * 32) {
        const double r = s.r_comov[o + i], m = s.dist_m[o + i], w = a.weights[o + i];
        const double ra = a.r_comov[o + i], ma = a.dist_m[o + i];
        const float rho = (float)(r - ref), d = (float)m;
        const float rho_a = (float)(ra - ref_a), d_a = (float)ma;
        if (SECOND)
            f[i] = make_float4(-__fmul_rn(cp, rho), __fmaf_rn(st, d, -0.5f),
                               w != 0. ? -__fmul_rn(cpm, rho_a) : kFar,
                               __fmaf_rn(stm, d_a, -0.5f));
        else
            f[i] = make_float4(rho, d, w != 0. ? rho_a : kFar, d_a);
        q.w[i] = w;
        q.wz[i] = __dmul_rn(__dmul_rn(w, a.zfac[o + i]), wz_scale);
        q.r[i] = ra;
        q.m[i] = ma;
        q.z[i] = a.z[o + i];
        top = fmaxf(top, fabsf(rho));
        top_a = fmaxf(top_a, fabsf(rho_a));
        if (i + 1 < n)
            ordered &= (float)(s.r_comov[o + i + 1] - ref) >= rho &&
                       (float)s.dist_m[o + i + 1] >= d;
    }
    if (!SECOND) {
        atomicMax(&max_rho[0], __float_as_uint(top));
        atomicMax(&max_rho[1], __float_as_uint(top_a));
    }
    return ordered;
}

__global__ void __launch_bounds__(kMrWarps * 32, 5) metal_runs_kernel(
    const __grid_constant__ MetalConst c, const __grid_constant__ FastConst fd,
    const __grid_constant__ FastConst fm, const __grid_constant__ pg_forest_set s1,
    const __grid_constant__ pg_forest_set s2, const __grid_constant__ pg_metal_pixels a1,
    const __grid_constant__ pg_metal_pixels a2, const int32_t *__restrict__ pair_first,
    const int32_t *__restrict__ pair_second, const double *__restrict__ pair_angle,
    int64_t num_pairs, const __grid_constant__ pg_dmat_sums out, Scratch *scratch, int max1,
    int max2) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_item, s_group;
    __shared__ unsigned max_rho[2];
    __shared__ int band[2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned lt_mask = (1u << lane) - 1u;
    const MrSmem L = mr_smem(max1, max2);
    float4 *f1 = reinterpret_cast<float4 *>(smem + L.f1);
    float4 *f2 = reinterpret_cast<float4 *>(smem + L.f2);
    const MetalPix q1 = metal_pix(smem + L.q1, max1), q2 = metal_pix(smem + L.q2, max2);
    unsigned char *wbase = smem + L.warps + (size_t)warp * L.per_warp;
    double *ring = reinterpret_cast<double *>(wbase + L.ring);
    int2 *ring_bin = reinterpret_cast<int2 *>(wbase + L.ring_bin);
    uint32_t *queue = reinterpret_cast<uint32_t *>(wbase + L.queue);
    const bool folded = !c.b.x_correlation;
    const float pmin_f = fd.pc - 0.5f;
    const float p_hi = pmin_f + (float)fd.np + 1.f, p_lo = folded ? -p_hi : pmin_f - 1.f;
    const float t_end = (float)fd.nt + 1.f;
    for (;;) {
        __syncthreads();
        if (tid == 0) {
            s_item = atomicAdd(&scratch->work_counter, 1);
            s_group = 0;
            max_rho[0] = max_rho[1] = 0u;
            band[0] = INT_MAX;
            band[1] = INT_MIN;
        }
        __syncthreads();
        const int64_t item = s_item;
        if (item >= num_pairs) break;
        const int f = pair_first[item], g = pair_second[item];
        MetalPair p;
        const double ang = pair_angle ? pair_angle[item]
                                      : angle_between(s1.x_cart[f], s1.y_cart[f], s1.z_cart[f],
                                                      s1.ra[f], s1.dec[f], s1.cos_dec[f],
                                                      s2.x_cart[g], s2.y_cart[g], s2.z_cart[g],
                                                      s2.ra[g], s2.dec[g]);
        p.cc = cos(ang / 2);
        p.ss = sin(ang / 2);
        p.shp = false;
        if (c.b.remove_shp && s1.plate[f] == s2.plate[g]) {
            const int64_t fa = s1.fiberid[f], fb = s2.fiberid[g];
            p.shp = (fa <= 500 && fb <= 500) || (fa > 500 && fb > 500);
        }
        p.o1 = s1.pix_offset[f];
        p.o2 = s2.pix_offset[g];
        const int64_t n1_64 = s1.pix_offset[f + 1] - p.o1, n2_64 = s2.pix_offset[g + 1] - p.o2;
        if (tid == 0) atomicAdd(&scratch->work_items, 1ull);
        if (n1_64 > max1 || n2_64 > max2) {
            if (tid == 0) report_error(scratch, PG_ERR_UNSUPPORTED, (int32_t)item);
            continue;
        }
        const int n1 = (int)n1_64, n2 = (int)n2_64;
        if (n1 < 1 || n2 < 1) continue;
        const double ref = reference_distance(s1.r_comov[p.o1 + n1 / 2], &max_rho[0]);
        const double ref_a = reference_distance(a1.r_comov[p.o1 + n1 / 2], &max_rho[1]);
        const float cp = (float)(p.cc * fd.inv_p), st = (float)(p.ss * fd.inv_t);
        const float cpm = (float)(p.cc * fm.inv_p), stm = (float)(p.ss * fm.inv_t);
        bool ordered = stage_metal<false>(s1, a1, p.o1, n1, ref, ref_a, cp, st, cpm, stm,
                                          c.inv_zevol_den, f1, q1, max_rho);
        ordered &= stage_metal<true>(s2, a2, p.o2, n2, ref, ref_a, cp, st, cpm, stm, 1., f2, q2,
                                     max_rho);
        ordered = __syncthreads_and(ordered) != 0;
        const ParGuard gd = par_guard_exact(&fd, __uint_as_float(max_rho[0]));
        const ParGuard gm = par_guard_exact(&fm, __uint_as_float(max_rho[1]));
        ordered &= !gd.wide;
        // diagonals j - i that can hold a pair within one bin of the r_par
        // range (both forests in order; else all of them)
        int d_lo = -(n1 - 1), d_hi = n2;
        if (ordered) {
            int lo = INT_MAX, hi = INT_MIN;
            for (int i = tid; i < n1; i += kMrWarps * 32) {
                const float x = __fmul_rn(cp, f1[i].x);
                const int j1 = count_leading<false>(f2, n2, p_hi - x);
                const int j2 = count_leading<true>(f2, n2, p_lo - x);
                if (j1 < j2) {
                    lo = min(lo, j1 - i);
                    hi = max(hi, j2 - i);
                }
            }
            lo = __reduce_min_sync(0xffffffffu, lo);
            hi = __reduce_max_sync(0xffffffffu, hi);
            if (lane == 0) {
                atomicMin(&band[0], lo);
                atomicMax(&band[1], hi);
            }
            __syncthreads();
            const bool any = band[0] < band[1];
            d_lo = any ? band[0] : 0;
            d_hi = any ? band[1] : 0;
        }
        const bool t_trim = ordered && st > 0.f;
        int head = 0, tail = 0, qn = 0;  // run ring and queue (warp-uniform)
        for (;;) {
            int grp = 0;
            if (lane == 0) grp = atomicAdd(&s_group, 1);
            const int d0 = d_lo + 32 * __shfl_sync(0xffffffffu, grp, 0);
            if (d0 >= d_hi) break;
            const int d = d0 + lane;
            int ia = max(0, -d), ib = min(n1, n2 - d);
            if (d >= d_hi) ib = ia;
            if (t_trim && ia < ib) {
                int lo = ia, hi = ib;
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (__fmaf_rn(st, f1[mid].y, f2[mid + d].y) < t_end) lo = mid + 1;
                    else hi = mid;
                }
                ib = lo;
            }
            // the lanes step forest 2 together (a broadcast read)
            const int ja = ia + d, jb = ib + d;
            const int g_lo = __reduce_min_sync(0xffffffffu, ia < ib ? ja : INT_MAX);
            const int g_hi = __reduce_max_sync(0xffffffffu, ia < ib ? jb : INT_MIN);
            int run_b = -1, run_m = -1;
            double k_w = 0., k_wz = 0., k_rp = 0., k_rt = 0., k_z = 0.;
            auto store_runs = [&](bool flag) {
                const unsigned m = __ballot_sync(0xffffffffu, flag);
                if (flag) {
                    const int pos = (tail + __popc(m & lt_mask)) & (kMrRing - 1);
                    ring[pos] = k_w;
                    ring[kMrRing + pos] = k_wz;
                    ring[2 * kMrRing + pos] = k_rp;
                    ring[3 * kMrRing + pos] = k_rt;
                    ring[4 * kMrRing + pos] = k_z;
                    ring_bin[pos] = make_int2(run_b, run_m);
                }
                tail += __popc(m);
                if (tail - head >= 32) {
                    metal_apply(c, ring, ring_bin, head, 32, p, out);
                    head += 32;
                }
            };
            for (int j = g_lo; j < g_hi; ++j) {
                const bool in = (j >= ja) & (j < jb);
                const int i = in ? j - d : 0;
                const float4 x = f1[i], y = f2[j];
                const float pp = __fmaf_rn(cp, x.x, y.x), v = fabsf(pp);
                const float xt = __fmaf_rn(st, x.y, y.y);
                const float xp0 = (folded ? v : pp) - fd.pc;
                const float xp = fd.lower_exact ? clamp_low(xp0, gd.low_clamp) : xp0;
                float rem_p, rem_t;
                const unsigned ip = round_rem(xp, rem_p), it = round_rem(xt, rem_t);
                bool near = (fabsf(rem_p) > gd.h_par) | (fabsf(rem_t) > fd.h_tr);
                bool ok = (ip < fd.np) & (it < fd.nt);
                if (p.shp) {
                    near |= fabsf(v - 1.f) < gd.guard_v;
                    ok &= !(v < 1.f);
                }
                // the model bin
                const float pa = __fmaf_rn(cpm, x.z, y.z);
                const float ta = __fmaf_rn(stm, x.w, y.w);
                const float xa0 = (folded ? fabsf(pa) : pa) - fm.pc;
                const float xa = fm.lower_exact ? clamp_low(xa0, gm.low_clamp) : xa0;
                const unsigned mp = round_rem(xa, rem_p), mt = round_rem(ta, rem_t);
                near |= ok & ((fabsf(rem_p) > gm.h_par) | (fabsf(rem_t) > fm.h_tr));
                const bool live = in & (x.z < kFar) & (y.z < kFar);
                near &= live;
                ok &= live & !near;
                const int bin = (int)(ip * fd.nt + it);
                const int model = (mp < fm.np) & (mt < fm.nt) ? (int)(mp * fm.nt + mt) : -1;
                const bool brk = ok & ((bin != run_b) | (model != run_m));
                const bool flush = brk & (run_b >= 0);
                if (__any_sync(0xffffffffu, flush)) store_runs(flush);
                if (brk) {
                    run_b = bin;
                    run_m = model;
                    k_w = k_wz = k_rp = k_rt = k_z = 0.;
                }
                if (ok) {
                    k_w = fma(q1.w[i], q2.w[j], k_w);
                    const double wz = __dmul_rn(q1.wz[i], q2.wz[j]);
                    const double dr = __dsub_rn(q1.r[i], q2.r[j]);
                    k_wz = __dadd_rn(k_wz, wz);
                    k_rp = fma(folded ? fabs(dr) : dr, wz, k_rp);
                    k_rt = fma(__dadd_rn(q1.m[i], q2.m[j]), wz, k_rt);
                    k_z = fma(__dadd_rn(q1.z[i], q2.z[j]), wz, k_z);
                }
                const unsigned nmask = __ballot_sync(0xffffffffu, near);
                if (nmask) {
                    if (qn > kMrQueue - 32) {
                        metal_drain(c, s1, s2, a1, a2, p, queue, qn, out);
                        qn = 0;
                    }
                    if (near)
                        queue[qn + __popc(nmask & lt_mask)] = ((uint32_t)i << 16) | (uint32_t)j;
                    qn += __popc(nmask);
                }
            }
            store_runs(run_b >= 0);
        }
        if (tail != head) metal_apply(c, ring, ring_bin, head, tail - head, p, out);
        if (qn) metal_drain(c, s1, s2, a1, a2, p, queue, qn, out);
    }
}

struct MetalFast {
    FastConst data, model;
};

MetalFast metal_fast(const MetalConst &c) {
    Binning data = c.b, model = c.b;
    data.rmu = model.rmu = 0;
    model.np = c.nmp;
    model.nt = c.nmt;
    model.nbins = c.nm;
    return {make_fast_const(data), make_fast_const(model)};
}

// What the sweeps cover: both forests staged, pixel indices of 16 bits, bins
// that FP32 resolves.
bool metal_runs_covers(const MetalConst &c, const pg_forest_set &s1, const pg_forest_set &s2) {
    const MetalFast f = metal_fast(c);
    return s1.max_pixels <= 65535 && s2.max_pixels <= 65535 &&
           mr_smem(s1.max_pixels, s2.max_pixels).total <= kMaxDynSmem &&
           fast_const_exact(f.data) && fast_const_exact(f.model);
}

int launch_metal_runs(const MetalConst &c, const pg_forest_set &s1, const pg_forest_set &s2,
                      const pg_metal_pixels &a1, const pg_metal_pixels &a2,
                      const int32_t *pair_first, const int32_t *pair_second,
                      const double *pair_angle, int64_t num_pairs, const pg_dmat_sums &out,
                      Scratch *scratch, int num_sms, cudaStream_t stream) {
    const MetalFast fast = metal_fast(c);
    const size_t smem = mr_smem(s1.max_pixels, s2.max_pixels).total;
    cudaError_t err = cudaFuncSetAttribute(
        metal_runs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxDynSmem);
    if (err != cudaSuccess) return check_cuda(err);
    int occ = 0;
    err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, metal_runs_kernel, kMrWarps * 32,
                                                        smem);
    if (err != cudaSuccess) return check_cuda(err);
    if (occ < 1) return PG_ERR_UNSUPPORTED;
    const int64_t grid = std::min<int64_t>((int64_t)num_sms * occ, num_pairs);
    metal_runs_kernel<<<(int)grid, kMrWarps * 32, smem, stream>>>(
        c, fast.data, fast.model, s1, s2, a1, a2, pair_first, pair_second, pair_angle, num_pairs, out,
        scratch, s1.max_pixels, s2.max_pixels);
    return check_cuda(cudaGetLastError());
}

}  // namespace

int launch_metal_dmat(const pg_corr_params &p, const pg_dmat_params &d, double zevol_den,
                      const pg_forest_set &s1, const pg_forest_set &s2,
                      const pg_metal_pixels &a1, const pg_metal_pixels &a2,
                      const int32_t *pair_first, const int32_t *pair_second,
                      const double *pair_angle, int64_t num_pairs, const pg_dmat_sums &out,
                      Scratch *scratch, int num_sms, cudaStream_t stream, bool xcf) {
    if (num_pairs == 0) return PG_OK;
    MetalConst c;
    c.b = make_binning(p);
    c.nmp = d.num_model_bins_r_par;
    c.nmt = d.num_model_bins_r_trans;
    c.nm = c.nmp * c.nmt;
    c.inv_range = 1. / c.b.r_par_range;
    c.inv_rtmax = 1. / c.b.r_trans_max;
    c.inv_zevol_den = 1. / zevol_den;
    c.xcf = xcf;
    if (xcf) {  // r_par is signed and the cross has no half-plate veto
        c.b.x_correlation = 1;
        c.b.remove_shp = 0;
    }
    if (!xcf && metal_runs_covers(c, s1, s2))
        return launch_metal_runs(c, s1, s2, a1, a2, pair_first, pair_second, pair_angle,
                                 num_pairs, out, scratch, num_sms, stream);
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, metal_dmat_kernel, kMdBlock, 0) !=
            cudaSuccess ||
        occ < 1)
        return PG_ERR_CUDA;
    const int64_t grid = std::min<int64_t>((int64_t)num_sms * occ, num_pairs);
    metal_dmat_kernel<<<(int)grid, kMdBlock, 0, stream>>>(c, s1, s2, a1, a2, pair_first,
                                                          pair_second, pair_angle, num_pairs,
                                                          out, scratch);
    return check_cuda(cudaGetLastError());
}

}  // namespace pg
