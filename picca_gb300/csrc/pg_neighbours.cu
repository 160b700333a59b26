// Neighbour search: cf.fill_neighs (py/picca/cf.py:82-135) and
// xcf.fill_neighs (py/picca/xcf.py:71-123).
//
// The reference asks healpy.query_disc for candidate healpix and then keeps
// objects with angle < ang_max; the result is exactly "every object of the
// other set within ang_max" (plus the thingid / RA-order / zerr / r_comov
// filters). A warp owns kNbrQueries query forests and streams the other set
// through shared memory in tiles, a candidate per lane. An FP32 test decides
// almost every pair; the others are decided in FP64 with the reference's
// formula.
#include "pg_internal.cuh"

namespace pg {
namespace {

constexpr int kNbrBlock = 256;   // threads of a CTA
constexpr int kNbrTile = 1024;   // candidates staged at a time
constexpr int kNbrQueries = 4;   // queries per warp: a staged candidate is read once for all
constexpr int kNbrCta = kNbrBlock / 32 * kNbrQueries;  // queries of a CTA
constexpr int kNbrGroupBlock = 256;  // most queries of a block of pg_nbr_groups

struct NbrArgs {
    // query set
    int64_t n1;
    const double *x1, *y1, *z1, *ra1, *dec1, *cosdec1, *zq1, *rfirst1, *rlast1;
    const int64_t *id1;
    // other set
    int64_t n2;
    const double *x2, *y2, *z2, *ra2, *dec2, *zq2, *robj2;
    const int64_t *id2;
    double ang_max;
    float dot_threshold;  // below: certainly farther than ang_max
    float dot_sure;       // above: certainly closer than ang_max
    double dot_far, dot_near;  // the same for the FP64 dot product
    // xcf filters
    double zerr_deg, zerr_kms, r_par_min_f, r_par_max_f;
    int32_t zerr_on, precut_on;
};

// One query against one candidate g of the other set (after the FP32
// prefilter): thingid, exact FP64 angle with the reference's formula, and
// the mode's filters. True when g is a neighbour.
struct Query {
    double x, y, z, ra, dec, cosdec, zq, rfirst, rlast;
    int64_t id;
};

// The FP64 angle (and, for the xcf pre-cut, cos(ang / 2)) is formed only
// where a decision needs it: a pair whose FP32 cosine is above dot_sure is
// within ang_max whatever the rounding, and a pre-cut whose FP32 estimate is
// farther than its error bound from the limit has the exact outcome. Both
// shortcuts give the FP64 decision itself, so the lists are unchanged; they
// remove the FP64 trigonometry that otherwise runs for almost every
// candidate (a warp executes it when any of its lanes needs it).
template <int MODE>
__device__ __forceinline__ bool is_neighbour(const NbrArgs &a, const Query &q, int64_t g,
                                             float dot) {
    if (a.id2[g] == q.id) return false;
    double ang = -1.0;
    auto exact_angle = [&]() {
        if (ang < 0.0)
            ang = angle_between(q.x, q.y, q.z, q.ra, q.dec, q.cosdec, a.x2[g], a.y2[g], a.z2[g],
                                a.ra2[g], a.dec2[g]);
        return ang;
    };
    if (!(dot > a.dot_sure)) {
        // the FP64 dot product decides unless it is within rounding of
        // cos(ang_max): the arc cosine of its clipped value moves by less than
        // 1e-9 rad for 1e-12 of it, far more than its own rounding, and the
        // flat-sky branch (below 2 arcsec) only takes pairs that are near
        const double d64 = __dadd_rn(
            __dadd_rn(__dmul_rn(a.x2[g], q.x), __dmul_rn(a.y2[g], q.y)), __dmul_rn(a.z2[g], q.z));
        if (d64 < a.dot_far) return false;
        if (!(d64 > a.dot_near) && !(exact_angle() < a.ang_max)) return false;
    }
    if (MODE == 1 && !(q.ra > a.ra2[g])) return false;
    if (MODE == 2) {
        if (a.zerr_on) {
            const double ang_deg = __dmul_rn(180.0 / kPi, exact_angle());
            const double zq = a.zq2[g];
            const double z_qq = __dmul_rn(0.5, __dadd_rn(q.zq, zq));
            double dv = fabs(__dsub_rn(q.zq, zq)) / __dadd_rn(1.0, z_qq);
            dv = __dmul_rn(dv, kSpeedLight);
            if (ang_deg < a.zerr_deg && dv < a.zerr_kms) return false;
        }
        if (a.precut_on) {
            const double robj = a.robj2[g];
            const double u1 = __dsub_rn(q.rfirst, robj), u2 = __dsub_rn(q.rlast, robj);
            // cos(ang / 2) = sqrt(x), x = (1 + cos ang) / 2, from the FP32
            // cosine (within 4e-7): for x >= 1/4 (ang <= 120 deg) its
            // relative error is below 1e-6, and a limit farther than 4e-6
            // of |u| from the product is decided from it; otherwise (and
            // for wider angles) the FP64 cos(ang / 2) decides
            const float xh = 0.5f * (1.f + dot);
            const bool est = xh >= 0.25f;
            const float ch = sqrtf(fmaxf(xh, 0.f));
            const double e1 = fabs(u1) * 4e-6 + 1e-9, e2 = fabs(u2) * 4e-6 + 1e-9;
            const double p1 = u1 * (double)ch, p2 = u2 * (double)ch;
            bool lo_ok, hi_ok;
            if (est && p1 < a.r_par_max_f - e1) hi_ok = true;
            else if (est && p1 > a.r_par_max_f + e1) hi_ok = false;
            else hi_ok = __dmul_rn(u1, cos(exact_angle() / 2.)) < a.r_par_max_f;
            if (!hi_ok) return false;
            if (est && p2 > a.r_par_min_f + e2) lo_ok = true;
            else if (est && p2 < a.r_par_min_f - e2) lo_ok = false;
            else lo_ok = __dmul_rn(u2, cos(exact_angle() / 2.)) > a.r_par_min_f;
            if (!lo_ok) return false;
        }
    }
    return true;
}

// The FP64 decision of a pair the FP32 test left open (rare: its own
// function keeps its registers out of the scan).
template <int MODE>
__device__ __noinline__ bool decide_fp64(const NbrArgs &a, int64_t f, int64_t g, float dot) {
    Query q{a.x1[f], a.y1[f], a.z1[f], a.ra1[f], a.dec1[f], a.cosdec1[f], 0, 0, 0, a.id1[f]};
    if (MODE == 2) {
        q.zq = a.zq1[f];
        q.rfirst = a.rfirst1[f];
        q.rlast = a.rlast1[f];
    }
    return is_neighbour<MODE>(a, q, g, dot);
}

// One query of a warp as the FP32 test sees it (the same in every lane).
struct Query32 {
    float x, y, z;
    float u, v;       // mode 1: RA; mode 2: first and last distance of the forest
    float err;        // FP32 rounding of u (and v), with margin
    unsigned id;      // low half of the thingid
};

// A candidate of the tile: FP32 unit vector and the mode's scalar (RA,
// quasar distance), and the low half of its thingid.
struct NbrTile {
    float4 v[kNbrTile];
    unsigned id[kNbrTile];
};

enum NbrDecision { NBR_OUT, NBR_IN, NBR_UNSURE };

// FP32 decision of one pair. Every comparison that decides keeps a margin
// over the FP32 rounding of its operands, so that it is the FP64 decision;
// whatever it cannot decide (equal low halves of the thingid, NaN, the
// redshift-error cut) is left to is_neighbour. The distance pre-cut of the
// cross (xcf.py:96-103): cos(ang / 2) = sqrt(x), x = (1 + cos ang) / 2, from
// the FP32 cosine (within 4e-7) has a relative error below 1e-6 for
// x >= 1/4 (ang <= 120 deg); u = r - r_obj carries the FP32 rounding of both
// distances.
template <int MODE>
__device__ __forceinline__ NbrDecision nbr_decide(const NbrArgs &a, const Query32 &q,
                                                  const float4 &t, unsigned id, float rp_max,
                                                  float rp_min, float rp_err) {
    const float dot = __fmaf_rn(q.z, t.z, __fmaf_rn(q.y, t.y, q.x * t.x));
    if (dot <= a.dot_threshold) return NBR_OUT;
    bool sure = dot > a.dot_sure && id != q.id;
    if (MODE == 1) {
        const float d = q.u - t.w, m = q.err + 2e-7f * fabsf(t.w);
        if (d < -m) return NBR_OUT;
        sure &= d > m;
    }
    if (MODE == 2) {
        if (a.zerr_on) sure = false;
        if (a.precut_on) {
            const float xh = 0.5f * (1.f + dot);
            const float ch = sqrtf(fmaxf(xh, 0.f));
            const float m = q.err + 2e-7f * fabsf(t.w) + rp_err;
            const float u1 = q.u - t.w, u2 = q.v - t.w;
            const float p1 = u1 * ch, p2 = u2 * ch;
            const float e1 = __fmaf_rn(fabsf(u1), 5e-6f, m), e2 = __fmaf_rn(fabsf(u2), 5e-6f, m);
            const bool est = xh >= 0.25f;
            if (est && (p1 > rp_max + e1 || p2 < rp_min - e2)) return NBR_OUT;
            sure &= est && p1 < rp_max - e1 && p2 > rp_min + e2;
        }
    }
    return sure ? NBR_IN : NBR_UNSURE;
}

// MODE 0: cf cross (two sets), 1: cf auto, 2: xcf.
//
// A CTA takes kNbrCta consecutive queries (GROUPED: of one group of the query
// set) and scans the other set (GROUPED: only the candidate groups, object
// ranges in ascending order; the candidate lists are a superset built from
// bounding caps). A warp tests 32 candidates against its queries at a time,
// a candidate per lane, so the lanes' hits come out in increasing index
// order: the ballot gives each its place and the index is written coalesced.
// Bound by FP32 issue (the FP64 pipe of this chip has 1/64 of the FP32 lanes,
// which is why no FP64 operation is left in the common path). With a thread
// per query, 9,000 forests filled 45 CTAs and formed the pre-cut in FP64:
// 11.6 ms a pass against 13,500 quasars, and 0.45 ms now (12,000 forests in
// the auto-correlation: 4.2 ms and 0.33 ms).
template <int MODE, bool GROUPED>
__global__ void __launch_bounds__(kNbrBlock) neighbours_kernel(
    const __grid_constant__ NbrArgs a, const __grid_constant__ pg_nbr_groups gr,
    int64_t *counts, const int64_t *offsets, int32_t *index) {
    __shared__ NbrTile tile;
    const int lane = threadIdx.x & 31;
    int64_t first, end;
    int c0 = 0, c1 = 1;
    if (GROUPED) {
        const int grp = gr.block_group[blockIdx.x];
        first = gr.block_first[blockIdx.x] + (int64_t)blockIdx.y * kNbrCta;
        end = gr.block_end[blockIdx.x];
        c0 = gr.cand_offsets[grp];
        c1 = gr.cand_offsets[grp + 1];
    } else {
        first = (int64_t)blockIdx.x * kNbrCta;
        end = a.n1;
    }
    if (first >= end) return;
    const int64_t f0 = first + (threadIdx.x >> 5) * kNbrQueries;
    const float rp_max = (float)a.r_par_max_f, rp_min = (float)a.r_par_min_f;
    const float rp_err = 1e-6f + 2e-7f * (fabsf(rp_max) + fabsf(rp_min));
    Query32 q[kNbrQueries];
    int64_t out[kNbrQueries];
    int n[kNbrQueries];
#pragma unroll
    for (int k = 0; k < kNbrQueries; ++k) {
        // past the end: any valid query (not scanned, see nq)
        const int64_t f = f0 + k < end ? f0 + k : end - 1;
        q[k].x = (float)a.x1[f];
        q[k].y = (float)a.y1[f];
        q[k].z = (float)a.z1[f];
        q[k].id = (unsigned)a.id1[f];
        q[k].u = q[k].v = 0.f;
        if (MODE == 1) q[k].u = (float)a.ra1[f];
        if (MODE == 2) {
            q[k].u = (float)a.rfirst1[f];
            q[k].v = (float)a.rlast1[f];
        }
        q[k].err = 2e-7f * fmaxf(fabsf(q[k].u), fabsf(q[k].v)) + 1e-30f;
        out[k] = offsets ? offsets[f] : 0;
        n[k] = 0;
    }
    const int nq = f0 >= end ? 0 : (end - f0 < kNbrQueries ? (int)(end - f0) : kNbrQueries);
    for (int c = c0; c < c1; ++c) {
        int64_t lo = 0, hi = a.n2;
        if (GROUPED) {
            const int g2 = gr.cand_groups[c];
            lo = gr.start2[g2];
            hi = gr.start2[g2 + 1];
        }
        for (int64_t t0 = lo; t0 < hi; t0 += kNbrTile) {
            const int tn = (int)min((int64_t)kNbrTile, hi - t0);
            __syncthreads();
            for (int k = threadIdx.x; k < tn; k += blockDim.x) {
                const int64_t g = t0 + k;
                float w = 0.f;
                if (MODE == 1) w = (float)a.ra2[g];
                if (MODE == 2) w = (float)a.robj2[g];
                tile.v[k] = make_float4((float)a.x2[g], (float)a.y2[g], (float)a.z2[g], w);
                tile.id[k] = (unsigned)a.id2[g];
            }
            __syncthreads();
            for (int k0 = 0; k0 < tn; k0 += 32) {
                const int k = k0 + lane;
                const bool have = k < tn;
                const float4 t = tile.v[have ? k : 0];
                const unsigned id = tile.id[have ? k : 0];
#pragma unroll
                for (int r = 0; r < kNbrQueries; ++r) {
                    if (r >= nq) break;
                    NbrDecision d = have ? nbr_decide<MODE>(a, q[r], t, id, rp_max, rp_min, rp_err)
                                         : NBR_OUT;
                    if (d == NBR_UNSURE) {
                        const float dot =
                            __fmaf_rn(q[r].z, t.z, __fmaf_rn(q[r].y, t.y, q[r].x * t.x));
                        d = decide_fp64<MODE>(a, f0 + r, t0 + k, dot) ? NBR_IN : NBR_OUT;
                    }
                    const unsigned m = __ballot_sync(0xffffffffu, d == NBR_IN);
                    if (offsets && d == NBR_IN)
                        index[out[r] + n[r] + __popc(m & ((1u << lane) - 1u))] = (int32_t)(t0 + k);
                    n[r] += __popc(m);
                }
            }
        }
    }
    if (!offsets) {
#pragma unroll
        for (int r = 0; r < kNbrQueries; ++r)
            if (r < nq && lane == r) counts[f0 + r] = n[r];
    }
}

template <int MODE>
int launch_neighbours(const NbrArgs &a, const pg_nbr_groups *groups, int64_t *counts,
                      const int64_t *offsets, int32_t *index, cudaStream_t stream) {
    if (a.n1 == 0) return PG_OK;
    if (groups) {
        if (groups->num_blocks <= 0) return PG_OK;
        const dim3 grid((unsigned)groups->num_blocks, kNbrGroupBlock / kNbrCta);
        neighbours_kernel<MODE, true><<<grid, kNbrBlock, 0, stream>>>(a, *groups, counts, offsets,
                                                                      index);
    } else {
        const dim3 grid((unsigned)((a.n1 + kNbrCta - 1) / kNbrCta));
        neighbours_kernel<MODE, false><<<grid, kNbrBlock, 0, stream>>>(a, pg_nbr_groups{}, counts,
                                                                       offsets, index);
    }
    return check_cuda(cudaGetLastError());
}

float dot_threshold(double ang_max) {
    // below ~1e-3 rad the 1e-5 cosine margin is no longer small; test all
    if (ang_max < 1e-3 || ang_max >= kPi) return -2.0f;
    return (float)cos(ang_max) - 1e-5f;
}

// FP32 unit-vector cosines are accurate to ~4e-7: above this value the FP64
// angle is below ang_max (2 = never: decide every pair in FP64)
float dot_sure(double ang_max) {
    if (ang_max < 1e-3 || ang_max >= kPi) return 2.0f;
    return (float)cos(ang_max) + 1e-5f;
}

// Limits of the FP64 dot product (see is_neighbour); never decided by it
// where the FP32 tests are off.
void set_dot_limits(NbrArgs &a) {
    a.dot_threshold = dot_threshold(a.ang_max);
    a.dot_sure = dot_sure(a.ang_max);
    const bool off = a.dot_sure > 1.5f;
    a.dot_far = off ? -INFINITY : cos(a.ang_max) - 1e-12;
    a.dot_near = off ? INFINITY : cos(a.ang_max) + 1e-12;
}

}  // namespace

int launch_cf_neighbours(const pg_corr_params &p, const pg_forest_set &s1, const pg_forest_set &s2,
                         bool auto_mode, const pg_nbr_groups *groups, int64_t *counts,
                         const int64_t *offsets, int32_t *index, cudaStream_t stream) {
    NbrArgs a{};
    a.n1 = s1.num;
    a.x1 = s1.x_cart; a.y1 = s1.y_cart; a.z1 = s1.z_cart;
    a.ra1 = s1.ra; a.dec1 = s1.dec; a.cosdec1 = s1.cos_dec; a.id1 = s1.thingid;
    a.n2 = s2.num;
    a.x2 = s2.x_cart; a.y2 = s2.y_cart; a.z2 = s2.z_cart;
    a.ra2 = s2.ra; a.dec2 = s2.dec; a.id2 = s2.thingid;
    a.ang_max = p.ang_max;
    set_dot_limits(a);
    return auto_mode ? launch_neighbours<1>(a, groups, counts, offsets, index, stream)
                     : launch_neighbours<0>(a, groups, counts, offsets, index, stream);
}

int launch_xcf_neighbours(const pg_corr_params &p, const pg_forest_set &forests,
                          const pg_forest_set &objs, const pg_nbr_groups *groups,
                          int64_t *counts, const int64_t *offsets, int32_t *index,
                          cudaStream_t stream) {
    NbrArgs a{};
    a.n1 = forests.num;
    a.x1 = forests.x_cart; a.y1 = forests.y_cart; a.z1 = forests.z_cart;
    a.ra1 = forests.ra; a.dec1 = forests.dec; a.cosdec1 = forests.cos_dec;
    a.zq1 = forests.z_qso; a.rfirst1 = forests.r_first; a.rlast1 = forests.r_last;
    a.id1 = forests.thingid;
    a.n2 = objs.num;
    a.x2 = objs.x_cart; a.y2 = objs.y_cart; a.z2 = objs.z_cart;
    a.ra2 = objs.ra; a.dec2 = objs.dec; a.zq2 = objs.z_qso; a.robj2 = objs.obj_r_comov;
    a.id2 = objs.thingid;
    a.ang_max = p.ang_max;
    set_dot_limits(a);
    a.zerr_on = !isnan(p.zerr_cut_deg) && !isnan(p.zerr_cut_kms);
    a.zerr_deg = p.zerr_cut_deg;
    a.zerr_kms = p.zerr_cut_kms;
    a.precut_on = !p.ang_correlation;
    const double f = p.rmu_binning ? p.r_trans_max : 1;
    a.r_par_max_f = p.r_par_max * f;
    a.r_par_min_f = p.r_par_min * f;
    return launch_neighbours<2>(a, groups, counts, offsets, index, stream);
}

}  // namespace pg
