// All-FP64 sums of the auto-correlation, of two delta fields and (second half)
// of deltas and quasars with the pair decisions taken in FP32 (PG_MODE_FP64 on the (r_par, r_trans)
// geometry). The accepted pairs, bins and counts are those of the all-FP64
// loop: a pair near a bin edge or a cut is queued and decided with the
// reference's FP64 expressions (guard bands: pg_pairs_common.cuh), and every
// term that is summed is formed and added in FP64.
//
// Bound: the FP64 pipe, which has 1/64 of the FP32 lanes here (16 cycles a
// warp instruction and SM). The all-FP64 loop (pg_pairs_fp64.cu) spends about
// 45 of its operations on every candidate (two divisions, two floors, the
// comparisons) and adds five sums per pair by compare-and-swap on shared
// memory; this kernel spends nine on an accepted pair and none on a rejected
// one. As in cf_xi_diag_kernel (pg_pairs_fast.cu) the pairs are swept along
// diagonals, a lane per diagonal, so that consecutive accepted pairs of a
// lane share their bin for tens of steps: they are summed in registers as a
// run, and a run goes to the FP64 row of the healpix through a ring that
// applies 32 runs at a time. The rows are global memory (the additions do not
// return, so nothing waits for them), which leaves shared memory to the
// staged pixels and lets several CTAs share one forest. 331 forests
// (1.9e9 candidate pairs, 50 x 50 bins): 125 ms with the all-FP64 loop, 12.4 ms
// here.
#include <algorithm>

#include "pg_internal.cuh"
#include "pg_pairs_common.cuh"

namespace pg {
namespace {

constexpr int kR64Warps = 8;
constexpr int kR64Chunk = 64;   // forest-2 pixels staged per warp at a time
constexpr int kR64Ring = 64;    // runs held per warp (<= 31 + 32)
constexpr int kR64Queue = 128;  // FP64 re-decision entries per warp

// One forest's pixels in FP64 (structure of arrays in shared memory).
struct Pix64 {
    double *r, *m, *z, *w, *dw;
};

__device__ __forceinline__ Pix64 pix64(void *base, int n) {
    double *d = static_cast<double *>(base);
    return {d, d + n, d + 2 * n, d + 3 * n, d + 4 * n};
}

// Byte offsets: forest 1 as float4 (rho, dist_m, z, w) and Pix64; then per
// warp the staged forest-2 chunk in the same two forms (float4 nB, t, z, w),
// the run ring (five sums, then bin and count), the re-decision queue and the
// forest-1 zerr veto bits.
struct R64Smem {
    size_t p1, q1, warps, per_warp, buf, q2, ring, ring_bin, queue, veto, total;
};

__host__ __device__ inline R64Smem r64_smem(int max_pix1) {
    R64Smem l;
    const size_t mp = (size_t)((max_pix1 + 1) & ~1);
    l.p1 = 0;
    l.q1 = l.p1 + mp * 16;
    l.warps = l.q1 + mp * 40;
    l.buf = 0;
    l.q2 = l.buf + (size_t)kR64Chunk * 16;
    l.ring = l.q2 + (size_t)kR64Chunk * 40;
    l.ring_bin = l.ring + (size_t)kR64Ring * 40;
    l.queue = l.ring_bin + (size_t)kR64Ring * 8;
    l.veto = l.queue + (size_t)kR64Queue * 4;
    l.per_warp = (l.veto + ((mp + 31) / 32) * 4 + 15) & ~(size_t)15;
    l.total = l.warps + kR64Warps * l.per_warp;
    return l;
}

__device__ __forceinline__ void add_row(const pg_xi_rows &out, size_t at, double xi, double we,
                                        double rp, double rt, double z, int count) {
    atomicAdd(&out.xi[at], xi);
    atomicAdd(&out.weights[at], we);
    atomicAdd(&out.r_par[at], rp);
    atomicAdd(&out.r_trans[at], rt);
    atomicAdd(&out.z[at], z);
    atomicAdd((unsigned long long *)&out.num_pairs[at], (unsigned long long)count);
}

// Queued (i, j) pairs: the reference's decision and terms.
__device__ __noinline__ void r64_drain(const Binning &b, const pg_forest_set &s1,
                                       const pg_forest_set &s2, const CfPairCtx &ctx,
                                       const uint32_t *queue, int count, const pg_xi_rows &out,
                                       size_t row, Scratch *scratch) {
    __syncwarp();
    const int lane = threadIdx.x & 31;
    for (int e = lane; e < count; e += 32) {
        const uint32_t entry = queue[e];
        const int64_t ia = ctx.a0 + (entry >> 16), jb = ctx.b0 + (entry & 0xFFFF);
        double r_par, r_trans, z;
        const int64_t bin = cf_pair_bin(b, s1.z[ia], s1.r_comov[ia], s1.dist_m[ia], s2.z[jb],
                                        s2.r_comov[jb], s2.dist_m[jb], ctx.ang, ctx.c, ctx.s,
                                        ctx.shp, r_par, r_trans, z);
        if (bin < 0) continue;
        if (bin >= b.nbins) {
            report_error(scratch, PG_ERR_BIN_RANGE, (int32_t)bin);
            continue;
        }
        const double w1 = s1.weights[ia], w2 = s2.weights[jb];
        const double w12 = __dmul_rn(w1, w2);
        const double dw12 = __dmul_rn(__dmul_rn(s1.delta[ia], w1), __dmul_rn(s2.delta[jb], w2));
        add_row(out, row + bin, dw12, w12, __dmul_rn(r_par, w12), __dmul_rn(r_trans, w12),
                __dmul_rn(z, w12), 1);
    }
    if (lane == 0) atomicAdd(&scratch->rechecked_pairs, (unsigned long long)count);
    __syncwarp();
}

// Adds n (<= 32) runs of the ring, from position head, to the row.
__device__ __forceinline__ void r64_apply(const double *ring, const uint2 *ring_bin, int head,
                                          int n, double c, double s, const pg_xi_rows &out,
                                          size_t row) {
    __syncwarp();
    const int lane = threadIdx.x & 31;
    if (lane < n) {
        const int e = (head + lane) & (kR64Ring - 1);
        const uint2 u = ring_bin[e];
        add_row(out, row + u.x, ring[e], ring[kR64Ring + e],
                __dmul_rn(ring[2 * kR64Ring + e], c), __dmul_rn(ring[3 * kR64Ring + e], s),
                __dmul_rn(ring[4 * kR64Ring + e], 0.5), (int)u.y);
    }
    __syncwarp();
}

// AUTO, EXTRA, LOWX as in cf_xi_diag_kernel. A work unit is a slice of one
// forest's neighbours: with fewer forests than a few per CTA a forest is
// shared by several CTAs (its rows are global).
template <bool AUTO, bool EXTRA, bool LOWX>
__global__ void __launch_bounds__(kR64Warps * 32, 2) cf_xi_runs64_kernel(
    const __grid_constant__ Binning b, const __grid_constant__ FastConst fc,
    const __grid_constant__ pg_forest_set s1, const __grid_constant__ pg_forest_set s2,
    const int64_t *__restrict__ nbr_offsets, const int32_t *__restrict__ nbr_index,
    const double *__restrict__ nbr_angle, const int32_t *__restrict__ work_order,
    int64_t num_work, int slices, const __grid_constant__ pg_xi_rows out, Scratch *scratch,
    int max_pix1) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int64_t unit_slot;
    __shared__ unsigned max_rho_bits;
    __shared__ unsigned long long nbr_next;
    __shared__ CfPairCtx pair_ctx[kR64Warps];
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const unsigned lt_mask = (1u << lane) - 1u;
    const R64Smem L = r64_smem(max_pix1);
    const int mp = (max_pix1 + 1) & ~1;
    float4 *p1 = reinterpret_cast<float4 *>(smem + L.p1);
    const Pix64 q1 = pix64(smem + L.q1, mp);
    unsigned char *wbase = smem + L.warps + (size_t)warp * L.per_warp;
    float4 *buf = reinterpret_cast<float4 *>(wbase + L.buf);
    const Pix64 q2 = pix64(wbase + L.q2, kR64Chunk);
    double *ring = reinterpret_cast<double *>(wbase + L.ring);
    uint2 *ring_bin = reinterpret_cast<uint2 *>(wbase + L.ring_bin);
    uint32_t *queue = reinterpret_cast<uint32_t *>(wbase + L.queue);
    uint32_t *veto1 = reinterpret_cast<uint32_t *>(wbase + L.veto);
    CfPairCtx &ctx = pair_ctx[warp];
    const unsigned np = fc.np, nt = fc.nt;
    const float t_end = (float)nt + 1.f;  // x_tr' at or above this: rejected, a bin of margin
    // accepted range of p with one bin of margin each side
    const float pmin_f = fc.pc - 0.5f;
    const float p_hi = pmin_f + (float)np + 1.f;
    const float p_lo = AUTO ? -p_hi : pmin_f - 1.f;

    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) {
            unit_slot = atomicAdd(&scratch->work_counter, 1);
            max_rho_bits = 0u;
        }
        __syncthreads();
        const int64_t unit = unit_slot;
        if (unit >= num_work * slices) break;
        const int64_t item = unit / slices;
        const int slice = (int)(unit - item * slices);
        const int64_t f1 = work_order ? work_order[item] : item;
        const size_t row = (size_t)s1.row[f1] * b.nbins;
        const int64_t a0 = s1.pix_offset[f1];
        const int64_t n1_64 = s1.pix_offset[f1 + 1] - a0;
        const int64_t nk = nbr_offsets[f1 + 1] - nbr_offsets[f1];
        const int64_t k_lo = nbr_offsets[f1] + nk * slice / slices;
        const int64_t k_hi = nbr_offsets[f1] + nk * (slice + 1) / slices;
        if (threadIdx.x == 0) {
            nbr_next = (unsigned long long)k_lo;
            if (slice == 0) atomicAdd(&scratch->work_items, 1ull);
        }
        if (n1_64 > max_pix1) {
            if (threadIdx.x == 0) report_error(scratch, PG_ERR_UNSUPPORTED, (int32_t)f1);
            continue;
        }
        const int n1 = (int)n1_64;
        if (n1 < 1 || k_lo == k_hi) continue;
        const double r_ref = reference_distance(s1.r_comov[a0 + n1 / 2], &max_rho_bits);
        // forest 1: FP32 relative to its middle pixel, and FP64
        bool ordered = true;
        float local_max = 0.f;
        for (int i = threadIdx.x; i < n1; i += blockDim.x) {
            const double w = s1.weights[a0 + i], r = s1.r_comov[a0 + i], m = s1.dist_m[a0 + i];
            const double z = s1.z[a0 + i];
            const float rho = (float)(r - r_ref), d = (float)m;
            p1[i] = make_float4(rho, d, (float)z, weight32(w));
            q1.r[i] = r;
            q1.m[i] = m;
            q1.z[i] = z;
            q1.w[i] = w;
            q1.dw[i] = __dmul_rn(s1.delta[a0 + i], w);
            local_max = fmaxf(local_max, fabsf(rho));
            if (i + 1 < n1)
                ordered &= (float)(s1.r_comov[a0 + i + 1] - r_ref) >= rho &&
                           (float)s1.dist_m[a0 + i + 1] >= d;
        }
        if (local_max > 0.f) atomicMax(&max_rho_bits, __float_as_uint(local_max));
        bool sorted1 = __syncthreads_and(ordered) != 0;
        const ParGuard pg = par_guard_exact(&fc, __uint_as_float(max_rho_bits));
        sorted1 &= !pg.wide;
        const float h_par = pg.h_par, low_clamp = pg.low_clamp, h_tr = fc.h_tr, pc = fc.pc;
        const double x1 = s1.x_cart[f1], y1 = s1.y_cart[f1], zc1 = s1.z_cart[f1];
        for (;;) {
            unsigned long long kt = 0;
            if (lane == 0) kt = atomicAdd(&nbr_next, 1ull);
            const int64_t k = (int64_t)__shfl_sync(0xffffffffu, kt, 0);
            if (k >= k_hi) break;
            const int64_t g = nbr_index[k];
            const int64_t b0 = s2.pix_offset[g];
            const int64_t n2_64 = s2.pix_offset[g + 1] - b0;
            if (n2_64 > 65535) {
                if (lane == 0) report_error(scratch, PG_ERR_UNSUPPORTED, (int32_t)g);
                continue;
            }
            const int n2 = (int)n2_64;
            const double ang =
                nbr_angle ? nbr_angle[k]
                          : angle_between(x1, y1, zc1, s1.ra[f1], s1.dec[f1], s1.cos_dec[f1],
                                          s2.x_cart[g], s2.y_cart[g], s2.z_cart[g], s2.ra[g],
                                          s2.dec[g]);
            const double c = cos(ang / 2), s = sin(ang / 2);
            bool shp = false, zerr_pair = false;
            if (EXTRA) {
                if (b.remove_shp) {
                    const int64_t fb1 = s1.fiberid[f1], fb2 = s2.fiberid[g];
                    shp = (s1.plate[f1] == s2.plate[g]) &&
                          ((fb1 <= 500 && fb2 <= 500) || (fb1 > 500 && fb2 > 500));
                }
                zerr_pair = b.zerr_on && (ang < b.zerr_ang);
            }
            __syncwarp();
            if (lane == 0) {
                ctx.a0 = a0;
                ctx.b0 = b0;
                ctx.ang = ang;
                ctx.c = c;
                ctx.s = s;
                ctx.shp = shp;
            }
            if (EXTRA && zerr_pair) {
                // forest-1 pixels vetoed against quasar 2 (py/picca/cf.py:321-328)
                const double zq2 = s2.z_qso[g];
                for (int i0 = 0; i0 < n1; i0 += 32) {
                    const int i = i0 + lane;
                    const bool v = i < n1 && zerr_veto(q1.z[i], zq2, b.zerr_kms);
                    const unsigned m = __ballot_sync(0xffffffffu, v);
                    if (lane == 0) veto1[i0 >> 5] = m;
                }
            }
            __syncwarp();
            const float cp = (float)(c * fc.inv_p), st = (float)(s * fc.inv_t);
            int head = 0, tail = 0, qn = 0;  // run ring and queue (warp-uniform)
            for (int jc = 0; jc < n2; jc += kR64Chunk) {
                const int jn = min(kR64Chunk, n2 - jc);
                bool ordered2 = true, valid2 = true;
                __syncwarp();
                for (int jl = lane; jl < jn; jl += 32) {
                    const int64_t jj = b0 + jc + jl;
                    const double w2 = s2.weights[jj], r2 = s2.r_comov[jj], m2 = s2.dist_m[jj];
                    const double z2 = s2.z[jj];
                    bool ok = w2 != 0;
                    if (EXTRA && zerr_pair && ok) ok = !zerr_veto(z2, s1.z_qso[f1], b.zerr_kms);
                    const float rho2 = (float)(r2 - r_ref), d2 = (float)m2;
                    buf[jl] = make_float4(-__fmul_rn(cp, rho2),
                                          ok ? __fmaf_rn(st, d2, -0.5f) : kFar, (float)z2,
                                          ok ? weight32(w2) : 0.f);
                    q2.r[jl] = r2;
                    q2.m[jl] = m2;
                    q2.z[jl] = z2;
                    q2.w[jl] = w2;
                    q2.dw[jl] = __dmul_rn(s2.delta[jj], w2);
                    valid2 &= ok;
                    if (jl + 1 < jn)
                        ordered2 &= (float)(s2.r_comov[jj + 1] - r_ref) >= rho2 &&
                                    (float)s2.dist_m[jj + 1] >= d2;
                }
                ordered2 = __all_sync(0xffffffffu, ordered2);
                valid2 = __all_sync(0xffffffffu, valid2);
                __syncwarp();
                // band of diagonals holding every pair within one bin of the
                // accepted r_par range (both forests ordered; else all)
                int d_lo = jc - (n1 - 1), d_hi = jc + jn;
                if (sorted1 && ordered2) {
                    int lo = INT_MAX, hi = INT_MIN;
                    for (int i = lane; i < n1; i += 32) {
                        const float a = __fmul_rn(cp, p1[i].x);
                        const int j1 = count_leading<false>(buf, jn, p_hi - a);
                        const int j2 = count_leading<true>(buf, jn, p_lo - a);
                        if (j1 < j2) {
                            lo = min(lo, jc + j1 - i);
                            hi = max(hi, jc + j2 - i);
                        }
                    }
                    d_lo = __reduce_min_sync(0xffffffffu, lo);
                    d_hi = __reduce_max_sync(0xffffffffu, hi);
                }
                const bool t_trim = sorted1 && ordered2 && valid2 && st > 0.f;
                for (int d0 = d_lo; d0 < d_hi; d0 += 32) {
                    const int d = d0 + lane;
                    int ia = max(0, jc - d), ib = min(n1, jc + jn - d);
                    if (d >= d_hi) ib = ia;
                    const int joff = d - jc;
                    if (t_trim && ia < ib) {
                        int lo = ia, hi = ib;
                        while (lo < hi) {
                            const int mid = (lo + hi) >> 1;
                            if (__fmaf_rn(st, p1[mid].y, buf[mid + joff].y) < t_end) lo = mid + 1;
                            else hi = mid;
                        }
                        ib = lo;
                    }
                    const int sa = ia + joff, sb = ib + joff;
                    const int g_lo = __reduce_min_sync(0xffffffffu, ia < ib ? sa : INT_MAX);
                    const int g_hi = __reduce_max_sync(0xffffffffu, ia < ib ? sb : INT_MIN);
                    if (g_lo >= g_hi) continue;
                    unsigned run_bin = 0xFFFFFFFFu;
                    int run_n = 0;
                    double r_xi = 0., r_we = 0., r_rp = 0., r_rt = 0., r_z = 0.;
                    auto store_runs = [&](bool flag) {
                        const unsigned m = __ballot_sync(0xffffffffu, flag);
                        if (flag) {
                            const int pos = (tail + __popc(m & lt_mask)) & (kR64Ring - 1);
                            ring[pos] = r_xi;
                            ring[kR64Ring + pos] = r_we;
                            ring[2 * kR64Ring + pos] = r_rp;
                            ring[3 * kR64Ring + pos] = r_rt;
                            ring[4 * kR64Ring + pos] = r_z;
                            ring_bin[pos] = make_uint2(run_bin, (unsigned)run_n);
                        }
                        tail += __popc(m);
                        if (tail - head >= 32) {
                            r64_apply(ring, ring_bin, head, 32, c, s, out, row);
                            head += 32;
                        }
                    };
                    for (int js = g_lo; js < g_hi; ++js) {
                        bool in = (js >= sa) & (js < sb);
                        const int i = in ? js - joff : 0;
                        if (EXTRA && zerr_pair && in) in = ((veto1[i >> 5] >> (i & 31)) & 1u) == 0u;
                        const float4 f1p = p1[i];
                        const float4 f2p = buf[js];
                        const float pp = __fmaf_rn(cp, f1p.x, f2p.x);
                        const float v = fabsf(pp);
                        const float pv = AUTO ? v : pp;
                        const float xt = __fmaf_rn(st, f1p.y, f2p.y);
                        const float xp = LOWX ? clamp_low(pv - pc, low_clamp) : pv - pc;
                        float fp, ft;
                        const unsigned ip = round_rem(xp, fp), it = round_rem(xt, ft);
                        bool near = (fabsf(fp) > h_par) | (fabsf(ft) > h_tr);
                        in &= (f1p.w != 0.f) & (f2p.w != 0.f);
                        bool ok = (ip < np) & (it < nt);
                        if (EXTRA) {
                            const float zs = f1p.z + f2p.z;
                            // guard_z covers z1 + z2 up to 20
                            const float gz = fc.guard_z * fmaxf(1.f, 0.05f * fabsf(zs));
                            if (shp) {
                                near |= fabsf(v - 1.f) < pg.guard_v;
                                ok &= !(v < 1.f);
                            }
                            if (b.zmin_on) {
                                near |= fabsf(zs - fc.zmin2) < gz;
                                ok &= !(zs < fc.zmin2);
                            }
                            if (b.zmax_on) {
                                near |= fabsf(zs - fc.zmax2) < gz;
                                ok &= !(zs > fc.zmax2);
                            }
                        }
                        near &= in;
                        const bool acc = in & ok & !near;
                        const unsigned bin = ip * nt + it;
                        const bool brk = acc & (bin != run_bin);
                        const bool flush = brk & (run_n > 0);
                        if (__any_sync(0xffffffffu, flush)) {
                            store_runs(flush);
                            if (flush) {
                                run_n = 0;
                                r_xi = r_we = r_rp = r_rt = r_z = 0.;
                            }
                        }
                        if (brk) run_bin = bin;
                        if (acc) {
                            // nine FP64 operations; cos, sin and 1/2 are
                            // applied once per run
                            const double w12 = __dmul_rn(q1.w[i], q2.w[js]);
                            const double dr = __dsub_rn(q1.r[i], q2.r[js]);
                            r_we = __dadd_rn(r_we, w12);
                            r_xi = fma(q1.dw[i], q2.dw[js], r_xi);
                            r_rp = fma(AUTO ? fabs(dr) : dr, w12, r_rp);
                            r_rt = fma(__dadd_rn(q1.m[i], q2.m[js]), w12, r_rt);
                            r_z = fma(__dadd_rn(q1.z[i], q2.z[js]), w12, r_z);
                            ++run_n;
                        }
                        const unsigned nmask = __ballot_sync(0xffffffffu, near);
                        if (nmask) {
                            if (qn > kR64Queue - 32) {
                                r64_drain(b, s1, s2, ctx, queue, qn, out, row, scratch);
                                if (lane == 0) atomicAdd(&scratch->recheck_overflows, 1ull);
                                qn = 0;
                            }
                            if (near)
                                queue[qn + __popc(nmask & lt_mask)] =
                                    ((uint32_t)i << 16) | (uint32_t)(i + d);
                            qn += __popc(nmask);
                        }
                    }
                    store_runs(run_n > 0);
                }
            }
            // the ring's sums are scaled by this pair's cos and sin
            if (tail != head) r64_apply(ring, ring_bin, head, tail - head, c, s, out, row);
            if (qn) r64_drain(b, s1, s2, ctx, queue, qn, out, row, scratch);
        }
    }
}

// ---------------------------------------------------------------------------
// Delta x quasar. As in xcf_xi_fast_kernel a lane owns a quasar of a group of
// 32 (in order of distance) and steps the forest's pixels with the others, and
// the bins are decided in FP32. A run's sums hold the forest's side alone (dw,
// w, w (r1 - rq), w dist_m1, w z1: six FP64 operations a pair); the quasar's
// weight, distance, redshift and half angle come in when the run leaves the
// ring, with all lanes at work (seven a run of about two pixels), where the
// all-FP64 loop (pg_pairs_fp64.cu) spends about 70 a candidate. Bound: the
// FP64 pipe. 1,500 forests against 2,250 quasars: 18.5 ms with the loop, 2.4 ms
// here; 6,000 against 9,000: 100 ms and 11.7 ms.
constexpr int kXr64Block = 4096;      // neighbours ordered and swept at a time
constexpr int kXr64Buckets = 128;     // of kXr64BucketMpc along the line of sight
constexpr float kXr64BucketMpc = 8.f;

// Forest pixels in FP64 (structure of arrays in shared memory).
struct XPix64 {
    double *r, *w, *dw, *wm, *wz;
};

// A group's quasars (per warp, an entry per lane).
struct XQso64 {
    double *w, *cw, *sw, *m, *z;
};

struct Xr64Smem {
    size_t p1, q1, order, buckets, warps, per_warp, qso, ring, ring_bin, queue, total;
};

__host__ __device__ inline Xr64Smem xr64_smem(int max_pix1) {
    Xr64Smem l;
    const size_t mp = (size_t)((max_pix1 + 1) & ~1);
    l.p1 = 0;
    l.q1 = l.p1 + mp * 16;
    l.order = l.q1 + mp * 40;
    l.buckets = l.order + (size_t)kXr64Block * 2;
    l.warps = l.buckets + (size_t)kXr64Buckets * 4;
    l.qso = 0;
    l.ring = l.qso + 32 * 40;
    l.ring_bin = l.ring + (size_t)kR64Ring * 40;
    l.queue = l.ring_bin + (size_t)kR64Ring * 8;
    l.per_warp = l.queue + (size_t)kR64Queue * 4;
    l.total = l.warps + kR64Warps * l.per_warp;
    return l;
}

struct Xr64Ctx {
    int64_t a0, k0;
    double x1, y1, zc1, ra1, dec1, cd1;
};

__device__ __forceinline__ double xr64_angle(const Xr64Ctx &ctx, const pg_forest_set &objs,
                                             const double *nbr_angle, int64_t k, int64_t g) {
    return nbr_angle ? nbr_angle[k]
                     : angle_between(ctx.x1, ctx.y1, ctx.zc1, ctx.ra1, ctx.dec1, ctx.cd1,
                                     objs.x_cart[g], objs.y_cart[g], objs.z_cart[g], objs.ra[g],
                                     objs.dec[g]);
}

// Queued (pixel, neighbour) pairs: the reference's decision and terms.
__device__ __noinline__ void xr64_drain(const Binning &b, const pg_forest_set &fs,
                                        const pg_forest_set &objs, const int32_t *nbr_index,
                                        const double *nbr_angle, const Xr64Ctx &ctx,
                                        const uint32_t *queue, int count, const pg_xi_rows &out,
                                        size_t row, Scratch *scratch) {
    __syncwarp();
    const int lane = threadIdx.x & 31;
    for (int e = lane; e < count; e += 32) {
        const uint32_t entry = queue[e];
        const int64_t ia = ctx.a0 + (entry >> 16), k = ctx.k0 + (entry & 0xFFFF);
        const int64_t g = nbr_index[k];
        const double ang = xr64_angle(ctx, objs, nbr_angle, k, g);
        double r_par, r_trans, z;
        const int64_t bin = xcf_pair_bin(b, fs.z[ia], fs.r_comov[ia], fs.dist_m[ia], objs.z_qso[g],
                                         objs.obj_r_comov[g], objs.obj_dist_m[g], ang,
                                         cos(ang / 2), sin(ang / 2), r_par, r_trans, z);
        if (bin < 0) continue;
        if (bin >= b.nbins) {
            report_error(scratch, PG_ERR_BIN_RANGE, (int32_t)bin);
            continue;
        }
        const double w1 = fs.weights[ia], wq = objs.obj_weight[g];
        const double w12 = __dmul_rn(w1, wq);
        const double dw12 = __dmul_rn(__dmul_rn(fs.delta[ia], w1), wq);
        add_row(out, row + bin, dw12, w12, __dmul_rn(r_par, w12), __dmul_rn(r_trans, w12),
                __dmul_rn(z, w12), 1);
    }
    if (lane == 0) atomicAdd(&scratch->rechecked_pairs, (unsigned long long)count);
    __syncwarp();
}

// Adds n (<= 32) runs of the ring, from position head, to the row.
__device__ __forceinline__ void xr64_apply(const double *ring, const uint2 *ring_bin,
                                           const XQso64 &qso, int head, int n,
                                           const pg_xi_rows &out, size_t row) {
    __syncwarp();
    const int lane = threadIdx.x & 31;
    if (lane < n) {
        const int e = (head + lane) & (kR64Ring - 1);
        const uint2 u = ring_bin[e];
        const int q = u.y >> 16;
        const double we = ring[kR64Ring + e], wq = qso.w[q];
        add_row(out, row + u.x, __dmul_rn(ring[e], wq), __dmul_rn(we, wq),
                __dmul_rn(ring[2 * kR64Ring + e], qso.cw[q]),
                __dmul_rn(fma(qso.m[q], we, ring[3 * kR64Ring + e]), qso.sw[q]),
                __dmul_rn(fma(qso.z[q], we, ring[4 * kR64Ring + e]), 0.5 * wq),
                (int)(u.y & 0xFFFFu));
    }
    __syncwarp();
}

template <bool EXTRA>
__global__ void __launch_bounds__(kR64Warps * 32, 3) xcf_xi_runs64_kernel(
    const __grid_constant__ Binning b, const __grid_constant__ FastConst fc,
    const __grid_constant__ pg_forest_set fs, const __grid_constant__ pg_forest_set objs,
    const int64_t *__restrict__ nbr_offsets, const int32_t *__restrict__ nbr_index,
    const double *__restrict__ nbr_angle, const int32_t *__restrict__ work_order,
    int64_t num_work, int slices, const __grid_constant__ pg_xi_rows out, Scratch *scratch,
    int max_pix1) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int64_t unit_slot;
    __shared__ unsigned max_rho_bits;
    __shared__ int next_group;
    __shared__ Xr64Ctx ctx;
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    const unsigned lt_mask = (1u << lane) - 1u;
    const Xr64Smem L = xr64_smem(max_pix1);
    const int mp = (max_pix1 + 1) & ~1;
    float4 *p1 = reinterpret_cast<float4 *>(smem + L.p1);
    double *qd = reinterpret_cast<double *>(smem + L.q1);
    const XPix64 q1 = {qd, qd + mp, qd + 2 * mp, qd + 3 * mp, qd + 4 * mp};
    uint16_t *order = reinterpret_cast<uint16_t *>(smem + L.order);
    int *buckets = reinterpret_cast<int *>(smem + L.buckets);
    unsigned char *wbase = smem + L.warps + (size_t)warp * L.per_warp;
    double *qs = reinterpret_cast<double *>(wbase + L.qso);
    const XQso64 qso = {qs, qs + 32, qs + 64, qs + 96, qs + 128};
    double *ring = reinterpret_cast<double *>(wbase + L.ring);
    uint2 *ring_bin = reinterpret_cast<uint2 *>(wbase + L.ring_bin);
    uint32_t *queue = reinterpret_cast<uint32_t *>(wbase + L.queue);
    const unsigned np = fc.np, nt = fc.nt;
    // accepted range of p with one bin of margin each side, and of x_tr'
    const float p_lo = (fc.pc - 0.5f) - 1.f, p_hi = (fc.pc - 0.5f) + (float)np + 1.f;
    const float t_end = (float)nt + 1.f;

    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) {
            unit_slot = atomicAdd(&scratch->work_counter, 1);
            max_rho_bits = 0u;
        }
        __syncthreads();
        const int64_t unit = unit_slot;
        if (unit >= num_work * slices) break;
        const int64_t item = unit / slices;
        const int slice = (int)(unit - item * slices);
        const int64_t f = work_order ? work_order[item] : item;
        const size_t row = (size_t)fs.row[f] * b.nbins;
        const int64_t a0 = fs.pix_offset[f];
        const int64_t n1_64 = fs.pix_offset[f + 1] - a0;
        const int64_t nk = nbr_offsets[f + 1] - nbr_offsets[f];
        const int64_t k_lo = nbr_offsets[f] + nk * slice / slices;
        const int64_t k_hi = nbr_offsets[f] + nk * (slice + 1) / slices;
        if (threadIdx.x == 0 && slice == 0) atomicAdd(&scratch->work_items, 1ull);
        if (n1_64 > max_pix1) {
            if (threadIdx.x == 0) report_error(scratch, PG_ERR_UNSUPPORTED, (int32_t)f);
            continue;
        }
        if (n1_64 < 1 || k_lo >= k_hi) continue;
        const int n1 = (int)n1_64;
        if (threadIdx.x == 0)
            ctx = {a0, 0, fs.x_cart[f], fs.y_cart[f], fs.z_cart[f], fs.ra[f], fs.dec[f],
                   fs.cos_dec[f]};
        const double r_ref = reference_distance(fs.r_comov[a0 + n1 / 2], &max_rho_bits);
        float local_max = 0.f;
        for (int i = threadIdx.x; i < n1; i += blockDim.x) {
            const double w = fs.weights[a0 + i], r = fs.r_comov[a0 + i];
            const double m = fs.dist_m[a0 + i], z = fs.z[a0 + i];
            const float rho = f64_to_f32(r - r_ref);
            p1[i] = make_float4(rho, f64_to_f32(m), f64_to_f32(z), w != 0. ? 1.f : 0.f);
            q1.r[i] = r;
            q1.w[i] = w;
            q1.dw[i] = __dmul_rn(fs.delta[a0 + i], w);
            q1.wm[i] = __dmul_rn(w, m);
            q1.wz[i] = __dmul_rn(w, z);
            local_max = fmaxf(local_max, fabsf(rho));
        }
        if (local_max > 0.f) atomicMax(&max_rho_bits, __float_as_uint(local_max));
        __syncthreads();
        bool sorted1 = true;
        for (int i = threadIdx.x; i + 1 < n1; i += blockDim.x)
            sorted1 &= p1[i + 1].x >= p1[i].x && p1[i + 1].y >= p1[i].y;
        sorted1 = __syncthreads_and(sorted1) != 0;
        const ParGuard pg = par_guard_exact(&fc, __uint_as_float(max_rho_bits));
        sorted1 &= !pg.wide;

        for (int64_t kb = k_lo; kb < k_hi; kb += kXr64Block) {
            const int nq = (int)min((int64_t)kXr64Block, k_hi - kb);
            // the block's quasars in order of distance (a counting sort)
            for (int e = threadIdx.x; e < kXr64Buckets; e += blockDim.x) buckets[e] = 0;
            if (threadIdx.x == 0) {
                ctx.k0 = kb;
                next_group = 0;
            }
            __syncthreads();
            auto bucket_of = [&](int k) {
                const float rq = f64_to_f32(objs.obj_r_comov[nbr_index[kb + k]] - r_ref);
                const int e = __float2int_rd(rq * (1.f / kXr64BucketMpc)) + kXr64Buckets / 2;
                return e < 0 ? 0 : (e >= kXr64Buckets ? kXr64Buckets - 1 : e);
            };
            for (int k = threadIdx.x; k < nq; k += blockDim.x) atomicAdd(&buckets[bucket_of(k)], 1);
            __syncthreads();
            if (warp == 0) {
                int carry = 0;
                for (int e0 = 0; e0 < kXr64Buckets; e0 += 32) {
                    const int n = buckets[e0 + lane];
                    int incl = n;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int v = __shfl_up_sync(0xffffffffu, incl, o);
                        if (lane >= o) incl += v;
                    }
                    buckets[e0 + lane] = carry + incl - n;
                    carry += __shfl_sync(0xffffffffu, incl, 31);
                }
            }
            __syncthreads();
            for (int k = threadIdx.x; k < nq; k += blockDim.x)
                order[atomicAdd(&buckets[bucket_of(k)], 1)] = (uint16_t)k;
            __syncthreads();

            int qn = 0;  // FP64 re-decision queue of this warp
            for (;;) {
                int group = 0;
                if (lane == 0) group = atomicAdd(&next_group, 1);
                group = __shfl_sync(0xffffffffu, group, 0);
                if (group * 32 >= nq) break;
                const int slot = group * 32 + lane;
                const int kk = slot < nq ? (int)order[slot] : 0;
                float cp = 1.f, st = 0.f, nb = kFar, t = kFar, zv = kFar;
                double rq = 0.;
                bool valid = false;
                if (slot < nq) {
                    const int64_t g = nbr_index[kb + kk];
                    const double wq = objs.obj_weight[g];
                    if (wq != 0) {
                        valid = true;
                        const double ang = xr64_angle(ctx, objs, nbr_angle, kb + kk, g);
                        const double c = cos(ang / 2), sn = sin(ang / 2);
                        const double mq = objs.obj_dist_m[g], zq = objs.z_qso[g];
                        rq = objs.obj_r_comov[g];
                        qso.w[lane] = wq;
                        qso.cw[lane] = __dmul_rn(c, wq);
                        qso.sw[lane] = __dmul_rn(sn, wq);
                        qso.m[lane] = mq;
                        qso.z[lane] = zq;
                        cp = (float)(c * fc.inv_p);
                        st = (float)(sn * fc.inv_t);
                        nb = -__fmul_rn(cp, f64_to_f32(rq - r_ref));
                        t = __fmaf_rn(st, f64_to_f32(mq), -0.5f);
                        zv = f64_to_f32(zq);
                    }
                }
                // this lane's pixels [ia, ib): p and x_tr' are non-decreasing
                // along a sorted forest
                int ia = 0, ib = valid ? n1 : 0;
                if (sorted1 && valid) {
                    int lo = 0, hi = n1;
                    while (lo < hi) {
                        const int mid = (lo + hi) >> 1;
                        if (__fmaf_rn(cp, p1[mid].x, nb) < p_lo) lo = mid + 1;
                        else hi = mid;
                    }
                    ia = lo;
                    hi = n1;
                    while (lo < hi) {
                        const int mid = (lo + hi) >> 1;
                        if (__fmaf_rn(cp, p1[mid].x, nb) <= p_hi) lo = mid + 1;
                        else hi = mid;
                    }
                    ib = lo;
                    lo = ia;
                    hi = ib;
                    while (lo < hi) {
                        const int mid = (lo + hi) >> 1;
                        if (__fmaf_rn(st, p1[mid].y, t) < t_end) lo = mid + 1;
                        else hi = mid;
                    }
                    ib = lo;
                }
                const int g_lo = __reduce_min_sync(0xffffffffu, ia < ib ? ia : INT_MAX);
                const int g_hi = __reduce_max_sync(0xffffffffu, ia < ib ? ib : 0);
                int head = 0, tail = 0;  // run ring of this warp (warp-uniform)
                unsigned run_bin = 0xFFFFFFFFu;
                int run_n = 0;
                double r_xi = 0., r_we = 0., r_rp = 0., r_rm = 0., r_rz = 0.;
                auto store_runs = [&](bool flag) {
                    const unsigned m = __ballot_sync(0xffffffffu, flag);
                    if (flag) {
                        const int e = (tail + __popc(m & lt_mask)) & (kR64Ring - 1);
                        ring[e] = r_xi;
                        ring[kR64Ring + e] = r_we;
                        ring[2 * kR64Ring + e] = r_rp;
                        ring[3 * kR64Ring + e] = r_rm;
                        ring[4 * kR64Ring + e] = r_rz;
                        ring_bin[e] = make_uint2(run_bin, (unsigned)run_n | (unsigned)lane << 16);
                    }
                    tail += __popc(m);
                    if (tail - head >= 32) {
                        xr64_apply(ring, ring_bin, qso, head, 32, out, row);
                        head += 32;
                    }
                };
                for (int i = g_lo; i < g_hi; ++i) {
                    const float4 q = p1[i];
                    const bool in = (i >= ia) & (i < ib) & (q.w != 0.f);
                    float fp, ft;
                    const unsigned ip = round_rem(__fmaf_rn(cp, q.x, nb) - fc.pc, fp);
                    const unsigned it = round_rem(__fmaf_rn(st, q.y, t), ft);
                    bool near = (fabsf(fp) > pg.h_par) | (fabsf(ft) > fc.h_tr);
                    bool ok = (ip < np) & (it < nt);
                    if (EXTRA) {
                        const float zs = q.z + zv;
                        const float gz = fc.guard_z * fmaxf(1.f, 0.05f * fabsf(zs));
                        if (b.zmin_on) {
                            near |= fabsf(zs - fc.zmin2) < gz;
                            ok &= !(zs < fc.zmin2);
                        }
                        if (b.zmax_on) {
                            near |= fabsf(zs - fc.zmax2) < gz;
                            ok &= !(zs > fc.zmax2);
                        }
                    }
                    near &= in;
                    const bool acc = in & ok & !near;
                    const unsigned bin = ip * nt + it;
                    const bool brk = acc & (bin != run_bin);
                    const bool flush = brk & (run_n > 0);
                    if (__any_sync(0xffffffffu, flush)) {
                        store_runs(flush);
                        if (flush) {
                            run_n = 0;
                            r_xi = r_we = r_rp = r_rm = r_rz = 0.;
                        }
                    }
                    if (brk) run_bin = bin;
                    if (acc) {
                        const double w1 = q1.w[i];
                        r_xi = __dadd_rn(r_xi, q1.dw[i]);
                        r_we = __dadd_rn(r_we, w1);
                        r_rp = fma(__dsub_rn(q1.r[i], rq), w1, r_rp);
                        r_rm = __dadd_rn(r_rm, q1.wm[i]);
                        r_rz = __dadd_rn(r_rz, q1.wz[i]);
                        ++run_n;
                    }
                    const unsigned nmask = __ballot_sync(0xffffffffu, near);
                    if (nmask) {
                        if (qn > kR64Queue - 32) {
                            xr64_drain(b, fs, objs, nbr_index, nbr_angle, ctx, queue, qn, out, row,
                                       scratch);
                            if (lane == 0) atomicAdd(&scratch->recheck_overflows, 1ull);
                            qn = 0;
                        }
                        if (near)
                            queue[qn + __popc(nmask & lt_mask)] =
                                ((uint32_t)i << 16) | (uint32_t)kk;
                        qn += __popc(nmask);
                    }
                }
                store_runs(run_n > 0);
                // the ring's sums are scaled by this group's quasars
                if (tail != head) xr64_apply(ring, ring_bin, qso, head, tail - head, out, row);
            }
            if (qn)
                xr64_drain(b, fs, objs, nbr_index, nbr_angle, ctx, queue, qn, out, row, scratch);
            __syncthreads();
        }
    }
}

// enough units that the last ones are short (the order is longest first);
// staging a forest again for a slice is small against its pairs
int runs64_slices(int64_t num_work, int64_t resident) {
    int slices = 1;
    while (slices < 16 && num_work * slices < 4 * resident) slices *= 2;
    return slices;
}

template <bool EXTRA>
int launch_xruns64(const Binning &b, const pg_forest_set &fs, const pg_forest_set &objs,
                   const int64_t *nbr_offsets, const int32_t *nbr_index, const double *nbr_angle,
                   const int32_t *work_order, int64_t num_work, const pg_xi_rows &out,
                   Scratch *scratch, int num_sms, cudaStream_t stream) {
    auto kernel = xcf_xi_runs64_kernel<EXTRA>;
    const size_t smem = xr64_smem(fs.max_pixels).total;
    cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)kMaxDynSmem);
    if (err != cudaSuccess) return check_cuda(err);
    int per_sm = 0;
    err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kR64Warps * 32, smem);
    if (err != cudaSuccess) return check_cuda(err);
    if (per_sm < 1) return PG_ERR_UNSUPPORTED;
    const int64_t resident = (int64_t)num_sms * per_sm;
    const int slices = runs64_slices(num_work, resident);
    const int64_t grid = std::min(num_work * slices, resident);
    kernel<<<(int)grid, kR64Warps * 32, smem, stream>>>(
        b, make_fast_const(b), fs, objs, nbr_offsets, nbr_index, nbr_angle, work_order, num_work,
        slices, out, scratch, fs.max_pixels);
    return check_cuda(cudaGetLastError());
}

template <bool AUTO, bool EXTRA, bool LOWX>
int launch_runs64(const Binning &b, const pg_forest_set &s1, const pg_forest_set &s2,
                  const int64_t *nbr_offsets, const int32_t *nbr_index, const double *nbr_angle,
                  const int32_t *work_order, int64_t num_work, const pg_xi_rows &out,
                  Scratch *scratch, int num_sms, cudaStream_t stream) {
    auto kernel = cf_xi_runs64_kernel<AUTO, EXTRA, LOWX>;
    const size_t smem = r64_smem(s1.max_pixels).total;
    cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)kMaxDynSmem);
    if (err != cudaSuccess) return check_cuda(err);
    int per_sm = 0;
    err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kR64Warps * 32, smem);
    if (err != cudaSuccess) return check_cuda(err);
    if (per_sm < 1) return PG_ERR_UNSUPPORTED;
    const int64_t resident = (int64_t)num_sms * per_sm;
    const int slices = runs64_slices(num_work, resident);
    const int64_t grid = std::min(num_work * slices, resident);
    kernel<<<(int)grid, kR64Warps * 32, smem, stream>>>(
        b, make_fast_const(b), s1, s2, nbr_offsets, nbr_index, nbr_angle, work_order, num_work,
        slices, out, scratch, s1.max_pixels);
    return check_cuda(cudaGetLastError());
}

}  // namespace

// The (r_par, r_trans) geometry with any cut; pixel indices of a queued pair
// are 16 bits, forest 1 must fit in shared memory, the work counter (an int)
// counts slices, and FP32 has to resolve the bins. The r-mu and angular binnings and longer forests stay
// on the all-FP64 loop.
bool runs64_covers(const Binning &b, const pg_forest_set &s1, const pg_forest_set &s2,
                   int64_t num_work) {
    return !b.rmu && !b.ang_corr && s1.max_pixels <= 65535 && s2.max_pixels <= 65535 &&
           r64_smem(s1.max_pixels).total <= kMaxDynSmem && num_work < (INT32_MAX >> 5) &&
           fast_const_exact(make_fast_const(b));
}

int launch_cf_xi_runs64(const Binning &b, const pg_forest_set &s1, const pg_forest_set &s2,
                        const int64_t *nbr_offsets, const int32_t *nbr_index,
                        const double *nbr_angle, const int32_t *work_order, int64_t num_work,
                        const pg_xi_rows &out, Scratch *scratch, int num_sms,
                        cudaStream_t stream) {
    if (num_work <= 0) return PG_OK;
    const bool extra = b.remove_shp || b.zmin_on || b.zmax_on || b.zerr_on;
    const bool autoc = !b.x_correlation, lowx = autoc && b.r_par_min == 0.0;
#define PG_LAUNCH_R64(A, E, L)                                                                  \
    launch_runs64<A, E, L>(b, s1, s2, nbr_offsets, nbr_index, nbr_angle, work_order, num_work, \
                           out, scratch, num_sms, stream)
    if (!autoc) return extra ? PG_LAUNCH_R64(false, true, false) : PG_LAUNCH_R64(false, false, false);
    if (lowx) return extra ? PG_LAUNCH_R64(true, true, true) : PG_LAUNCH_R64(true, false, true);
    return extra ? PG_LAUNCH_R64(true, true, false) : PG_LAUNCH_R64(true, false, false);
#undef PG_LAUNCH_R64
}

// The same for delta x quasar.
bool xruns64_covers(const Binning &b, const pg_forest_set &fs, int64_t num_work) {
    return !b.rmu && !b.ang_corr && fs.max_pixels <= 65535 &&
           xr64_smem(fs.max_pixels).total <= kMaxDynSmem && num_work < (INT32_MAX >> 5) &&
           fast_const_exact(make_fast_const(b));
}

int launch_xcf_xi_runs64(const Binning &b, const pg_forest_set &fs, const pg_forest_set &objs,
                         const int64_t *nbr_offsets, const int32_t *nbr_index,
                         const double *nbr_angle, const int32_t *work_order, int64_t num_work,
                         const pg_xi_rows &out, Scratch *scratch, int num_sms,
                         cudaStream_t stream) {
    const auto launch = b.zmin_on || b.zmax_on ? launch_xruns64<true> : launch_xruns64<false>;
    return launch(b, fs, objs, nbr_offsets, nbr_index, nbr_angle, work_order, num_work, out,
                  scratch, num_sms, stream);
}

}  // namespace pg
