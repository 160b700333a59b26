// Wick covariance of the auto-correlation, T1-T3, over segments of equal bin
// (the terms and the reference are described in pg_wick.cu).
//
// For a forest pair with X1, X2 the weighted 1D correlations of its forests
// and b(i, j) the bin of a pixel pair,
//     T3[P, Q] = sum over b(i, j) = P, b(i', j') = Q of X1[i, i'] X2[j, j'].
// pg_wick.cu visits all pairs of listed pixel pairs, one FP64 FMA each. Here
// the sums over j of one row i and one bin P, and over i' of one column j'
// and one bin Q, are taken first:
//     V(i, P)[j'] = sum over j of X2[j, j'],  Z(j', Q)[i] = sum over i' of X1[i, i'],
//     T3[P, Q] = sum over rows (i, P) and columns (j', Q) of V(i, P)[j'] Z(j', Q)[i],
// and, as T3 is symmetric, only cells with Q not below P are swept and both
// are written. Bound: the FP64 pipe (16 cycles a warp FMA and SM). A bin of
// 4 Mpc/h holds about two pixels of a row, and folding r_par about four, so
// there are two to four times fewer row and column segments than pixel pairs
// and the sweep has 8 to 30 times fewer FMAs. The T2 terms of a shared pixel
// of forest 1 are sums of V over the row's own segments, those of forest 2 the
// same with the roles exchanged.
//
// Two kernels per batch of forest pairs: wick_list_kernel (a CTA per pair)
// bins the pixel pairs (decided in FP32 with the guard bands of
// pg_pairs_common.cuh, in FP64 next to an edge), adds WALL, NB and T1, and
// lists the column segments sorted by bin; wick_rows_kernel (persistent)
// takes one row or one column of one pair at a time, so that few pairs still
// fill the chip. The pairs of one kept forest of a 250-forest patch (50 x 50
// bins): 159 ms with the sweep (a CTA per pair), 0.25 + 5.6 ms here.
#include <algorithm>

#include "pg_internal.cuh"
#include "pg_pairs_common.cuh"

namespace pg {
namespace {

constexpr int kWsBlock = 256;
constexpr int kWsLanes = 32;       // bins P of a row swept together, a lane each
constexpr int kWsPitch = 33;       // doubles between the V of consecutive pixels
constexpr unsigned kWsEnd = 0x80000000u;  // last segment of its bin
constexpr size_t kWsMaxSmem = kMaxDynSmem;
constexpr uint64_t kWsBatchBytes = 256ull << 20;  // lists of a batch of pairs

// The lists of one forest pair in the work buffer: nonempty-bin index (or
// -1) of every pixel pair, [j][i]; column segments (first i | length << 16,
// j | end mark) sorted by bin; per nonempty bin its first segment and its
// bin; the counts.
struct PairLists {
    int32_t *index;
    uint2 *segs;
    int32_t *q_start, *q_bin, *head;
};

__host__ __device__ inline uint64_t pair_bytes(int64_t cap, int nb) {
    const uint64_t b = (uint64_t)cap * 12 + (uint64_t)(2 * nb + 1 + 4) * 4;
    return (b + 255) & ~(uint64_t)255;
}

__device__ __forceinline__ PairLists pair_lists(unsigned char *work, int64_t cap, int nb,
                                                int64_t k) {
    unsigned char *p = work + (uint64_t)k * pair_bytes(cap, nb);
    PairLists l;
    l.segs = reinterpret_cast<uint2 *>(p);
    l.index = reinterpret_cast<int32_t *>(p + (uint64_t)cap * 8);
    l.q_start = l.index + cap;
    l.q_bin = l.q_start + nb + 1;
    l.head = l.q_bin + nb;
    return l;
}

struct WickUnits {
    const double *zw1, *zw2;
    const int64_t *xo1, *xo2;
    const double *xa1, *xa2;
    const int32_t *first, *second, *slice;
    const double *angle;
    int64_t base;  // first pair of the batch
    int64_t cap;
    int32_t nb, max1, max2;
};

// Exclusive prefix sum over n values of an array in shared memory, in place;
// returns the total (every thread).
__device__ int block_prefix(int32_t *v, int n, int32_t *part) {
    const int tid = threadIdx.x, per = (n + kWsBlock - 1) / kWsBlock;
    const int lo = min(n, tid * per), hi = min(n, lo + per);
    int sum = 0;
    for (int k = lo; k < hi; ++k) sum += v[k];
    part[tid] = sum;
    __syncthreads();
    for (int o = 1; o < kWsBlock; o <<= 1) {
        const int add = tid >= o ? part[tid - o] : 0;
        __syncthreads();
        part[tid] += add;
        __syncthreads();
    }
    int run = part[tid] - sum;
    const int total = part[kWsBlock - 1];
    for (int k = lo; k < hi; ++k) {
        const int c = v[k];
        v[k] = run;
        run += c;
    }
    __syncthreads();
    return total;
}

// Bin of a pixel pair with the reference's FP64 expressions, or -1
// (cf.py:1561-1594); a quotient that rounds up to 1 is dropped.
__device__ __noinline__ int wick_bin64(const Binning &b, double r1, double r2, double cc,
                                       double ss) {
    double r_par = __dmul_rn(__dsub_rn(r1, r2), cc);
    if (!b.x_correlation) r_par = fabs(r_par);
    const double r_trans = __dmul_rn(__dadd_rn(r1, r2), ss);
    if (!(r_par < b.r_par_max && r_trans < b.r_trans_max && r_par >= b.r_par_min)) return -1;
    const int bp =
        (int)__dmul_rn(__ddiv_rn(__dsub_rn(r_par, b.r_par_min), b.r_par_range), (double)b.np);
    const int bt = (int)__dmul_rn(__ddiv_rn(r_trans, b.r_trans_max), (double)b.nt);
    if (bp >= b.np || bt >= b.nt) return -1;
    return bt + b.nt * bp;
}

size_t list_smem(int nb, int max2) {
    return (size_t)nb * (8 + 8 + 4 + 4) + (size_t)max2 * (8 + 8 + 4 + 4) +
           (size_t)kWsBlock * 4 + 32;
}

__global__ void __launch_bounds__(kWsBlock) wick_list_kernel(
    const __grid_constant__ Binning b, const __grid_constant__ FastConst fc,
    const __grid_constant__ pg_forest_set s1, const __grid_constant__ pg_forest_set s2,
    const __grid_constant__ WickUnits u, unsigned char *work, const __grid_constant__ pg_wick_sums out,
    Scratch *scratch) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ unsigned max_rho_bits;
    const int tid = threadIdx.x, nb = u.nb;
    double *wall = reinterpret_cast<double *>(smem), *t1 = wall + nb;
    double *w2 = t1 + nb, *z2 = w2 + u.max2;
    float *rho2 = reinterpret_cast<float *>(z2 + u.max2), *tr2 = rho2 + u.max2;
    int32_t *count = reinterpret_cast<int32_t *>(tr2 + u.max2), *rank = count + nb;
    int32_t *part = rank + nb;
    const PairLists l = pair_lists(work, u.cap, nb, blockIdx.x);
    const int64_t q = u.base + blockIdx.x;
    if (tid == 0) l.head[0] = l.head[1] = 0;
    // the first slice of a unit that was cut does all of it
    if (u.slice && u.slice[q] != 0) return;
    const int f = u.first[q], g = u.second[q];
    const int64_t o1 = s1.pix_offset[f], o2 = s2.pix_offset[g];
    const int64_t n1_64 = s1.pix_offset[f + 1] - o1, n2_64 = s2.pix_offset[g + 1] - o2;
    if (n1_64 > u.max1 || n2_64 > u.max2) {
        if (tid == 0) report_error(scratch, PG_ERR_INVALID_ARGUMENT, (int32_t)q);
        return;
    }
    const int n1 = (int)n1_64, n2 = (int)n2_64;
    if (tid == 0) {
        atomicAdd(&scratch->work_items, 1ull);
        max_rho_bits = 0u;
    }
    if (n1 < 1 || n2 < 1) return;
    const double ang =
        u.angle ? u.angle[q]
                : angle_between(s1.x_cart[f], s1.y_cart[f], s1.z_cart[f], s1.ra[f], s1.dec[f],
                                s1.cos_dec[f], s2.x_cart[g], s2.y_cart[g], s2.z_cart[g], s2.ra[g],
                                s2.dec[g]);
    const double cc = cos(ang / 2), ss = sin(ang / 2);
    const float cp = (float)(cc * fc.inv_p), st = (float)(ss * fc.inv_t);
    __syncthreads();  // max_rho_bits
    const double r_ref = reference_distance(s1.r_comov[o1 + n1 / 2], &max_rho_bits);
    for (int k = tid; k < nb; k += kWsBlock) {
        wall[k] = t1[k] = 0.;
        count[k] = 0;
    }
    for (int j = tid; j < n2; j += kWsBlock) {
        const double r = s2.r_comov[o2 + j];
        rho2[j] = -__fmul_rn(cp, (float)(r - r_ref));
        tr2[j] = __fmaf_rn(st, (float)r, -0.5f);
        w2[j] = s2.weights[o2 + j];
        z2[j] = u.zw2[o2 + j];
    }
    __syncthreads();
    for (int i = tid; i < n1; i += kWsBlock)
        atomicMax(&max_rho_bits, __float_as_uint(fabsf((float)(s1.r_comov[o1 + i] - r_ref))));
    __syncthreads();
    const ParGuard pg = par_guard_exact(&fc, __uint_as_float(max_rho_bits));
    const float pc = fc.pc, h_tr = fc.h_tr;
    // a thread per row: bins, and runs of one bin into the per-bin sums
    for (int i = tid; i < n1; i += kWsBlock) {
        const double r1 = s1.r_comov[o1 + i], w1 = s1.weights[o1 + i], z1 = u.zw1[o1 + i];
        const float rho1 = (float)(r1 - r_ref), d1 = (float)r1;
        int run = -1, n = 0;
        double sw = 0., st1 = 0.;
        auto flush = [&]() {
            atomicAdd(&count[run], n);
            atomicAdd(&wall[run], sw);
            atomicAdd(&t1[run], st1);
        };
        for (int j = 0; j < n2; ++j) {
            const float pp = __fmaf_rn(cp, rho1, rho2[j]);
            const float pv = b.x_correlation ? pp : fabsf(pp);
            const float xp = fc.lower_exact ? clamp_low(pv - pc, pg.low_clamp) : pv - pc;
            const float xt = __fmaf_rn(st, d1, tr2[j]);
            float fp, ft;
            const unsigned ip = round_rem(xp, fp), it = round_rem(xt, ft);
            int bin = ip < fc.np && it < fc.nt ? (int)(it + fc.nt * ip) : -1;
            if (fabsf(fp) > pg.h_par || fabsf(ft) > h_tr)
                bin = wick_bin64(b, r1, s2.r_comov[o2 + j], cc, ss);
            l.index[(int64_t)j * n1 + i] = bin;
            if (bin != run) {
                if (run >= 0) flush();
                run = bin;
                n = 0;
                sw = st1 = 0.;
            }
            if (bin >= 0) {
                const double w12 = __dmul_rn(w1, w2[j]);
                ++n;
                sw += w12;
                st1 = fma(w12, __dmul_rn(z1, z2[j]), st1);
            }
        }
        if (run >= 0) flush();
    }
    __syncthreads();
    // nonempty bins, ascending
    for (int k = tid; k < nb; k += kWsBlock) rank[k] = count[k] > 0 ? 1 : 0;
    __syncthreads();
    const int nz = block_prefix(rank, nb, part);
    unsigned long long listed = 0;
    for (int k = tid; k < nb; k += kWsBlock) {
        if (count[k] == 0) continue;
        l.q_bin[rank[k]] = k;
        listed += (unsigned long long)count[k];
        atomicAdd(&out.weights_wick[k], wall[k]);
        atomicAdd(reinterpret_cast<unsigned long long *>(&out.num_pairs_wick[k]),
                  (unsigned long long)count[k]);
        atomicAdd(&out.t1[(int64_t)k * nb + k], t1[k]);
    }
    __shared__ unsigned long long total_listed;
    if (tid == 0) total_listed = 0;
    __syncthreads();
    atomicAdd(&total_listed, listed);
    __syncthreads();
    // column segments per bin: count, prefix, place (a thread per column)
    for (int k = tid; k < nz; k += kWsBlock) count[k] = 0;
    __syncthreads();
    auto walk = [&](auto &&segment) {
        for (int j = tid; j < n2; j += kWsBlock) {
            int32_t *col = l.index + (int64_t)j * n1;
            int run = -1, from = 0;
            for (int i = 0; i < n1; ++i) {
                const int v = col[i];
                if (v != run) {
                    if (run >= 0) segment(run, from, i, j, col);
                    run = v;
                    from = i;
                }
            }
            if (run >= 0) segment(run, from, n1, j, col);
        }
    };
    walk([&](int bin, int from, int to, int, int32_t *col) {
        const int k = rank[bin];
        atomicAdd(&count[k], 1);
        for (int i = from; i < to; ++i) col[i] = k;  // nonempty-bin index from here on
    });
    __syncthreads();
    const int segs = block_prefix(count, nz, part);
    for (int k = tid; k < nz; k += kWsBlock) l.q_start[k] = count[k];
    if (tid == 0) {
        l.q_start[nz] = segs;
        l.head[0] = nz;
        l.head[1] = segs;
        // (a, b) pairs of listed pixel pairs, the reference's count of terms
        atomicAdd(&scratch->visited_pairs, total_listed * total_listed);
    }
    __syncthreads();
    walk([&](int k, int from, int to, int j, int32_t *) {
        const int pos = atomicAdd(&count[k], 1);
        const int end = k + 1 < nz ? l.q_start[k + 1] : segs;
        l.segs[pos] = make_uint2((unsigned)from | ((unsigned)(to - from) << 16),
                                 (unsigned)j | (pos == end - 1 ? kWsEnd : 0u));
    });
}

size_t rows_smem(int max1, int max2) {
    const size_t n = (size_t)std::max(max1, max2);
    return (size_t)max2 * kWsPitch * 8 + (size_t)max1 * 8 + n * 4 * 3 + 16;
}

__global__ void __launch_bounds__(kWsBlock, 3) wick_rows_kernel(
    const __grid_constant__ pg_forest_set s1, const __grid_constant__ pg_forest_set s2,
    const __grid_constant__ WickUnits u, int64_t num_pairs, unsigned char *work,
    const __grid_constant__ pg_wick_sums out, Scratch *scratch) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_task, s_bins, s_listed;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nb = u.nb;
    constexpr int kWarps = kWsBlock / 32;
    const int cap_n = max(u.max1, u.max2);
    double *v = reinterpret_cast<double *>(smem);
    double *x1row = v + (size_t)u.max2 * kWsPitch;
    uint32_t *keys = reinterpret_cast<uint32_t *>(x1row + u.max1), *sorted = keys + cap_n;
    int32_t *p_start = reinterpret_cast<int32_t *>(sorted + cap_n);  // [cap_n + 1]
    const int per_pair = u.max1 + u.max2;
    unsigned long long macs = 0;  // FMAs of T3 and additions of V
    for (;;) {
        __syncthreads();
        if (tid == 0) s_task = atomicAdd(&scratch->work_counter, 1);
        __syncthreads();
        const int64_t pair = s_task / per_pair;
        if (pair >= num_pairs) break;
        int line = s_task - (int)pair * per_pair;
        const bool is_row = line < u.max1;
        if (!is_row) line -= u.max1;
        const PairLists l = pair_lists(work, u.cap, nb, pair);
        const int nz = l.head[0];
        if (nz == 0) continue;
        const int64_t q = u.base + pair;
        const int f = u.first[q], g = u.second[q];
        const int64_t o1 = s1.pix_offset[f], o2 = s2.pix_offset[g];
        const int n1 = (int)(s1.pix_offset[f + 1] - o1), n2 = (int)(s2.pix_offset[g + 1] - o2);
        if (line >= (is_row ? n1 : n2)) continue;
        const double *__restrict__ x1 = u.xa1 + u.xo1[f], *__restrict__ x2 = u.xa2 + u.xo2[g];
        // the line's listed pixels sorted by bin (then pixel): rank by counting
        const int n = is_row ? n2 : n1;
        if (tid == 0) s_listed = 0;
        for (int t = tid; t < n; t += kWsBlock) {
            const int k = is_row ? l.index[(int64_t)t * n1 + line] : l.index[(int64_t)line * n1 + t];
            keys[t] = k < 0 ? 0xFFFFFFFFu : ((unsigned)k << 16) | (unsigned)t;
        }
        if (is_row)
            for (int t = tid; t < n1; t += kWsBlock) x1row[t] = x1[(int64_t)line * n1 + t];
        __syncthreads();
        int mine = 0;
        for (int t = tid; t < n; t += kWsBlock) {
            const uint32_t key = keys[t];
            if (key == 0xFFFFFFFFu) continue;
            int r = 0;
            for (int e = 0; e < n; ++e) r += keys[e] < key ? 1 : 0;
            sorted[r] = key;
            ++mine;
        }
        if (mine) atomicAdd(&s_listed, mine);
        __syncthreads();
        const int listed = s_listed;
        if (listed == 0) continue;
        if (warp == 0) {
            int bins = 0;
            for (int e0 = 0; e0 < listed; e0 += 32) {
                const int e = e0 + lane;
                const bool first =
                    e < listed && (e == 0 || (sorted[e] >> 16) != (sorted[e - 1] >> 16));
                const unsigned m = __ballot_sync(0xffffffffu, first);
                if (first) p_start[bins + __popc(m & ((1u << lane) - 1u))] = e;
                bins += __popc(m);
            }
            if (lane == 0) {
                p_start[bins] = listed;
                s_bins = bins;
            }
        }
        __syncthreads();
        const int bins = s_bins;
        for (int g0 = 0; g0 < bins; g0 += kWsLanes) {
            const bool active = g0 + lane < bins;
            const int my_s0 = active ? p_start[g0 + lane] : 0;
            const int my_s1 = active ? p_start[g0 + lane + 1] : 0;
            const int my_p = active ? (int)(sorted[my_s0] >> 16) : INT_MAX;
            const int my_bin = active ? l.q_bin[my_p] : 0;
            const int64_t my_row = (int64_t)my_bin * nb;
            if (!is_row) {
                // T2 of the shared pixel `line` of forest 2
                const double c2 = __dmul_rn(s2.weights[o2 + line], u.zw2[o2 + line]);
                for (int k = warp; k < bins; k += kWarps) {
                    double acc = 0.;
                    for (int e = p_start[k]; e < p_start[k + 1]; ++e) {
                        const double *__restrict__ x = x1 + (int64_t)(sorted[e] & 0xffffu) * n1;
                        for (int s = my_s0; s < my_s1; ++s) acc += x[sorted[s] & 0xffffu];
                    }
                    if (active && acc != 0.)
                        atomicAdd(&out.t2[my_row + l.q_bin[sorted[p_start[k]] >> 16]],
                                  __dmul_rn(acc, c2));
                }
                continue;
            }
            // V(i, P)[j'] of the group's bins
            __syncthreads();
            for (int p = warp; p < kWsLanes; p += kWarps) {
                const bool have = g0 + p < bins;
                const int e0 = have ? p_start[g0 + p] : 0, e1 = have ? p_start[g0 + p + 1] : 0;
                for (int t = lane; t < n2; t += 32) {
                    double sum = 0.;
                    for (int e = e0; e < e1; ++e)
                        sum += __ldg(x2 + (int64_t)(sorted[e] & 0xffffu) * n2 + t);
                    v[t * kWsPitch + p] = sum;
                }
            }
            __syncthreads();
            // T2 of the shared pixel `line` of forest 1
            const double c1 = __dmul_rn(s1.weights[o1 + line], u.zw1[o1 + line]);
            for (int k = warp; k < bins; k += kWarps) {
                double acc = 0.;
                for (int e = p_start[k]; e < p_start[k + 1]; ++e)
                    acc += v[(sorted[e] & 0xffffu) * kWsPitch + lane];
                if (active && acc != 0.)
                    atomicAdd(&out.t2[my_row + l.q_bin[sorted[p_start[k]] >> 16]],
                              __dmul_rn(acc, c1));
            }
            // T3: the column segments of the bins from the group's first on,
            // shared among the warps at bin boundaries
            const int p0 = (int)(sorted[p_start[g0]] >> 16);
            const int lo = l.q_start[p0], hi = l.head[1];
            if (tid == 0)
                macs += (unsigned long long)(hi - lo) * min(kWsLanes, bins - g0) +
                        (unsigned long long)(p_start[min(bins, g0 + kWsLanes)] - my_s0) * n2;
            auto first_bin = [&](int w) {
                const int target = lo + (int)((int64_t)(hi - lo) * w / kWarps);
                int a = p0, z = nz;
                while (a < z) {
                    const int mid = (a + z) >> 1;
                    if (l.q_start[mid] < target) a = mid + 1;
                    else z = mid;
                }
                return a;
            };
            int kq = first_bin(warp);
            const int k_end = warp == kWarps - 1 ? nz : first_bin(warp + 1);
            const int s_end = l.q_start[k_end];
            double acc = 0.;
            for (int s0 = l.q_start[kq]; s0 < s_end; s0 += 32) {
                const int batch = min(32, s_end - s0);
                uint2 seg = make_uint2(0u, 0u);
                double z = 0.;
                if (lane < batch) {
                    seg = l.segs[s0 + lane];
                    const int i0 = (int)(seg.x & 0xffffu), len = (int)(seg.x >> 16);
                    z = x1row[i0];
                    for (int t = 1; t < len; ++t) z += x1row[i0 + t];
                }
                for (int k = 0; k < batch; k += 4) {
                    unsigned y[4];
                    double zz[4], vv[4];
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        y[r] = __shfl_sync(0xffffffffu, seg.y, (k + r) & 31);
                        zz[r] = __shfl_sync(0xffffffffu, z, (k + r) & 31);
                        vv[r] = v[(y[r] & 0x7fffffffu) * kWsPitch + lane];
                    }
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        if (k + r >= batch) break;
                        acc = fma(vv[r], zz[r], acc);
                        if (y[r] & kWsEnd) {
                            if (kq >= my_p && active && acc != 0.) {
                                const int bq = l.q_bin[kq];
                                atomicAdd(&out.t3[my_row + bq], acc);
                                if (kq != my_p)
                                    atomicAdd(&out.t3[(int64_t)bq * nb + my_bin], acc);
                            }
                            acc = 0.;
                            ++kq;
                        }
                    }
                }
            }
        }
    }
    if (tid == 0 && macs) atomicAdd(&scratch->gemm_macs, macs);
}

}  // namespace

uint64_t wick_segments_bytes(int nb, int max1, int max2, int64_t num_pairs) {
    const uint64_t per = pair_bytes((int64_t)max1 * max2, nb);
    uint64_t n = std::max<uint64_t>(16, kWsBatchBytes / per);
    n = std::min<uint64_t>(n, 4096);
    if (num_pairs > 0 && (uint64_t)num_pairs < n) n = (uint64_t)num_pairs;
    return n * per;
}

// Lists and V in shared memory: up to about 810 pixels (V; the lists hold the
// 6,000 bins that a call may have up to 3,600 pixels). Longer forests stay on the
// sweep over listed pairs (wick_t123_kernel), and so does a work buffer that holds
// no pair's lists.
bool wick_segments_covers(int nb, int max1, int max2, uint64_t work_bytes) {
    return nb < 65535 && max1 <= 32767 && max2 <= 32767 && list_smem(nb, max2) <= kWsMaxSmem &&
           rows_smem(max1, max2) <= kWsMaxSmem &&
           work_bytes >= pair_bytes((int64_t)max1 * max2, nb);
}

int launch_wick_segments(const pg_corr_params &p, const pg_forest_set &s1,
                         const pg_forest_set &s2, const double *zw1, const double *zw2,
                         const int64_t *xo1, const double *xa1, const int64_t *xo2,
                         const double *xa2, const int32_t *pair_first, const int32_t *pair_second,
                         const double *pair_angle, const int32_t *unit_slice, int64_t num_pairs,
                         void *work, uint64_t work_bytes, const pg_wick_sums &out,
                         Scratch *scratch, int num_sms, cudaStream_t stream) {
    Binning b = make_binning(p);
    b.rmu = b.ang_corr = 0;
    const FastConst fc = make_fast_const(b);
    WickUnits u;
    u.zw1 = zw1; u.zw2 = zw2;
    u.xo1 = xo1; u.xo2 = xo2;
    u.xa1 = xa1; u.xa2 = xa2;
    u.first = pair_first; u.second = pair_second;
    u.slice = unit_slice;
    u.angle = pair_angle;
    u.max1 = s1.max_pixels;
    u.max2 = s2.max_pixels;
    u.cap = (int64_t)u.max1 * u.max2;
    u.nb = b.nbins;
    const size_t smem_a = list_smem(u.nb, u.max2), smem_b = rows_smem(u.max1, u.max2);
    cudaError_t err = cudaFuncSetAttribute(
        wick_list_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWsMaxSmem);
    if (err != cudaSuccess) return check_cuda(err);
    err = cudaFuncSetAttribute(wick_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)kWsMaxSmem);
    if (err != cudaSuccess) return check_cuda(err);
    int occ = 0;
    err = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, wick_rows_kernel, kWsBlock, smem_b);
    if (err != cudaSuccess) return check_cuda(err);
    if (occ < 1) return PG_ERR_UNSUPPORTED;
    // pairs of a batch: their lists fit in the work buffer, their tasks in an int
    int64_t batch = (int64_t)(work_bytes / pair_bytes(u.cap, u.nb));
    batch = std::min<int64_t>(batch, (INT32_MAX / 2) / (u.max1 + u.max2));
    unsigned char *base = static_cast<unsigned char *>(work);
    for (u.base = 0; u.base < num_pairs; u.base += batch) {
        const int64_t n = std::min(batch, num_pairs - u.base);
        if (u.base > 0) {
            const int rc = check_cuda(cudaMemsetAsync(&scratch->work_counter, 0,
                                                      sizeof(scratch->work_counter), stream));
            if (rc) return rc;
        }
        wick_list_kernel<<<(unsigned)n, kWsBlock, smem_a, stream>>>(b, fc, s1, s2, u, base, out,
                                                                    scratch);
        const int64_t tasks = n * (u.max1 + u.max2);
        const int grid = (int)std::min<int64_t>(tasks, (int64_t)num_sms * occ);
        wick_rows_kernel<<<grid, kWsBlock, smem_b, stream>>>(s1, s2, u, n, base, out, scratch);
        const int rc = check_cuda(cudaGetLastError());
        if (rc) return rc;
    }
    return PG_OK;
}

}  // namespace pg
