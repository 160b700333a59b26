// Training pass of the warm-start network: the BF16 tile GEMM that every
// layer runs on, and the forward and backward passes as two calls.
//
// The products are small (a batch of 4,096 rows and layers of 256: 0.5 GFLOP
// each, a fraction of a microsecond of tensor work), so a pass is bound by
// latency: by how soon the operands are on chip, how many SMs share one
// product, and the number of launches. Every accumulator is one chain of
// mma.sync steps in ascending k (and every bias gradient one chain of
// additions in ascending row), so that the sums do not depend on the tile or
// on the batch's split; what is left to choose is how the chains are fed:
//  * K in chunks of 64, requested several chunks ahead with 16-byte cp.async
//    (zero filled past the edges, so ragged M, N, K need no padding);
//    fragments come from XOR-swizzled 128-byte rows with ldmatrix (transposed
//    for operands stored the other way round).
//  * CTA tile 64 x 64, or 32 x 32 where the larger tiles would leave SMs idle
//    (weight gradients X^T dZ: 256 x 256 and K = batch; small batches).
//  * All weight gradients and the bias gradients are one launch: the bias
//    CTAs (a lane per column, rows staged ahead) run beside the tiles.
//  * The 256 -> 2 layer is a warp per 16 rows (forward) and a kernel that
//    forms the loss gradient and the first dZ together (backward).
// Batch 4,096 (eleven GEMMs, four column sums, the loss): 2.04 ms with scalar
// staged 64 x 64 x 32 tiles and a thread per column, 0.085 ms here.
#include <initializer_list>

#include "pg_mlp_common.cuh"

namespace pg {
namespace {

constexpr int kChunk = 64;         // k of a stage
constexpr int kPitch = 128;        // bytes of a staged row (64 elements)
constexpr int kOperand = 64 * kPitch;
constexpr int kStage = 2 * kOperand;
constexpr int kMaxGroup = 4;
constexpr int kMaxBias = 4;
constexpr int kBiasCols = 32;      // columns (lanes) of a bias CTA
constexpr int kBiasRows = kStage / (kBiasCols * 2);  // rows of a stage

// One launch: products p < count own the tiles [first[p], first[p + 1]), then
// bias jobs (column sums of a bf16 [m, ld] matrix) the CTAs after them.
struct GemmGroup {
    GemmArgs g[kMaxGroup];
    int first[kMaxGroup + 1];
    int tiles_n[kMaxGroup];
    int a_t[kMaxGroup], b_t[kMaxGroup];  // operand stored [k][m], [n][k]
    int vec[kMaxGroup];                  // paired epilogue accesses are aligned
    int count;
    int stages;
    const __nv_bfloat16 *bias_x[kMaxBias];
    float *bias_out[kMaxBias];
    int bias_n[kMaxBias], bias_ld[kMaxBias], bias_first[kMaxBias + 1];
    int bias_count, bias_m;
};

__device__ __forceinline__ uint32_t smem_addr(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void cp_async_commit() {
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// At most n groups left in flight (n is uniform, 0 to 11).
__device__ __forceinline__ void cp_async_wait(int n) {
    switch (n) {
#define PG_WAIT(N) \
    case N: asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); break;
        PG_WAIT(1) PG_WAIT(2) PG_WAIT(3) PG_WAIT(4) PG_WAIT(5) PG_WAIT(6) PG_WAIT(7) PG_WAIT(8)
        PG_WAIT(9) PG_WAIT(10) PG_WAIT(11)
#undef PG_WAIT
        default: asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
}

// One operand's share of a thread: 16-byte pieces of an R x C tile of a
// row-major [rows, cols] matrix, zero outside it, into 128-byte rows with the
// piece index XORed by the row (conflict-free ldmatrix). Along K (ALONG_ROWS:
// the rows are k) only the last chunk can be ragged; the other edge is fixed.
template <int R, int C, int THREADS, bool ALONG_ROWS>
struct TileLoader {
    static constexpr int kPieces = R * (C / 8) / THREADS;
    const __nv_bfloat16 *src[kPieces];
    int bytes[kPieces];
    __device__ __forceinline__ void start(const __nv_bfloat16 *base, int64_t ld, int fixed0,
                                          int fixed_end) {
#pragma unroll
        for (int q = 0; q < kPieces; ++q) {
            const int e = threadIdx.x + q * THREADS, r = e / (C / 8), c = e % (C / 8) * 8;
            const int at = fixed0 + (ALONG_ROWS ? c : r);
            int n = ALONG_ROWS ? 2 * (fixed_end - at) : (at < fixed_end ? 16 : 0);
            n = n < 0 ? 0 : (n > 16 ? 16 : n);
            bytes[q] = n;
            src[q] = n ? base + (ALONG_ROWS ? (int64_t)r * ld + at : at * ld + c) : base;
        }
    }
    // chunk k0 of K = k; step: elements from one chunk to the next
    __device__ __forceinline__ void load(uint32_t dst, int chunk, int64_t step, int k) const {
        const int left = k - chunk * kChunk;
#pragma unroll
        for (int q = 0; q < kPieces; ++q) {
            const int e = threadIdx.x + q * THREADS, r = e / (C / 8), c = e % (C / 8);
            int n = bytes[q];
            if (left < kChunk) {  // the ragged last chunk
                if (ALONG_ROWS) n = r < left ? n : 0;
                else n = min(n, max(0, 2 * (left - c * 8)));
            }
            const __nv_bfloat16 *from = n ? src[q] + chunk * step : src[q];
            cp_async16(dst + r * kPitch + ((c ^ (r & 7)) << 4), from, n);
        }
    }
};

__device__ __forceinline__ void ldmatrix4(uint32_t r[4], uint32_t tile, int row, int col,
                                          bool trans) {
    const uint32_t addr = tile + row * kPitch + (((col >> 3) ^ (row & 7)) << 4);
    if (trans)
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                     : "r"(addr)
                     : "memory");
    else
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                     : "r"(addr)
                     : "memory");
}

// Bias, activation and stores of the accumulators of columns n and n + 1.
// zin: its pre-activations (GELU_GRAD).
__device__ __forceinline__ void store_pair(const GemmArgs &g, bool vec, int m, int n, float v0,
                                           float v1, float2 zin) {
    if (m >= g.m || n >= g.n) return;
    const bool two = n + 1 < g.n;
    if (g.bias) {
        v0 += g.bias[n];
        if (two) v1 += g.bias[n + 1];
    }
    if (g.zout) {
        float *z = g.zout + m * g.ldz + n;
        if (vec && two) *reinterpret_cast<float2 *>(z) = make_float2(v0, v1);
        else {
            z[0] = v0;
            if (two) z[1] = v1;
        }
    }
    if (g.epilogue & PG_MLP_EPI_GELU) {
        v0 = gelu(v0);
        v1 = gelu(v1);
    }
    if (g.epilogue & PG_MLP_EPI_GELU_GRAD) {
        v0 *= gelu_grad(zin.x);
        v1 *= gelu_grad(zin.y);
    }
    if (g.c) {
        __nv_bfloat16 *c = g.c + m * g.ldc + n;
        if (vec && two) *reinterpret_cast<__nv_bfloat162 *>(c) = __floats2bfloat162_rn(v0, v1);
        else {
            c[0] = __float2bfloat16(v0);
            if (two) c[1] = __float2bfloat16(v1);
        }
    }
    if (g.cf) {
        float *c = g.cf + m * g.ldc + n;
        if (g.beta != 0.f) {
            v0 += g.beta * c[0];
            if (two) v1 += g.beta * c[1];
        }
        if (vec && two) *reinterpret_cast<float2 *>(c) = make_float2(v0, v1);
        else {
            c[0] = v0;
            if (two) c[1] = v1;
        }
    }
}

// Sums a bias job's 32 columns, a lane per column, rows in ascending order.
__device__ void bias_columns(const GemmGroup &grp, int job_cta, unsigned char *smem) {
    int job = 0;
    while (job + 1 < grp.bias_count && job_cta >= grp.bias_first[job + 1]) ++job;
    const int c0 = (job_cta - grp.bias_first[job]) * kBiasCols;
    const int n = grp.bias_n[job], ld = grp.bias_ld[job], m = grp.bias_m;
    const __nv_bfloat16 *x = grp.bias_x[job];
    const int lane = threadIdx.x & 31;
    const int chunks = (m + kBiasRows - 1) / kBiasRows;
    const uint32_t sbase = smem_addr(smem);
    auto issue = [&](int c) {
        const uint32_t dst = sbase + c % grp.stages * kStage;
        for (int e = threadIdx.x; e < kBiasRows * (kBiasCols / 8); e += blockDim.x) {
            const int r = c * kBiasRows + e / (kBiasCols / 8), col = c0 + e % (kBiasCols / 8) * 8;
            int bytes = r < m ? 2 * (n - col) : 0;
            bytes = bytes < 0 ? 0 : (bytes > 16 ? 16 : bytes);
            cp_async16(dst + e * 16, bytes ? x + (int64_t)r * ld + col : x, bytes);
        }
    };
    float s = 0.f;
    for (int c = 0; c + 1 < grp.stages; ++c) {
        if (c < chunks) issue(c);
        cp_async_commit();
    }
    for (int c = 0; c < chunks; ++c) {
        cp_async_wait(grp.stages - 2);
        __syncthreads();
        if (c + grp.stages - 1 < chunks) issue(c + grp.stages - 1);
        cp_async_commit();
        if (threadIdx.x < 32) {
            const __nv_bfloat16 *t =
                reinterpret_cast<const __nv_bfloat16 *>(smem + c % grp.stages * kStage) + lane;
            // rows past the batch are staged as zeros, which add nothing
            // (a sum is never -0 after the first row)
#pragma unroll 1
            for (int r0 = 0; r0 < kBiasRows; r0 += 32) {
                float v[32];
#pragma unroll
                for (int r = 0; r < 32; ++r) v[r] = __bfloat162float(t[(r0 + r) * kBiasCols]);
#pragma unroll
                for (int r = 0; r < 32; ++r) s += v[r];
            }
        }
    }
    if (threadIdx.x < 32 && c0 + lane < n) grp.bias_out[job][c0 + lane] = s;
}

// T x T tiles (64 or 32); a warp owns 16 x T / 2 of one.
template <int T>
constexpr int tile_threads() { return T * 4; }

// Main loop: acc = A B over the CTA's tile. One barrier a chunk: the chunk's
// loads have landed for every thread and the slot that is refilled was read
// in the previous step. All fragments of the chunk are requested before its
// first multiplication, so the chain of products waits for one another only.
template <int T, bool A_T, bool B_T>
__device__ __forceinline__ void tile_products(const GemmArgs &g, int m0, int n0, int stages,
                                              uint32_t sbase, float (&acc)[T / 16][4]) {
    constexpr int NJ = T / 16, THREADS = tile_threads<T>();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int wm = (warp >> 1) * 16, wn = (warp & 1) * (T / 2);
    const int chunks = (g.k + kChunk - 1) / kChunk;
    TileLoader<A_T ? kChunk : T, A_T ? T : kChunk, THREADS, A_T> la;
    TileLoader<B_T ? T : kChunk, B_T ? kChunk : T, THREADS, !B_T> lb;
    la.start(g.a, A_T ? g.sak : g.sam, m0, g.m);
    lb.start(g.b, B_T ? g.sbn : g.sbk, n0, g.n);
    const int64_t step_a = A_T ? kChunk * g.sak : kChunk, step_b = B_T ? kChunk : kChunk * g.sbk;
    auto issue = [&](int c, int slot) {
        const uint32_t dst = sbase + slot * kStage;
        la.load(dst, c, step_a, g.k);
        lb.load(dst + kOperand, c, step_b, g.k);
    };
    for (int c = 0; c + 1 < stages; ++c) {
        if (c < chunks) issue(c, c);
        cp_async_commit();
    }
    int slot = 0;
    for (int c = 0; c < chunks; ++c) {
        cp_async_wait(stages - 2);
        __syncthreads();
        {
            const int next = c + stages - 1;
            if (next < chunks) issue(next, slot == 0 ? stages - 1 : slot - 1);
            cp_async_commit();
        }
        const uint32_t ta = sbase + slot * kStage, tb = ta + kOperand;
        uint32_t af[4][4], bf[4][NJ / 2][4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int ks = q * 16;
            if (A_T)
                ldmatrix4(af[q], ta, ks + (lane & 7) + ((lane >> 4) & 1) * 8,
                          wm + ((lane >> 3) & 1) * 8, true);
            else
                ldmatrix4(af[q], ta, wm + (lane & 15), ks + (lane >> 4) * 8, false);
#pragma unroll
            for (int j = 0; j < NJ / 2; ++j) {
                const int nn = wn + j * 16;
                if (B_T)
                    ldmatrix4(bf[q][j], tb, nn + (lane & 7) + ((lane >> 4) & 1) * 8,
                              ks + ((lane >> 3) & 1) * 8, false);
                else
                    ldmatrix4(bf[q][j], tb, ks + (lane & 7) + ((lane >> 3) & 1) * 8,
                              nn + ((lane >> 4) & 1) * 8, true);
            }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int j = 0; j < NJ; ++j) mma_bf16(acc[j], af[q], bf[q][j >> 1] + (j & 1) * 2);
        if (++slot == stages) slot = 0;
    }
}

template <int T>
__global__ void __launch_bounds__(tile_threads<T>()) gemm_tile_kernel(
    const __grid_constant__ GemmGroup grp) {
    extern __shared__ __align__(128) unsigned char smem[];
    constexpr int NJ = T / 16;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // the bias CTAs first: their chains are the longest
    const int bias_ctas = grp.bias_first[grp.bias_count];
    if ((int)blockIdx.x < bias_ctas) {
        bias_columns(grp, blockIdx.x, smem);
        return;
    }
    const int tile = blockIdx.x - bias_ctas;
    int p = 0;
    while (p + 1 < grp.count && tile >= grp.first[p + 1]) ++p;
    const GemmArgs &g = grp.g[p];
    const bool vec = grp.vec[p] != 0;
    const int t = tile - grp.first[p];
    const int m0 = t / grp.tiles_n[p] * T, n0 = t % grp.tiles_n[p] * T;
    const int row = m0 + (warp >> 1) * 16 + (lane >> 2);
    const int col = n0 + (warp & 1) * (T / 2) + (lane & 3) * 2;
    // the activation derivative's inputs, requested ahead of the products
    float2 zin[NJ][2];
    if (g.epilogue & PG_MLP_EPI_GELU_GRAD) {
#pragma unroll
        for (int j = 0; j < NJ; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int m = row + h * 8, n = col + j * 8;
                const float *z = g.zin + m * g.ldz + n;
                zin[j][h] = make_float2(0.f, 0.f);
                if (m < g.m && n + 1 < g.n && vec)
                    zin[j][h] = *reinterpret_cast<const float2 *>(z);
                else if (m < g.m && n < g.n)
                    zin[j][h] = make_float2(z[0], n + 1 < g.n ? z[1] : 0.f);
            }
    }
    float acc[NJ][4];
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[j][r] = 0.f;
    const uint32_t sbase = smem_addr(smem);
    if (grp.a_t[p]) {
        if (grp.b_t[p]) tile_products<T, true, true>(g, m0, n0, grp.stages, sbase, acc);
        else tile_products<T, true, false>(g, m0, n0, grp.stages, sbase, acc);
    } else {
        if (grp.b_t[p]) tile_products<T, false, true>(g, m0, n0, grp.stages, sbase, acc);
        else tile_products<T, false, false>(g, m0, n0, grp.stages, sbase, acc);
    }
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h)
            store_pair(g, vec, row + h * 8, col + j * 8, acc[j][2 * h], acc[j][2 * h + 1],
                       zin[j][h]);
}

// Whether the tile GEMM takes the operands: one stride of each is 1, the
// other and the base keep every 16-byte chunk aligned (other layouts stay on
// gemm_bf16_kernel).
bool operand_ok(const void *p, int64_t unit, int64_t ld) {
    return unit == 1 && ld > 0 && ld % 8 == 0 && reinterpret_cast<uintptr_t>(p) % 16 == 0;
}

bool add_product(GemmGroup &grp, const GemmArgs &g) {
    const int p = grp.count;
    if (operand_ok(g.a, g.sak, g.sam)) grp.a_t[p] = 0;
    else if (operand_ok(g.a, g.sam, g.sak)) grp.a_t[p] = 1;
    else return false;
    if (operand_ok(g.b, g.sbn, g.sbk)) grp.b_t[p] = 0;
    else if (operand_ok(g.b, g.sbk, g.sbn)) grp.b_t[p] = 1;
    else return false;
    auto aligned = [](const void *q, int64_t ld, uintptr_t bytes) {
        return !q || (ld % 2 == 0 && reinterpret_cast<uintptr_t>(q) % bytes == 0);
    };
    grp.vec[p] = aligned(g.zin, g.ldz, 8) && aligned(g.zout, g.ldz, 8) && aligned(g.c, g.ldc, 4) && aligned(g.cf, g.ldc, 8);
    grp.g[p] = g;
    grp.count = p + 1;
    return true;
}

void add_bias(GemmGroup &grp, const __nv_bfloat16 *x, int m, int n, int ld, float *out) {
    const int q = grp.bias_count++;
    grp.bias_x[q] = x;
    grp.bias_out[q] = out;
    grp.bias_n[q] = n;
    grp.bias_ld[q] = ld;
    grp.bias_m = m;
    grp.bias_first[q + 1] = grp.bias_first[q] + (n + kBiasCols - 1) / kBiasCols;
}

// 64 x 64 tiles load half the operand bytes per product of 32 x 32 ones; the
// small tiles are taken where the large ones would not reach every SM (of 152):
// a layer of batch 4,096 (256 large tiles) takes 8.6 us in 64 x 64 and 14.3 us
// in 32 x 32 tiles, its weight gradients (40 large tiles) 39.9 us and 27.6 us.
// Stages: a stage is 16 KB and one of them is being read, so a K <= 256
// product requests all of its operands at once; a long chain keeps up to five
// chunks in flight with two CTAs on an SM.
template <int T>
int launch_tiles(GemmGroup &grp, cudaStream_t stream) {
    int max_chunks = 1;
    int64_t tiles = 0;
    for (int p = 0; p < grp.count; ++p) {
        const GemmArgs &g = grp.g[p];
        grp.tiles_n[p] = (g.n + T - 1) / T;
        tiles += (int64_t)((g.m + T - 1) / T) * grp.tiles_n[p];
        if (tiles > (1 << 30)) return PG_ERR_UNSUPPORTED;
        grp.first[p + 1] = (int)tiles;
        const int chunks = (g.k + kChunk - 1) / kChunk;
        if (chunks > max_chunks) max_chunks = chunks;
    }
    constexpr int most = T == 64 ? 5 : 6;
    grp.stages = max_chunks + 1 < most ? max_chunks + 1 : most;
    const int smem = grp.stages * kStage;
    cudaError_t err = cudaFuncSetAttribute(
        gemm_tile_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, most * kStage);
    if (err != cudaSuccess) return check_cuda(err);
    gemm_tile_kernel<T><<<(unsigned)tiles + grp.bias_first[grp.bias_count], tile_threads<T>(),
                          smem, stream>>>(grp);
    return check_cuda(cudaGetLastError());
}

int launch_group(GemmGroup &grp, cudaStream_t stream) {
    int64_t large = 0;
    for (int p = 0; p < grp.count; ++p)
        large += ((int64_t)(grp.g[p].m + 63) / 64) * ((grp.g[p].n + 63) / 64);
    int device = 0, sms = 0;
    cudaError_t err = cudaGetDevice(&device);
    if (err == cudaSuccess)
        err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (err != cudaSuccess) return check_cuda(err);
    return large >= sms ? launch_tiles<64>(grp, stream) : launch_tiles<32>(grp, stream);
}

// ---------------------------------------------------------------------------
// The 256 -> 2 layer and the column reductions
// ---------------------------------------------------------------------------
constexpr int kHid = 256;
constexpr int kHeadThreads = 256;
constexpr int kDyLd = 8;  // dY rows padded to a 16-byte chunk

// y = h W + b: a warp per 16 rows, the same products and order as the tile
// GEMM (the two columns in an 8-column tile), operands straight from global
// memory (they are read once).
__global__ void __launch_bounds__(kHeadThreads) head_forward_kernel(
    const __nv_bfloat16 *__restrict__ h, const __nv_bfloat16 *__restrict__ w,
    const float *__restrict__ bias, int m, float *__restrict__ y) {
    const int lane = threadIdx.x & 31, group = lane >> 2, tig = lane & 3;
    const int row = (int)((blockIdx.x * (unsigned)kHeadThreads + threadIdx.x) >> 5) * 16 + group;
    const uint32_t *h0 = reinterpret_cast<const uint32_t *>(h + (int64_t)min(row, m - 1) * kHid);
    const uint32_t *h1 =
        reinterpret_cast<const uint32_t *>(h + (int64_t)min(row + 8, m - 1) * kHid);
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int k0 = 0; k0 < kHid / 16; ++k0) {
        const int e = k0 * 8 + tig;  // pair of consecutive k
        const uint32_t af[4] = {h0[e], h1[e], h0[e + 4], h1[e + 4]};
        uint32_t bf[2] = {0u, 0u};
        if (group < 2) {
            bf[0] = pack_bf16(w[4 * e + group], w[4 * e + 2 + group]);
            bf[1] = pack_bf16(w[4 * (e + 4) + group], w[4 * (e + 4) + 2 + group]);
        }
        mma_bf16(acc, af, bf);
    }
    if (tig != 0) return;
    if (row < m)
        *reinterpret_cast<float2 *>(y + 2 * (int64_t)row) =
            make_float2(acc[0] + bias[0], acc[1] + bias[1]);
    if (row + 8 < m)
        *reinterpret_cast<float2 *>(y + 2 * (int64_t)(row + 8)) =
            make_float2(acc[2] + bias[0], acc[3] + bias[1]);
}

// dY = 2 (y - t) / m as bf16, the loss, and dZ of the layer before it,
// (dY W^T) gelu'(z): a CTA per 16 rows, a warp per 32 columns.
__global__ void __launch_bounds__(kHeadThreads) head_backward_kernel(
    const float *__restrict__ y, const float *__restrict__ target,
    const __nv_bfloat16 *__restrict__ w, const float *__restrict__ z, int m,
    __nv_bfloat16 *__restrict__ dy, __nv_bfloat16 *__restrict__ dz, float *__restrict__ loss) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int group = lane >> 2, tig = lane & 3;
    uint32_t af[4] = {0u, 0u, 0u, 0u};
    float l = 0.f;
    int row[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        row[r] = blockIdx.x * 16 + group + 8 * r;
        if (tig != 0 || row[r] >= m) continue;
        const float2 yy = *reinterpret_cast<const float2 *>(y + 2 * (int64_t)row[r]);
        const float2 tt = *reinterpret_cast<const float2 *>(target + 2 * (int64_t)row[r]);
        const float d0 = yy.x - tt.x, d1 = yy.y - tt.y;
        l += d0 * d0;
        l += d1 * d1;
        af[r] = pack_bf16(__float2bfloat16(2.f * d0 / (float)m),
                          __float2bfloat16(2.f * d1 / (float)m));
        if (warp == 0)
            *reinterpret_cast<uint4 *>(dy + kDyLd * (int64_t)row[r]) =
                make_uint4(af[r], 0u, 0u, 0u);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int n0 = warp * 32 + j * 8;
        const uint32_t bf[2] = {
            tig == 0 ? *reinterpret_cast<const uint32_t *>(w + 2 * (n0 + group)) : 0u, 0u};
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        mma_bf16(acc, af, bf);
        const int n = n0 + tig * 2;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            if (row[r] >= m) continue;
            const float2 zv = *reinterpret_cast<const float2 *>(z + (int64_t)row[r] * kHid + n);
            *reinterpret_cast<__nv_bfloat162 *>(dz + (int64_t)row[r] * kHid + n) =
                __floats2bfloat162_rn(acc[2 * r] * gelu_grad(zv.x),
                                      acc[2 * r + 1] * gelu_grad(zv.y));
        }
    }
    if (warp == 0) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
        if (lane == 0) atomicAdd(loss, l / (float)m);
    }
}

// Offsets of the flat parameter vector: per layer W [fan_in][fan_out], bias.
constexpr int kIn = 66, kOut = 2;
constexpr int64_t kW[4] = {0, kIn * kHid + kHid, kIn * kHid + kHid + kHid * kHid + kHid,
                           kIn * kHid + kHid + 2 * (kHid * kHid + kHid)};
constexpr int64_t bias_at(int l) {
    return kW[l] + (l == 0 ? kIn * kHid : l == 3 ? kHid * kOut : kHid * kHid);
}

GemmArgs product(const uint16_t *a, int64_t sam, int64_t sak, const uint16_t *b, int64_t sbk,
                 int64_t sbn, int m, int n, int k) {
    GemmArgs g = {};
    g.a = reinterpret_cast<const __nv_bfloat16 *>(a);
    g.sam = sam;
    g.sak = sak;
    g.b = reinterpret_cast<const __nv_bfloat16 *>(b);
    g.sbk = sbk;
    g.sbn = sbn;
    g.m = m;
    g.n = n;
    g.k = k;
    return g;
}

bool aligned_to(uintptr_t bytes, std::initializer_list<const void *> pointers) {
    for (const void *p : pointers)
        if (reinterpret_cast<uintptr_t>(p) % bytes) return false;
    return true;
}

int launch_one(const GemmArgs &g, cudaStream_t stream) {
    GemmGroup grp = {};
    if (!add_product(grp, g)) return PG_ERR_UNSUPPORTED;
    return launch_group(grp, stream);
}

}  // namespace

int launch_mlp_gemm_tile(const GemmArgs &g, cudaStream_t stream) {
    return g.k > 0 ? launch_one(g, stream) : PG_ERR_UNSUPPORTED;
}

}  // namespace pg

using namespace pg;

extern "C" {

int pg_mlp_train_forward(const uint16_t *params16, const float *params, const uint16_t *x,
                         int32_t m, int32_t stride, float *const *z, uint16_t *const *h, float *y,
                         void *stream) {
    if (m == 0) return PG_OK;
    if (!params16 || !params || !x || !h || !y || m < 0 || stride < kIn || stride % 8)
        return PG_ERR_INVALID_ARGUMENT;
    if (!aligned_to(16, {params16, x}) || !aligned_to(8, {y})) return PG_ERR_INVALID_ARGUMENT;
    for (int l = 0; l < 3; ++l)
        if (!h[l] || !aligned_to(16, {h[l]})) return PG_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    for (int l = 0; l < 3; ++l) {
        GemmArgs g = product(l == 0 ? x : h[l - 1], l == 0 ? stride : kHid, 1, params16 + kW[l],
                             kHid, 1, m, kHid, l == 0 ? kIn : kHid);
        g.bias = params + bias_at(l);
        g.epilogue = PG_MLP_EPI_GELU;
        g.zout = z ? z[l] : nullptr;
        g.ldz = kHid;
        g.c = reinterpret_cast<__nv_bfloat16 *>(h[l]);
        g.ldc = kHid;
        const int rc = launch_one(g, st);
        if (rc) return rc;
    }
    head_forward_kernel<<<(unsigned)((m + 127) / 128), kHeadThreads, 0, st>>>(
        reinterpret_cast<const __nv_bfloat16 *>(h[2]),
        reinterpret_cast<const __nv_bfloat16 *>(params16 + kW[3]), params + bias_at(3), m, y);
    return check_cuda(cudaGetLastError());
}

int pg_mlp_train_backward(const uint16_t *params16, const uint16_t *x, int32_t m, int32_t stride,
                          const float *const *z, const uint16_t *const *h, const float *y,
                          const float *target, uint16_t *work, float *grads, float *loss,
                          void *stream) {
    if (!params16 || !x || !z || !h || !y || !target || !work || !grads || !loss || m <= 0 ||
        stride < kIn || stride % 8)
        return PG_ERR_INVALID_ARGUMENT;
    if (!aligned_to(16, {params16, x, work}) || !aligned_to(8, {y, target}) ||
        !aligned_to(4, {grads, loss}))
        return PG_ERR_INVALID_ARGUMENT;
    for (int l = 0; l < 3; ++l)
        if (!z[l] || !h[l] || !aligned_to(16, {z[l], h[l]})) return PG_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    int rc = check_cuda(cudaMemsetAsync(loss, 0, sizeof(float), st));
    if (rc) return rc;
    uint16_t *dz[3];
    for (int l = 0; l < 3; ++l) dz[l] = work + (int64_t)l * m * kHid;
    uint16_t *dy = work + (int64_t)3 * m * kHid;
    head_backward_kernel<<<(unsigned)((m + 15) / 16), kHeadThreads, 0, st>>>(
        y, target, reinterpret_cast<const __nv_bfloat16 *>(params16 + kW[3]), z[2], m,
        reinterpret_cast<__nv_bfloat16 *>(dy), reinterpret_cast<__nv_bfloat16 *>(dz[2]), loss);
    if ((rc = check_cuda(cudaGetLastError()))) return rc;
    for (int l = 2; l > 0; --l) {
        // dZ of layer l - 1 = (dZ W^T) gelu'(z)
        GemmArgs g = product(dz[l], kHid, 1, params16 + kW[l], 1, kHid, m, kHid, kHid);
        g.epilogue = PG_MLP_EPI_GELU_GRAD;
        g.zin = z[l - 1];
        g.ldz = kHid;
        g.c = reinterpret_cast<__nv_bfloat16 *>(dz[l - 1]);
        g.ldc = kHid;
        if ((rc = launch_one(g, st))) return rc;
    }
    GemmGroup grp = {};
    for (int l = 0; l < 3; ++l) {
        GemmArgs g = product(l == 0 ? x : h[l - 1], 1, l == 0 ? stride : kHid, dz[l], kHid, 1,
                             l == 0 ? kIn : kHid, kHid, m);
        g.cf = grads + kW[l];
        g.ldc = kHid;
        if (!add_product(grp, g)) return PG_ERR_UNSUPPORTED;
        add_bias(grp, reinterpret_cast<const __nv_bfloat16 *>(dz[l]), m, kHid, kHid,
                 grads + bias_at(l));
    }
    GemmArgs g = product(h[2], 1, kHid, dy, kDyLd, 1, kHid, kOut, m);
    g.cf = grads + kW[3];
    g.ldc = kOut;
    if (!add_product(grp, g)) return PG_ERR_UNSUPPORTED;
    add_bias(grp, reinterpret_cast<const __nv_bfloat16 *>(dy), m, kOut, kDyLd, grads + bias_at(3));
    return launch_group(grp, st);
}

}  // extern "C"
