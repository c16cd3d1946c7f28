// OLS on the within-transformed columns, on the device: the data-sized parts
// of the reference's run_ols (src/ols.cpp:1237-1520, compute_covariance
// :495-700).  What touches every observation runs here with fixed-order
// reductions (bitwise reproducible); the p x p algebra stays on the host.
//
//   gram_kernel     sum_i f_i a_i b_i over the pairs (a <= b) of P columns, f_i
//                   a per-row factor or 1, on the FP64 matrix instruction:
//                     Gram  [X y]' W [X y]      f = w,          columns X, y
//                     robust meat               f = (w e)^2 (analytic weights)
//                                                   or w e^2 (frequency weights)
//                     cluster meat              f = 1, columns of the scores
//   residual_kernel e = y - x'b: the RSS sum_i w_i e_i^2, and per row w e (for
//                   the cluster scores) or the robust factor
//   cluster_*       the score sums sum w e x_j and sum w e per cluster, in
//                   cluster order
//
// Both row kernels are bound by reading the columns once (10M rows, 13 columns:
// 0.16 ms at the copy rate).  A thread per column pair out of staged shared
// memory took 0.63 ms a pass: two or three shared reads for every multiply-add.
// mma.m8n8k4 takes a lane's element of each of its two operands straight from
// global memory - the A and the B fragment of a column block have the same
// layout - and does 8 multiply-adds per lane with it.

#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "mma_f64.cuh"

#include "common_kernels.cuh"

namespace b200fe {

constexpr int kOlsMaxP = 32;      // regressors
constexpr int kOlsThreads = 256;
constexpr int kOlsChunk = 256;    // rows per cluster chunk
constexpr int kOlsSmallCluster = 32;  // clusters up to this many rows: one thread each

constexpr int kGramRows = 16;     // rows a warp takes per step
constexpr int kClusterBuf = 512;  // rows of 32 clusters a warp stages

struct GramArgs {
    int64_t n;
    int P;            // columns: X's p and, where y is given, y
    int p;
    const double* X;  // column j at X + j * ld
    int64_t ld;
    const double* y;  // or null
    const double* f;  // row factors or null
    double* partial;  // [grid][tiles][64]
};

__host__ __device__ constexpr int gram_tiles(int NB) { return NB * (NB + 1) / 2; }

// NB column blocks of 8; tile (bi, bj), bi <= bj, in row order of the upper
// triangle.  Lane (c, k) = (lane / 4, lane % 4) holds column 8 b + c of four of
// the step's rows; which rows does not matter as long as every column takes
// the same, so with VEC (16-byte aligned columns) they are two pairs.
template <int NB, bool VEC>
__global__ void __launch_bounds__(kOlsThreads) gram_kernel(const GramArgs m) {
    constexpr int NT = gram_tiles(NB);
    __shared__ double red[NT * 64];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c = lane >> 2, k = lane & 3;
    const double* col[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const int j = 8 * b + c;
        col[b] = j < m.p ? m.X + static_cast<int64_t>(j) * m.ld : (j == m.p && m.P > m.p) ? m.y : nullptr;
    }
    double acc[NT][2];
#pragma unroll
    for (int t = 0; t < NT; ++t) acc[t][0] = acc[t][1] = 0.0;
    const int64_t steps = (m.n + kGramRows - 1) / kGramRows;
    const int64_t nw = static_cast<int64_t>(gridDim.x) * (kOlsThreads / 32);
    for (int64_t st = static_cast<int64_t>(blockIdx.x) * (kOlsThreads / 32) + warp; st < steps; st += nw) {
        const int64_t r0 = st * kGramRows;
        double v[NB][4], f[4];
        if (VEC && r0 + kGramRows <= m.n) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int64_t r = r0 + 8 * q + 2 * k;
#pragma unroll
                for (int b = 0; b < NB; ++b) {
                    const double2 t = col[b] ? *reinterpret_cast<const double2*>(col[b] + r) : make_double2(0.0, 0.0);
                    v[b][2 * q] = t.x;
                    v[b][2 * q + 1] = t.y;
                }
                f[2 * q] = m.f ? m.f[r] : 1.0;
                f[2 * q + 1] = m.f ? m.f[r + 1] : 1.0;
            }
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int64_t r = r0 + 4 * q + k;
                const bool in = r < m.n;
#pragma unroll
                for (int b = 0; b < NB; ++b) v[b][q] = in && col[b] ? col[b][r] : 0.0;
                f[q] = in && m.f ? m.f[r] : 1.0;
            }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            int t = 0;
#pragma unroll
            for (int bi = 0; bi < NB; ++bi) {
                const double a = f[q] * v[bi][q];
#pragma unroll
                for (int bj = bi; bj < NB; ++bj, ++t) dmma_8x8x4(acc[t], a, v[bj][q]);
            }
        }
    }
    // warps added in order
    for (int i = threadIdx.x; i < NT * 64; i += kOlsThreads) red[i] = 0.0;
    __syncthreads();
    for (int w = 0; w < kOlsThreads / 32; ++w) {
        if (warp == w) {
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                red[t * 64 + c * 8 + 2 * k] += acc[t][0];
                red[t * 64 + c * 8 + 2 * k + 1] += acc[t][1];
            }
        }
        __syncthreads();
    }
    for (int i = threadIdx.x; i < NT * 64; i += kOlsThreads)
        m.partial[static_cast<int64_t>(blockIdx.x) * NT * 64 + i] = red[i];
}

// a warp's sum over b of part[b * stride], four reads in flight per lane
__device__ __forceinline__ double warp_partial_sum(const double* __restrict__ part, int nparts, int64_t stride) {
    double s = 0.0;
    for (int b = threadIdx.x & 31; b < nparts; b += 128) {
        double v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = b + 32 * u < nparts ? part[(b + 32 * u) * stride] : 0.0;
#pragma unroll
        for (int u = 0; u < 4; ++u) s += v[u];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// Pairs (a, b), a <= b < P, row by row of the upper triangle, from the CTAs'
// tiles; a warp per pair.
__global__ void gram_pairs_kernel(const double* __restrict__ partial, int nparts, int NB, int P,
                                  double* __restrict__ out) {
    const int npairs = P * (P + 1) / 2;
    const int nw = gridDim.x * (blockDim.x / 32);
    for (int i = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; i < npairs; i += nw) {
        int a = 0, rem = i;
        while (rem >= P - a) {
            rem -= P - a;
            ++a;
        }
        const int b = a + rem, bi = a / 8, bj = b / 8;
        const int t = bi * NB - bi * (bi - 1) / 2 + bj - bi;
        const double s = warp_partial_sum(partial + t * 64 + (a & 7) * 8 + (b & 7), nparts,
                                          static_cast<int64_t>(gram_tiles(NB)) * 64);
        if ((threadIdx.x & 31) == 0) out[i] = s;
    }
}

enum OlsRowOutput { kRowNone = 0, kRowScore = 1, kRowRobust = 2, kRowRobustFreq = 3 };

struct ResidualArgs {
    int64_t n;
    int p;
    const double* X;  // column-major, ld = n
    const double* y;
    const double* w;  // or null
    double beta[kOlsMaxP];
    int output;       // OlsRowOutput: w e, (w e)^2 or w e^2 per row
    double* row;      // [n] where output is set
    double* rss_partial;  // [grid]
};

// A thread takes two rows (VEC: 16-byte aligned columns, one load for both).
template <bool VEC>
__global__ void __launch_bounds__(kOlsThreads) residual_kernel(const ResidualArgs m) {
    __shared__ double red[kOlsThreads];
    double rss = 0.0;
    const int64_t half = (m.n + 1) / 2;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * kOlsThreads + threadIdx.x; i < half;
         i += static_cast<int64_t>(gridDim.x) * kOlsThreads) {
        const int64_t r = 2 * i;
        const bool two = r + 1 < m.n;
        double f0 = 0.0, f1 = 0.0;
#pragma unroll 4
        for (int j = 0; j < m.p; ++j) {
            const double* x = m.X + static_cast<int64_t>(j) * m.n + r;
            double2 v;
            if (VEC && two) v = *reinterpret_cast<const double2*>(x);
            else v = make_double2(x[0], two ? x[1] : 0.0);
            f0 = fma(v.x, m.beta[j], f0);
            f1 = fma(v.y, m.beta[j], f1);
        }
        const double fit[2] = {f0, f1};
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            if (q && !two) break;
            const double wr = m.w ? m.w[r + q] : 1.0;
            const double e = m.y[r + q] - fit[q];
            const double we = wr * e;
            rss = fma(we, e, rss);
            if (m.output != kRowNone)
                m.row[r + q] = m.output == kRowScore ? we : m.output == kRowRobust ? we * we : wr * e * e;
        }
    }
    red[threadIdx.x] = rss;
    __syncthreads();
    for (int h = kOlsThreads / 2; h > 0; h >>= 1) {
        if (threadIdx.x < h) red[threadIdx.x] += red[threadIdx.x + h];
        __syncthreads();
    }
    if (threadIdx.x == 0) m.rss_partial[blockIdx.x] = red[0];
}
// one warp: the CTAs' RSS
__global__ void rss_sum_kernel(const double* __restrict__ part, int nparts, double* __restrict__ out) {
    const double s = warp_partial_sum(part, nparts, 1);
    if (threadIdx.x == 0) *out = s;
}

struct ClusterArgs {
    int64_t nchunks;
    const int32_t* chunk_grp;   // cluster of each chunk
    const int32_t* chunk_beg;   // [nchunks] positions in cluster order
    const int32_t* chunk_end;
    const uint8_t* chunk_whole; // the cluster's only chunk
    const int32_t* perm;        // cluster order -> row (null: identity)
    int p;
    const double* X;
    int64_t ld;
    const double* we;           // w e per row
    int32_t G;
    double* scores;             // [p + 1][G]: sum w e x_j, then sum w e
    double* chunk_part;         // [nchunks][p + 1]
    int32_t small_max;          // whole-cluster chunks this short go to cluster_small_kernel
};

// One warp per chunk: lane l takes rows l, l + 32, ... of the chunk, then the
// lanes' sums are combined by a fixed shuffle tree.
__global__ void __launch_bounds__(kOlsThreads)
cluster_chunk_kernel(const ClusterArgs c) {
    const int lane = threadIdx.x & 31;
    const int64_t nwarps = static_cast<int64_t>(gridDim.x) * (kOlsThreads / 32);
    for (int64_t k = static_cast<int64_t>(blockIdx.x) * (kOlsThreads / 32) + (threadIdx.x >> 5);
         k < c.nchunks; k += nwarps) {
        if (c.chunk_whole[k] && c.chunk_end[k] - c.chunk_beg[k] <= c.small_max) continue;
        double s[kOlsMaxP + 1];
#pragma unroll
        for (int j = 0; j <= kOlsMaxP; ++j) s[j] = 0.0;
        for (int32_t r = c.chunk_beg[k] + lane; r < c.chunk_end[k]; r += 32) {
            const int64_t row = c.perm ? c.perm[r] : r;
            const double we = c.we[row];
#pragma unroll
            for (int j = 0; j < kOlsMaxP; ++j)
                if (j < c.p) s[j] = fma(we, c.X[static_cast<int64_t>(j) * c.ld + row], s[j]);
            s[kOlsMaxP] += we;
        }
#pragma unroll
        for (int j = 0; j <= kOlsMaxP; ++j) {
            if (j < c.p || j == kOlsMaxP) {
                double v = s[j];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                s[j] = v;
            }
        }
        if (lane == 0) {
            const bool whole = c.chunk_whole[k] != 0;
            double* dst = whole ? c.scores + c.chunk_grp[k] : c.chunk_part + k * (c.p + 1);
            const int64_t st = whole ? c.G : 1;
#pragma unroll
            for (int j = 0; j < kOlsMaxP; ++j)
                if (j < c.p) dst[j * st] = s[j];
            dst[c.p * st] = s[kOlsMaxP];
        }
    }
}

// Clusters of at most small_max rows (and empty ones): a warp takes 32
// consecutive clusters, whose rows are consecutive in cluster order; column
// after column it stages the rows' w e x_j in shared memory (coalesced) and
// every lane adds its cluster's, in cluster order (rows read by a thread per
// cluster, at a stride of a cluster, took 709 us for 10M rows and 12 columns).
// Rows beyond the buffer are read directly.  An empty cluster gets zero scores.
__global__ void __launch_bounds__(kOlsThreads)
cluster_small_kernel(const ClusterArgs c, const int32_t* __restrict__ off, int32_t G) {
    extern __shared__ double cl_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double* buf = cl_smem + warp * 2 * kClusterBuf;
    double* swe = buf + kClusterBuf;
    const int64_t nwarps = static_cast<int64_t>(gridDim.x) * (kOlsThreads / 32);
    for (int64_t g0 = (static_cast<int64_t>(blockIdx.x) * (kOlsThreads / 32) + warp) * 32; g0 < G; g0 += nwarps * 32) {
        const int64_t g = g0 + lane;
        const int32_t b = off[min(g, static_cast<int64_t>(G))], e = off[min(g + 1, static_cast<int64_t>(G))];
        const bool mine = g < G && e - b <= c.small_max;
        const int32_t rb = __shfl_sync(0xffffffffu, b, 0), re = __shfl_sync(0xffffffffu, e, 31);
        const int ns = min(re - rb, kClusterBuf);  // rows staged
        double s = 0.0;
        __syncwarp();
        for (int i = lane; i < ns; i += 32) swe[i] = c.we[c.perm ? c.perm[rb + i] : rb + i];
        __syncwarp();
        if (mine) {
            for (int32_t r = b; r < e; ++r)
                s += r - rb < ns ? swe[r - rb] : c.we[c.perm ? c.perm[r] : r];
            c.scores[static_cast<int64_t>(c.p) * G + g] = s;
        }
        for (int j = 0; j < c.p; ++j) {
            const double* x = c.X + static_cast<int64_t>(j) * c.ld;
            __syncwarp();
#pragma unroll 4
            for (int i = lane; i < ns; i += 32) buf[i] = x[c.perm ? c.perm[rb + i] : rb + i];
            __syncwarp();
            if (mine) {
                s = 0.0;
                for (int32_t r = b; r < e; ++r) {
                    if (r - rb < ns) {
                        s = fma(swe[r - rb], buf[r - rb], s);
                    } else {
                        const int64_t row = c.perm ? c.perm[r] : r;
                        s = fma(c.we[row], x[row], s);
                    }
                }
                c.scores[static_cast<int64_t>(j) * G + g] = s;
            }
        }
    }
}

// clusters the per-thread kernel takes get no chunks
__global__ void drop_small_chunks_kernel(const int32_t* __restrict__ off, int32_t G,
                                         int32_t small_max, int32_t* __restrict__ nch) {
    for (int64_t g = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; g < G;
         g += static_cast<int64_t>(gridDim.x) * blockDim.x)
        if (off[g + 1] - off[g] <= small_max) nch[g] = 0;
}

// clusters of several chunks: chunk sums in chunk order
__global__ void cluster_combine_kernel(int64_t nmulti, const int32_t* __restrict__ multi_grp,
                                       const int32_t* __restrict__ multi_c0,
                                       const int32_t* __restrict__ multi_c1,
                                       const double* __restrict__ chunk_part, int width, int32_t G,
                                       double* __restrict__ scores) {
    const int64_t total = nmulti * width;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int64_t r = i / width;
        const int j = static_cast<int>(i - r * width);
        double s = 0.0;
        for (int32_t k = multi_c0[r]; k < multi_c1[r]; ++k) s += chunk_part[static_cast<int64_t>(k) * width + j];
        scores[static_cast<int64_t>(j) * G + multi_grp[r]] = s;
    }
}

}  // namespace b200fe
