// Slopes, Schur form in coefficient space: the CG of slope_kernels.cuh on the
// coefficients alone, without the residual and its image per observation.
//
// With the primary dimension eliminated, S = D_r' W (I - P_p) D_r acts on the
// coefficients of the other dimensions: one large dimension L and small ones of
// Y basis columns together.  By blocks
//   S_LL = B - sum over primary groups j of V_j' M_j^-1 V_j
//          B the groups' own moments, V_j the moments of the runs (j, g): a run
//          is the rows of one pair of groups, its moments the sums of w times a
//          basis function of j times one of g
//   S_Ly [basis columns of L][Y], S_yy [Y][Y]: explicit, from S applied to the
//          small dims' unit vectors by the observation passes
// An iteration is: a_j = M_j^-1 V_j p (slope_worker_kernel, runs in primary
// order), V_j' a_j per group of L (slope_firm_kernel, runs in L's order), the
// products with S_Ly and S_yy, the vector updates.  FP64 throughout.
//
// The passes over the observations took 1,330 us an iteration (4M rows, 13
// columns, worker + firm##c.tenure + year: Q written, R read and written, both
// read through a permutation, 2.5 GB) - the runs (900,000) and S_Ly (41 MB) are
// a tenth of that and stay in L2: 185 us.
// The recursion's s can drift from the true gradient by rounding; the caller
// updates the residual with the image of the accumulated coefficients, takes the
// gradient of that, and starts again from it where it misses the threshold.

#pragma once

#include "mma_f64.cuh"
#include "slope_kernels.cuh"

namespace b200fe {

constexpr int kSpaceMaxCols = 32;      // columns of a lock step (a warp's lanes)
constexpr int kSpaceMaxSmall = 64;     // basis columns of the small dims
// Runs of one primary group (one lane slot walks them).  A call of 8 iterations, 7
// columns, every primary group with about 420 runs (1M rows) takes 3.8 ms with the form
// and 4.7 by observation passes; with 1,250 (4M rows) 11.5 and 10.7, with 2,200
// (16M rows) 28.9 and 34.8: above the limit it depends on the rows.
constexpr int kSpaceMaxRuns = 512;
// Rounds of C columns for S_Ly up to which the form is set up at once (never for a
// solve that the start already satisfies).  A solve of one check interval, 4
// iterations, on 1M rows takes 3.97 ms with the form and 3.95 by observation passes
// with 3 rounds (13 columns, 36 levels), 4.41 and 4.00 with 4, 3.24 and 2.70 with 6
// (6 columns), 4.66 and 2.82 with 16 (1 column, 16 levels).  With more rounds a check
// interval of observation passes comes first, and the form follows when at its rate
// more iterations than rounds are left: 8.0 ms for a solve of 52 iterations with 16
// rounds (7.5 with the form at once, 15.4 by observation passes).
// Up to kSpaceSureRounds that interval is left out where it cannot end the solve:
// where each of its iterations (of 4 at least) would have to lower the gradient by more
// than kSpaceDecades powers of ten of its square (random designs, the fastest seen, gain
// 2 to 3).  A solve of two intervals then gains with 6 rounds, 3.5 ms for 4.1 (6
// columns), and loses with 10, 3.3 for 3.0 (1 column); one of 56 iterations with 6
// rounds takes 6.8 ms, 7.9 after an interval of observation passes and 23.0 by them.
constexpr int kSpaceFreeRounds = 3;
constexpr int kSpaceSureRounds = 6;
constexpr double kSpaceDecades = 4.0;
constexpr int kSpaceRunBatch = 4;      // runs a slot has in flight (8: 76 us for 58 in the large dim's pass)
constexpr int kSpaceSerialChunks = 4;  // more chunks of a group: a warp sums them first
constexpr int kSpaceGroupBatch = 4;    // groups a thread of the vector updates has in flight

// per pair (j, g) in d's order: mom[q][m * d.nb + f] = sum of w times the primary's
// basis function m times g's basis function f, and j
__global__ void slope_run_moments_kernel(const SlopeDim d, const SlopeDim P, const double* __restrict__ w,
                                         const int32_t* __restrict__ start, int64_t npairs,
                                         double* __restrict__ mom, int32_t* __restrict__ primary) {
    const int K = P.nb * d.nb;
    for (int64_t q = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; q < npairs;
         q += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        double ca = 0.0, cb = 0.0, ta = 0.0, tb = 0.0;  // (1, t) x (1, z)
        const int32_t b = start[q], e = start[q + 1];
        for (int32_t pos = b; pos < e; ++pos) {
            const int32_t k = d.perm[pos];
            const double wk = w ? w[k] : 1.0;
            const double wz = d.has_b ? wk * d.z[k] : 0.0;
            const double tk = P.has_b ? P.z[k] : 0.0;
            ca += wk;
            cb += wz;
            ta = fma(wk, tk, ta);
            tb = fma(wz, tk, tb);
        }
        double* o = mom + q * K;
        if (P.has_a) {
            if (d.has_a) *o++ = ca;
            if (d.has_b) *o++ = cb;
        }
        if (P.has_b) {
            if (d.has_a) *o++ = ta;
            if (d.has_b) *o++ = tb;
        }
        primary[q] = P.ids[d.perm[b]];
    }
}

// the runs in primary order: the group of L and the moments of run ord[i]
__global__ void slope_run_order_kernel(const SlopeDim d, const int32_t* __restrict__ start,
                                       const int32_t* __restrict__ ord, int64_t npairs, int K,
                                       const double* __restrict__ mom, int32_t* __restrict__ group,
                                       double* __restrict__ mom_out) {
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < npairs;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int32_t q = ord[i];
        group[i] = d.ids[d.perm[start[q]]];
        for (int m = 0; m < K; ++m) mom_out[i * K + m] = mom[static_cast<int64_t>(q) * K + m];
    }
}

// *most = max over g of off[g + 1] - off[g] (set to 0 before)
__global__ void longest_range_kernel(const int32_t* __restrict__ off, int32_t G, int32_t* __restrict__ most) {
    int32_t m = 0;
    for (int64_t g = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; g < G;
         g += static_cast<int64_t>(gridDim.x) * blockDim.x)
        m = max(m, off[g + 1] - off[g]);
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0 && m > 0) atomicMax(most, m);
}

// blk[g * nb + f][f'] = g's moments (row f of [W Z; Z ZZ] over the basis)
__global__ void __launch_bounds__(kSlopeThreads)
slope_group_block_kernel(const SlopeDim d, const double* __restrict__ cm, double* __restrict__ blk) {
    for (int64_t base = static_cast<int64_t>(blockIdx.x) * blockDim.x; base < d.G;
         base += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int64_t g = base + threadIdx.x;
        double m[5];
        group_moments(d, cm, g, g < d.G, m);
        if (g >= d.G) continue;
        if (d.nb == 1) {
            blk[g] = d.has_a ? m[0] : m[2];
        } else {
            blk[4 * g] = m[0];
            blk[4 * g + 1] = blk[4 * g + 2] = m[1];
            blk[4 * g + 3] = m[2];
        }
    }
}

// out[(g * nb + f) * pitch + c] = the chunk sums of (g, f, c), c < cols of C, in chunk
// order (as slope_finalize_kernel takes them)
__global__ void slope_sums_kernel(const SlopeDim d, int C, int cols, int64_t pitch, double* __restrict__ out) {
    const int64_t total = static_cast<int64_t>(d.G) * d.nb * cols;
    for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < total;
         e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int64_t row = e / cols;
        const int c = static_cast<int>(e - row * cols);
        const int64_t g = row / d.nb;
        const int f = static_cast<int>(row - g * d.nb);
        double s = 0.0;
        if (d.big && d.grp_ch[g + 1] - d.grp_ch[g] > kFinSerialChunks)
            s = d.big[row * C + c];
        else
            for (int32_t j = d.grp_ch[g]; j < d.grp_ch[g + 1]; ++j)
                s += d.part[(static_cast<int64_t>(j) * d.nb + f) * C + c];
        out[row * pitch + c] = s;
    }
}

// x[(row0 + i) * C + c] = 1 where i == y0 + c, else 0, over `rows` rows
__global__ void slope_unit_kernel(double* __restrict__ x, int64_t rows, int C, int y0) {
    const int64_t total = rows * C;
    for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < total;
         e += static_cast<int64_t>(gridDim.x) * blockDim.x)
        x[e] = e / C == y0 + e % C ? 1.0 : 0.0;
}

// The coefficients of every CG dimension in one array [rows][C], dim i's from
// row0[i], a group's nb rows together.
struct SlopeSpace {
    int nd;
    int C, RB;
    int32_t G[8];
    int nb[8], has_a[8];
    int64_t row0[8];
    const double* minv[8];  // [G][3]
};

struct SlopeWorkerArgs {
    const int32_t* off;    // [Gp + 1] first run of every primary group
    const int32_t* group;  // [runs] group of L
    const double* mom;     // [runs][KP * KD]
    const double* minv;    // [Gp][3]
    int has_a;             // the primary has an intercept
    int32_t Gp;
    int C;
    const double* p;       // [G_L * KD][C]
    double* a;             // [Gp][KP][C]
};

// a_j = M_j^-1 V_j p.  Bound by the latency of the gathers (a group has two or
// three runs): a lane slot of C lanes per primary group - two groups a warp at 13
// columns - and kSpaceRunBatch runs in flight; 50 us for 400,000 groups, 240 MB
// out of L2.
template <int KP, int KD>
__global__ void __launch_bounds__(kSlopeThreads) slope_worker_kernel(const SlopeWorkerArgs a) {
    const int lane = threadIdx.x & 31;
    const int C = a.C, S = 32 / C, slot = lane / C, c = lane - slot * C;
    if (slot >= S) return;
    const int64_t step = static_cast<int64_t>(gridDim.x) * (kSlopeThreads / 32) * S;
    for (int64_t j = (static_cast<int64_t>(blockIdx.x) * (kSlopeThreads / 32) + (threadIdx.x >> 5)) * S + slot; j < a.Gp;
         j += step) {
        const int32_t b = a.off[j], e = a.off[j + 1];
        double v[KP];
#pragma unroll
        for (int m = 0; m < KP; ++m) v[m] = 0.0;
        for (int32_t i = b; i < e; i += kSpaceRunBatch) {
            int32_t g[kSpaceRunBatch];
            double x[kSpaceRunBatch][KD];
#pragma unroll
            for (int u = 0; u < kSpaceRunBatch; ++u) g[u] = i + u < e ? a.group[i + u] : -1;
#pragma unroll
            for (int u = 0; u < kSpaceRunBatch; ++u)
#pragma unroll
                for (int f = 0; f < KD; ++f)
                    x[u][f] = g[u] >= 0 ? a.p[(static_cast<int64_t>(g[u]) * KD + f) * C + c] : 0.0;
#pragma unroll
            for (int u = 0; u < kSpaceRunBatch; ++u)
                if (g[u] >= 0) {
                    const double* mr = a.mom + static_cast<int64_t>(i + u) * (KP * KD);
#pragma unroll
                    for (int m = 0; m < KP; ++m)
#pragma unroll
                        for (int f = 0; f < KD; ++f) v[m] = fma(mr[m * KD + f], x[u][f], v[m]);
                }
        }
        const double* mg = a.minv + j * 3;
        double* o = a.a + j * KP * C + c;
        if (KP == 1) {
            o[0] = v[0] * (a.has_a ? mg[0] : mg[2]);
        } else {
            o[0] = fma(mg[0], v[0], mg[1] * v[KP - 1]);
            o[C] = fma(mg[1], v[0], mg[2] * v[KP - 1]);
        }
    }
}

struct SlopeFirmArgs {
    const int32_t* ch_beg;   // chunks of runs of one group of L
    const int32_t* ch_end;
    int32_t nch;
    const int32_t* primary;  // [runs] in L's order
    const double* mom;       // [runs][KP * KD]
    const double* a;         // [Gp][KP][C]
    int C;
    double* part;            // [nch][KD][C]
};

// resident CTAs an SM of slope_firm_kernel (the grid is one wave of them)
__host__ __device__ constexpr int space_firm_ctas(int kp) { return kp == 1 ? 6 : 4; }

// chunk sums of V_j' a_j over the runs of L's groups: a warp per chunk, a lane
// slot per run, kSpaceRunBatch runs a slot in flight and the next batch's groups
// read ahead (a chunk of 64 runs is 8 steps: 58 us without, 47 with; a wave of
// CTAs with the registers for it)
template <int KP, int KD>
__global__ void __launch_bounds__(kSlopeThreads, space_firm_ctas(KP)) slope_firm_kernel(const SlopeFirmArgs a) {
    __shared__ double sred[kSlopeThreads / 32][KD][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int C = a.C, S = 32 / C, slot = lane / C, c = lane - slot * C;
    const int64_t nw = static_cast<int64_t>(gridDim.x) * (kSlopeThreads / 32);
    for (int64_t j = static_cast<int64_t>(blockIdx.x) * (kSlopeThreads / 32) + wid; j < a.nch; j += nw) {
        const int32_t b = a.ch_beg[j], e = a.ch_end[j];
        double v[KD];
#pragma unroll
        for (int f = 0; f < KD; ++f) v[f] = 0.0;
        if (slot < S) {
            int32_t next[kSpaceRunBatch];
#pragma unroll
            for (int u = 0; u < kSpaceRunBatch; ++u) {
                const int32_t i = b + slot + u * S;
                next[u] = i < e ? a.primary[i] : -1;
            }
            for (int32_t i = b + slot; i < e; i += kSpaceRunBatch * S) {
                int32_t g[kSpaceRunBatch];
                double x[kSpaceRunBatch][KP];
#pragma unroll
                for (int u = 0; u < kSpaceRunBatch; ++u) {
                    g[u] = next[u];
                    const int32_t in = i + (kSpaceRunBatch + u) * S;
                    next[u] = in < e ? a.primary[in] : -1;
                }
#pragma unroll
                for (int u = 0; u < kSpaceRunBatch; ++u)
#pragma unroll
                    for (int m = 0; m < KP; ++m)
                        x[u][m] = g[u] >= 0 ? a.a[(static_cast<int64_t>(g[u]) * KP + m) * C + c] : 0.0;
#pragma unroll
                for (int u = 0; u < kSpaceRunBatch; ++u)
                    if (g[u] >= 0) {
                        const double* mr = a.mom + static_cast<int64_t>(i + u * S) * (KP * KD);
#pragma unroll
                        for (int m = 0; m < KP; ++m)
#pragma unroll
                            for (int f = 0; f < KD; ++f) v[f] = fma(mr[m * KD + f], x[u][m], v[f]);
                    }
            }
        }
#pragma unroll
        for (int f = 0; f < KD; ++f) sred[wid][f][lane] = v[f];
        __syncwarp();
        if (lane < C)
#pragma unroll
            for (int f = 0; f < KD; ++f) {
                double t = 0.0;
                for (int s = 0; s < S; ++s) t += sred[wid][f][s * C + lane];
                a.part[(j * KD + f) * C + lane] = t;
            }
        __syncwarp();
    }
}

struct SlopeDenseArgs {
    int64_t NL;              // rows of L (G_L * KD)
    int Y, Yp;               // basis columns of the small dims, rounded up to 8
    int C;
    const double* Sly;       // [NL up to 8][Yp], zero padded
    const double* blk;       // [NL][KD]
    const double* p;         // [NL + Y][C]
    const int32_t* grp_ch;   // chunks of L's groups in part
    const double* part;      // [nch][KD][C]
    const double* big;       // groups of more than kSpaceSerialChunks chunks
    double* t;               // [NL][C] out
    double* dot;             // [grid][C] sums of p t
    double* part_y;          // [grid][Y * C] sums of S_Ly' p_L
};

// t_L = B p_L - (the chunk sums) + S_Ly p_y, and CTA partials of p_L' t_L and
// S_Ly' p_L.  A warp takes 8 rows at a time, the two products with S_Ly on the
// FP64 matrix instruction: the tile of S_Ly is read for the first and again, out
// of L1, transposed for the second, whose Yp x C sums stay in registers for the
// whole kernel.  S_Ly is 41 MB at 129,000 rows, 36 years; 29 us, bound by
// latency (two CTAs an SM for the registers of the sums).  Groups of 5 to 32
// chunks summed here, one chunk after the other, kept a few warps busy until 46 us.
template <int NT, int KD>
__global__ void __launch_bounds__(kSlopeThreads) slope_dense_kernel(const SlopeDenseArgs a) {
    constexpr int MT = kSpaceMaxSmall / 8;
    constexpr int LD = NT * 8 + 4;  // the four rows of a B fragment in different banks
    __shared__ double py[kSpaceMaxSmall * LD];  // p_y, then the partials
    __shared__ double dred[kSlopeThreads / 32][NT * 8];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, q = lane >> 2, r = lane & 3;
    const int C = a.C, mt = a.Yp / 8;
    for (int e = threadIdx.x; e < a.Yp * NT * 8; e += kSlopeThreads) {
        const int y = e / (NT * 8), c = e - y * (NT * 8);
        py[y * LD + c] = y < a.Y && c < C ? a.p[(a.NL + y) * C + c] : 0.0;
    }
    __syncthreads();
    double ty[MT][NT][2], dot[NT][2];
#pragma unroll
    for (int j = 0; j < NT; ++j) {
        dot[j][0] = dot[j][1] = 0.0;
#pragma unroll
        for (int i = 0; i < MT; ++i) ty[i][j][0] = ty[i][j][1] = 0.0;
    }
    const int64_t tiles = (a.NL + 7) / 8, nw = static_cast<int64_t>(gridDim.x) * (kSlopeThreads / 32);
    for (int64_t tile = static_cast<int64_t>(blockIdx.x) * (kSlopeThreads / 32) + wid; tile < tiles; tile += nw) {
        const int64_t r0 = tile * 8;
        const double* Sr = a.Sly + r0 * a.Yp;
        double u[NT][2];
#pragma unroll
        for (int j = 0; j < NT; ++j) u[j][0] = u[j][1] = 0.0;
#pragma unroll 5
        for (int k = 0; k < a.Yp; k += 4) {
            const double s = Sr[q * a.Yp + k + r];
#pragma unroll
            for (int j = 0; j < NT; ++j) dmma_8x8x4(u[j], s, py[(k + r) * LD + 8 * j + q]);
        }
        const int64_t row = r0 + q;
        if (row < a.NL) {
            const int64_t g = row / KD;
            const int f = static_cast<int>(row - g * KD);
            const int32_t cb = a.grp_ch[g], ce = a.grp_ch[g + 1];
            double v[NT][2], ph[NT][2][KD], bl[KD];
#pragma unroll
            for (int h = 0; h < KD; ++h) bl[h] = a.blk[row * KD + h];
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int c = 8 * j + 2 * r + e;
                    v[j][e] = 0.0;
#pragma unroll
                    for (int h = 0; h < KD; ++h) ph[j][e][h] = c < C ? a.p[(g * KD + h) * C + c] : 0.0;
                }
            // the chunks outside, the columns' loads together
            const bool big = ce - cb > kSpaceSerialChunks;
            const double* src = big ? a.big + row * C : a.part + (static_cast<int64_t>(cb) * KD + f) * C;
            const int nc = big ? 1 : ce - cb;
#pragma unroll 2
            for (int ch = 0; ch < nc; ++ch, src += KD * C)
#pragma unroll
                for (int j = 0; j < NT; ++j)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int c = 8 * j + 2 * r + e;
                        if (c < C) v[j][e] += src[c];
                    }
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int c = 8 * j + 2 * r + e;
                    if (c >= C) continue;
                    double own = 0.0, pr = 0.0;
#pragma unroll
                    for (int h = 0; h < KD; ++h) {
                        own = fma(bl[h], ph[j][e][h], own);
                        if (h == f) pr = ph[j][e][h];
                    }
                    const double t = (own - v[j][e]) + u[j][e];
                    a.t[row * C + c] = t;
                    dot[j][e] = fma(pr, t, dot[j][e]);
                }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int64_t rw = r0 + 4 * h + r;
            double pb[NT];
#pragma unroll
            for (int j = 0; j < NT; ++j) pb[j] = rw < a.NL && 8 * j + q < C ? a.p[rw * C + 8 * j + q] : 0.0;
#pragma unroll
            for (int i = 0; i < MT; ++i)
                if (i < mt) {
                    const double s = Sr[(4 * h + r) * a.Yp + 8 * i + q];
#pragma unroll
                    for (int j = 0; j < NT; ++j) dmma_8x8x4(ty[i][j], s, pb[j]);
                }
        }
    }
    // the dots: lanes of a column pair by a fixed shuffle tree, then the warps in order
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            double v = dot[j][e];
#pragma unroll
            for (int o = 4; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (q == 0) dred[wid][8 * j + 2 * r + e] = v;
        }
    __syncthreads();  // dred written, py no longer read
    if (static_cast<int>(threadIdx.x) < C) {
        double v = 0.0;
        for (int w8 = 0; w8 < kSlopeThreads / 32; ++w8) v += dred[w8][threadIdx.x];
        a.dot[static_cast<int64_t>(blockIdx.x) * C + threadIdx.x] = v;
    }
    for (int w8 = 0; w8 < kSlopeThreads / 32; ++w8) {
        if (wid == w8)
#pragma unroll
            for (int i = 0; i < MT; ++i)
                if (i < mt)
#pragma unroll
                    for (int j = 0; j < NT; ++j)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            double& x = py[(8 * i + q) * LD + 8 * j + 2 * r + e];
                            x = w8 == 0 ? ty[i][j][e] : x + ty[i][j][e];
                        }
        __syncthreads();
    }
    for (int e = threadIdx.x; e < a.Y * C; e += kSlopeThreads) {
        const int y = e / C, c = e - y * C;
        a.part_y[static_cast<int64_t>(blockIdx.x) * a.Y * C + e] = py[y * LD + c];
    }
}

// t_y = S_Ly' p_L (the partials of slope_dense_kernel) + S_yy p_y: a warp per element
__global__ void __launch_bounds__(kSlopeThreads)
slope_small_kernel(const double* __restrict__ part_y, int nparts, const double* __restrict__ Syy,
                   const double* __restrict__ p_y, int Y, int C, double* __restrict__ t_y) {
    const int lane = threadIdx.x & 31;
    const int e = static_cast<int>(blockIdx.x) * (kSlopeThreads / 32) + (threadIdx.x >> 5);
    if (e >= Y * C) return;
    const int y = e / C, c = e - y * C;
    double v = 0.0;
    for (int k = lane; k < Y; k += 32) v = fma(Syy[y * Y + k], p_y[k * C + c], v);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    v += warp_column_sum(part_y, nparts, Y * C, e);
    if (lane == 0) t_y[e] = v;
}

// scalars of one step; the next step's are written to a second set
struct SlopeScalars {
    double *gamma, *alpha;
    int* active;
};

struct SlopeStepArgs {
    SlopeSpace sp;
    SlopeScalars in, out;
    int64_t NL;
    int Y;
    int first;               // s is the gradient at the start: alpha = 0, beta = 0, x = 0
    const double* thr;       // [C]
    const double* dot;       // [ndot][C] partials of p_L' t_L
    int ndot;
    double *p, *x, *s, *t;   // [NL + Y][C]
    double* part_g;          // [grid][C] partials of s' M^-1 s
    int grid;                // CTAs of slope_space_update_kernel
    int* done;
};

// out[c] = sum over b of part[b * C + c]: thread (column, row) takes every RB-th
// partial, eight loads in flight, then the rows in order.  All threads call it.
__device__ __forceinline__ void block_column_sums(const double* __restrict__ part, int nparts, int C, int RB,
                                                  double* red, double* out) {
    const int col = threadIdx.x % C, rr = threadIdx.x / C;
    double s = 0.0;
    if (rr < RB)
        for (int b = rr; b < nparts; b += 8 * RB) {
            double v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = b + u * RB < nparts ? part[static_cast<int64_t>(b + u * RB) * C + col] : 0.0;
#pragma unroll
            for (int u = 0; u < 8; ++u) s += v[u];
        }
    column_reduce(red, s, C, RB, out);
}

// s -= alpha t and the sum of s' M^-1 s over the groups of one dim, column `col`
template <int NB>
__device__ __forceinline__ double space_update(const SlopeStepArgs& a, int i, int rr, int col, double alpha) {
    constexpr int U = kSpaceGroupBatch;
    const int C = a.sp.C;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * a.sp.RB;
    double acc = 0.0;
    for (int64_t g0 = static_cast<int64_t>(blockIdx.x) * a.sp.RB + rr; g0 < a.sp.G[i]; g0 += U * stride) {
        double s[U][NB], t[U][NB], m[U][3];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int64_t g = g0 + u * stride, o = (a.sp.row0[i] + g * NB) * C + col;
            const bool in = g < a.sp.G[i];
#pragma unroll
            for (int h = 0; h < 3; ++h) m[u][h] = in ? a.sp.minv[i][g * 3 + h] : 0.0;
#pragma unroll
            for (int f = 0; f < NB; ++f) {
                s[u][f] = in ? a.s[o + f * C] : 0.0;
                t[u][f] = in && !a.first ? a.t[o + f * C] : 0.0;
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int64_t g = g0 + u * stride, o = (a.sp.row0[i] + g * NB) * C + col;
            if (g >= a.sp.G[i]) break;
#pragma unroll
            for (int f = 0; f < NB; ++f) {
                s[u][f] = fma(-alpha, t[u][f], s[u][f]);
                if (!a.first) a.s[o + f * C] = s[u][f];
            }
            if (NB == 2) {
                const double za = fma(m[u][0], s[u][0], m[u][1] * s[u][NB - 1]);
                const double zb = fma(m[u][1], s[u][0], m[u][2] * s[u][NB - 1]);
                acc = fma(s[u][0], za, fma(s[u][NB - 1], zb, acc));
            } else {
                acc = fma(s[u][0], (a.sp.has_a[i] ? m[u][0] : m[u][2]) * s[u][0], acc);
            }
        }
    }
    return acc;
}

// x += alpha p, p = M^-1 s + beta p over the groups of one dim
template <int NB>
__device__ __forceinline__ void space_direction(const SlopeStepArgs& a, int i, int rr, int col, double alpha,
                                                double beta) {
    constexpr int U = kSpaceGroupBatch;
    const int C = a.sp.C;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * a.sp.RB;
    for (int64_t g0 = static_cast<int64_t>(blockIdx.x) * a.sp.RB + rr; g0 < a.sp.G[i]; g0 += U * stride) {
        double s[U][NB], p[U][NB], x[U][NB], m[U][3];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int64_t g = g0 + u * stride, o = (a.sp.row0[i] + g * NB) * C + col;
            const bool in = g < a.sp.G[i];
#pragma unroll
            for (int h = 0; h < 3; ++h) m[u][h] = in ? a.sp.minv[i][g * 3 + h] : 0.0;
#pragma unroll
            for (int f = 0; f < NB; ++f) {
                s[u][f] = in ? a.s[o + f * C] : 0.0;
                p[u][f] = in && !a.first ? a.p[o + f * C] : 0.0;
                x[u][f] = in && !a.first ? a.x[o + f * C] : 0.0;
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int64_t g = g0 + u * stride, o = (a.sp.row0[i] + g * NB) * C + col;
            if (g >= a.sp.G[i]) break;
            double z[NB];
            if (NB == 2) {
                z[0] = fma(m[u][0], s[u][0], m[u][1] * s[u][NB - 1]);
                z[NB - 1] = fma(m[u][1], s[u][0], m[u][2] * s[u][NB - 1]);
            } else {
                z[0] = (a.sp.has_a[i] ? m[u][0] : m[u][2]) * s[u][0];
            }
#pragma unroll
            for (int f = 0; f < NB; ++f) {
                a.x[o + f * C] = fma(alpha, p[u][f], x[u][f]);
                a.p[o + f * C] = fma(beta, p[u][f], z[f]);
            }
        }
    }
}

// alpha = gamma / p't, s -= alpha t, partials of gamma = s' M^-1 s.  Every CTA
// sums the dot partials itself (a few hundred): cheaper than a launch for it.
// Bound by latency, hence two CTAs an SM (few partials) with kSpaceGroupBatch
// groups a thread in flight: 11 us, 35 with one at a time (129,000 x 13).
__global__ void __launch_bounds__(kSlopeThreads) slope_space_update_kernel(const SlopeStepArgs a) {
    __shared__ double red[kSlopeThreads];
    __shared__ double dl[kSpaceMaxCols], al[kSpaceMaxCols];
    const int C = a.sp.C, RB = a.sp.RB, lane = threadIdx.x & 31;
    if (!a.first) block_column_sums(a.dot, a.ndot, C, RB, red, dl);
    for (int c = threadIdx.x >> 5; c < C; c += kSlopeThreads / 32) {
        double alpha = 0.0;
        if (!a.first) {
            double v = 0.0;
            for (int y = lane; y < a.Y; y += 32) v = fma(a.p[(a.NL + y) * C + c], a.t[(a.NL + y) * C + c], v);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            v += dl[c];
            alpha = a.in.active[c] && v > 0.0 ? a.in.gamma[c] / v : 0.0;
        }
        if (lane == 0) {
            al[c] = alpha;
            if (blockIdx.x == 0) a.in.alpha[c] = alpha;
        }
    }
    __syncthreads();
    const int col = threadIdx.x % C, rr = threadIdx.x / C;
    double acc = 0.0;
    if (rr < RB)
        for (int i = 0; i < a.sp.nd; ++i)
            acc += a.sp.nb[i] == 2 ? space_update<2>(a, i, rr, col, al[col]) : space_update<1>(a, i, rr, col, al[col]);
    column_reduce(red, acc, C, RB, a.part_g + static_cast<int64_t>(blockIdx.x) * C);
}

// x += alpha p, beta, p = M^-1 s + beta p, the stop test
__global__ void __launch_bounds__(kSlopeThreads) slope_space_direction_kernel(const SlopeStepArgs a) {
    __shared__ double red[kSlopeThreads];
    __shared__ double gm[kSpaceMaxCols], be[kSpaceMaxCols], al[kSpaceMaxCols];
    const int C = a.sp.C, RB = a.sp.RB;
    block_column_sums(a.part_g, a.grid, C, RB, red, gm);
    int go = 0;
    if (static_cast<int>(threadIdx.x) < C) {
        const int c = threadIdx.x;
        const double g = gm[c], old = a.in.gamma[c];
        const int was = a.first ? 1 : a.in.active[c];
        go = was && g > a.thr[c];
        al[c] = a.in.alpha[c];
        be[c] = !a.first && was && old > 0.0 ? g / old : 0.0;
        if (blockIdx.x == 0) {
            a.out.gamma[c] = was ? g : old;
            a.out.active[c] = go;
        }
    }
    go = __syncthreads_or(go);
    if (blockIdx.x == 0 && threadIdx.x == 0) *a.done = go ? 0 : 1;
    const int col = threadIdx.x % C, rr = threadIdx.x / C;
    if (rr >= RB) return;
    for (int i = 0; i < a.sp.nd; ++i) {
        if (a.sp.nb[i] == 2) space_direction<2>(a, i, rr, col, al[col], be[col]);
        else space_direction<1>(a, i, rr, col, al[col], be[col]);
    }
}

}  // namespace b200fe
