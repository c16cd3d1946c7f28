// Persistent preconditioned CG over the explicit Schur block (one launch per
// inner solve).
//
// Operator: rows [0, Gf) of the large dim (S_ff as CSR, sparse_kernels.cuh,
// plus the dense coupling C_fy x_small when a small dim is coupled) and rows
// [Gf, Gf + SG) of the small dim (C_fy' x_f + C_yy x_small).  Preconditioner:
// Jacobi (dinv).  Every column runs its own CG with its own mask; a column
// stops when r'r <= thr[c] (or r'z stops being positive) and then keeps its x.
//
// One launch of NB CTAs (all resident) runs every iteration:
//
//   A  q = S p for the large rows.  "Long" rows are cut into chunks of
//      kLongChunk nonzeros, one warp each (partials).  "Short" rows
//      (<= kShortNnz nonzeros, including empty ones) are taken twice by the
//      same warp: in row order for the products with C_fy (C_fy p_small, and
//      C_fy' p_f in registers, so C_fy is read once per iteration; the next
//      rows are copied to shared memory meanwhile), and in tiles of eight
//      rows of about equal length (PcgTiles) for the gathers of p, the next
//      tile's nonzeros copied meanwhile.  The dot p'q per CTA (by linearity
//      also for long-row chunks and small rows).
//   -- grid barrier --
//   B  alpha = r'z / p'q (every CTA reduces the NB partials in the same order,
//      so all hold the same alpha); long and small rows are finished, a warp
//      or a CTA each; r -= alpha q over the CTA's contiguous range of short
//      rows; per-CTA partials of r'z and r'r with z = dinv r.
//   -- grid barrier --
//   C  new r'z, r'r, beta, masks (again the same in every CTA); x += alpha p
//      and p = z + beta p over the CTA's contiguous range of all rows.
//   -- grid barrier --
//
// Data written by other CTAs during the launch is read with ld.global.cg (L2;
// L1 is not coherent across CTAs).  Every sum has a fixed order, so results
// are bitwise reproducible on devices of one number of SMs.  The launch is
// cooperative, one CTA per SM, and its barrier's wait is bounded (kBarrierCycles
// of clock64: on timeout it sets *status and every CTA leaves at its next
// barrier); or it is one thread-block cluster (kPcgClusterBytes), whose CTAs the
// device schedules together and which meet at the hardware's cluster barrier:
// that wait has no limit of its own, and no CTA leaves before the others.
//
// What bounds it: small systems by latency (three barriers and some ten
// dependent L2 reads an iteration), large ones by the gathers of p from L2,
// the shared-memory reads of the C_fy products and the vector passes.  Hence
// one CTA per SM, sums by shuffles with one CTA-wide barrier each, no z array,
// x updated where p is read anyway, lanes of a quad on one shared-memory
// address (an LDS.128 then takes 2 cycles instead of 4), rows in tiles of
// equal length (no lane of a warp waits for another row's nonzeros), and FP32
// -> FP64 by shifts in the gathers.  Per iteration (B200, FP32): 10k rows
// 2-way, 4 columns 28.0 -> 9.5 us; 300k rows 3-way, 4 columns 47 -> 19; 5M rows
// 3-way, 16 columns 72 -> 41 to 44; 50M rows 366 -> 248; FP64, 1M rows 3-way, 16
// columns 46 -> 30 to 32.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "sparse_kernels.cuh"

namespace b200fe {

constexpr int kShortNnz = 32;        // rows with at most this many nonzeros: one lane group
constexpr int kLongChunk = 256;      // nonzeros per warp chunk of a long row
constexpr int kPcgMaxSG = 64;        // small-dim rows the kernel handles (coupled levels)
constexpr int kHugeChunks = 16;      // long rows with more chunks: summed by a whole CTA
constexpr int kPcgRowsPerWarp = 8;   // short rows per warp step
constexpr int kPcgListsPerSm = 16;   // summation lists of C_fy' p_f per SM: the warps of the FP32 grid's CTA
constexpr int kPcgMinCtas = 16;      // CTAs of the smallest launch
constexpr int kPcgOwnRows = (kPcgMaxSG + kPcgMinCtas - 1) / kPcgMinCtas;  // small rows a CTA finishes, at most
// Whether a launch of `ctas` CTAs can hold SG small rows: CTA b keeps rows b, b + ctas, ...
// in kPcgOwnRows places.  Always so from kPcgMinCtas CTAs on; a device (or a
// partition of one) with fewer SMs than that launches fewer.
__host__ __device__ constexpr bool pcg_rows_fit(int ctas, int SG) {
    return SG <= kPcgMaxSG && SG <= ctas * kPcgOwnRows;
}
// Rows of p gathered per iteration, in bytes, up to which the launch is one
// cluster of kPcgMinCtas CTAs: there an iteration is a chain of L2 latencies
// and barriers, and the hardware barrier of 16 CTAs with 16 partials to add is
// shorter than the grid's; above it 16 SMs are too few.  us an iteration on B200,
// cluster / grid, at that many MB: 2-way panels of 10k to 1M rows in FP32 with 4
// columns 0.03: 9.3 / 13.4, 0.25: 9.9 / 13.1, 0.72: 11.8 / 13.3, 2.3: 21.8 / 14.1,
// with 16 columns 0.32: 11.7 / 16.2, 1.0: 13.4 / 16.4, 2.9: 17.7 / 16.4; in FP64 with
// 4 columns 0.50: 9.6 / 11.8, 1.4: 13.8 / 12.0, with 16 columns 0.64: 12.4 / 17.3,
// 2.0: 16.3 / 17.4, 5.8: 30.0 / 17.8.  3-way, 20 levels: FP32 0.72: 19.6 / 20.6; FP64,
// 16 columns 0.65: 17.0 / 21.6, 2.0: 24.9 / 22.3.
constexpr double kPcgClusterBytes = 1e6;
constexpr long long kBarrierCycles = 4000000000LL;  // ~2 s at 1.9 GHz

// One CTA per SM (16 warps in FP32, kPcgListsPerSm): half as many arrivals and partials per grid barrier as with
// two, and the registers a thread needs (128 in FP32, more in FP64).
template <typename T>
__host__ __device__ constexpr int pcg_threads() {
    return sizeof(T) == 4 ? 512 : 256;
}

template <typename T>
struct PcgArgs {
    int CP;
    int64_t Gf;                 // rows of the large dim (alpha rows 0..Gf-1)
    int SG, SGP;                // small-dim rows (0 without coupling); C_fy row stride
    const int32_t* row_off;     // [Gf+1] CSR of S_ff
    const int32_t* col;
    const T* val;
    int64_t nshort;
    const int32_t* short_rows;  // rows of at most kShortNnz nonzeros, ascending
    int64_t ntiles;             // tiles of short rows (PcgTiles)
    const int2* tile_meta;      // {first entry / 4, entries}
    const int2* tile_rows;      // [ntiles][8] {row or -1, first entry in the tile | nonzeros << 16}
    const int32_t* tile_col;
    const T* tile_val;
    int lists;                  // summation lists of C_fy' p_f (see the kernel)
    int cbuf;                   // staging buffers of the coupling step (1 or 2)
    int64_t nlchunks;           // chunks of long rows (kLongChunk nonzeros each)
    const int4* lchunk_meta;    // {row, begin, end, 1 for the row's first chunk}
    int64_t nlong;
    const int4* long_meta;      // [nlong] {row, first chunk, last chunk + 1, 0}
    int64_t nhuge;              // long rows of more than kHugeChunks chunks
    const int32_t* huge_li;     // [nhuge] their index in long_meta
    const T* cfy;               // [Gf][SGP] or null
    const double* cyy;          // [SG][SG] or null
    const T* dinv;              // [GR]
    T* x;
    T* r;
    T* p;
    T* q;
    double* lpart;              // [nlchunks][CP]
    double* cta_part;           // [NB][part_stride]
    int part_stride;            // CP * (3 + SG): pq | C_fy'p [SG][CP] | rz | rr
    const double* thr;          // [CP] stop threshold on r'r (<= 0: column inactive)
    int max_iter;
    // outputs for the host
    double* rz_out;             // [CP]
    int* iters_out;             // [CP] iterations while active
    int* loops_out;             // [1] iterations run
    unsigned int* bar;          // [1] grid barrier: arrivals since the launch (zero at launch)
    int* status;                // [1] 0 ok; 2 barrier timeout
};

__device__ __forceinline__ void v4_load_cg(const float* p, V4<float>& o) {
    const float4 t = __ldcg(reinterpret_cast<const float4*>(p));
    o.v[0] = t.x; o.v[1] = t.y; o.v[2] = t.z; o.v[3] = t.w;
}
__device__ __forceinline__ void v4_load_cg(const double* p, V4<double>& o) {
    const double2 a = __ldcg(reinterpret_cast<const double2*>(p));
    const double2 b = __ldcg(reinterpret_cast<const double2*>(p) + 1);
    o.v[0] = a.x; o.v[1] = a.y; o.v[2] = b.x; o.v[3] = b.y;
}
__device__ __forceinline__ void v4_store(float* p, const V4<float>& a) {
    *reinterpret_cast<float4*>(p) = make_float4(a.v[0], a.v[1], a.v[2], a.v[3]);
}
__device__ __forceinline__ void v4_store(double* p, const V4<double>& a) {
    reinterpret_cast<double2*>(p)[0] = make_double2(a.v[0], a.v[1]);
    reinterpret_cast<double2*>(p)[1] = make_double2(a.v[2], a.v[3]);
}

// A warp's slab in shared memory (byte offsets): two buffers of a tile's
// {columns, values}; with a coupled small dim cbuf buffers of a coupling
// step's rows of {p, C_fy} and one such row; the warp's C_fy' p_f in FP64
// [SG][CP] takes the front of the slab at the end of phase A.
template <typename T>
struct PcgSlab {
    int val, buf, step, step_bytes, row, bytes;
    __host__ __device__ constexpr PcgSlab(int CP, int SG, int SGP, int cbuf)
        : val(kPcgRowsPerWarp * kShortNnz * 4),
          buf(val + kPcgRowsPerWarp * kShortNnz * static_cast<int>(sizeof(T))),
          step(2 * buf),
          step_bytes(SG > 0 ? 128 / CP * (CP + SGP) * static_cast<int>(sizeof(T)) : 0),
          row(step + cbuf * step_bytes),
          bytes(row + (SG > 0 ? (CP + SGP) * static_cast<int>(sizeof(T)) : 0)) {
        if (bytes < SG * CP * 8) bytes = SG * CP * 8;
    }
};
// Dynamic shared memory of pcg_persistent_kernel: small rows of p [64][CP] and
// the warps' slabs.
template <typename T>
__host__ __device__ constexpr size_t pcg_smem_bytes(int CP, int SG, int SGP, int cbuf) {
    return align16(static_cast<size_t>(kPcgMaxSG) * CP * sizeof(T)) +
           static_cast<size_t>(pcg_threads<T>() / 32) * PcgSlab<T>(CP, SG, SGP, cbuf).bytes;
}

// 16-byte asynchronous copy global -> shared (cached in L2 only); the
// caller commits, waits and then __syncwarp()s before other lanes read it.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned sa = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// z = M^-1 r: the FP32 product rounded once, as the exact FP64 product would be
__device__ __forceinline__ float precond(float d, float r) { return __fmul_rn(d, r); }
__device__ __forceinline__ double precond(double d, double r) { return __dmul_rn(d, r); }

// q += sum over nonzeros j of val[j] p[col[j]] (4 columns of this lane) for
// j = j0, j0 + step, ... < je, U nonzeros per batch; the next batch's column
// ids and values are loaded while the current batch's rows of p are gathered.
template <typename T, int CP, int U>
__device__ __forceinline__ void gather_rows(const int32_t* __restrict__ col, const T* __restrict__ val,
                                            const T* p, int32_t j0, int32_t je, int step, int q4,
                                            Acc4& acc) {
    int32_t cj[U];
    T vj[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int32_t j = j0 + u * step;
        cj[u] = j < je ? __ldg(col + j) : -1;
        vj[u] = j < je ? __ldg(val + j) : T(0);
    }
    for (int32_t jb = j0; jb < je; jb += U * step) {
        V4<T> xv[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (cj[u] >= 0) v4_load_cg(p + static_cast<int64_t>(cj[u]) * CP + 4 * q4, xv[u]);
            else v4_zero(xv[u]);
        }
        double vc[U];
#pragma unroll
        for (int u = 0; u < U; ++u) vc[u] = static_cast<double>(vj[u]) * unscale64<T>();
        const int32_t jn = jb + U * step;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int32_t j = jn + u * step;
            cj[u] = j < je ? __ldg(col + j) : -1;
            vj[u] = j < je ? __ldg(val + j) : T(0);
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int i = 0; i < 4; ++i)
                acc.v[i] = fma(vc[u], scaled64(xv[u].v[i]), acc.v[i]);
    }
}

template <typename T>
__device__ __forceinline__ void lds4(const T* p, T (&v)[4]);
template <>
__device__ __forceinline__ void lds4<float>(const float* p, float (&v)[4]) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
}
template <>
__device__ __forceinline__ void lds4<double>(const double* p, double (&v)[4]) {
    const double2 a = reinterpret_cast<const double2*>(p)[0];
    const double2 b = reinterpret_cast<const double2*>(p)[1];
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}

// C_fy' p_f in registers: lane (hs, q4) keeps levels hs, hs + HS, ... (KH of
// them) of column quad q4, row after row.
template <typename T, int CQ, int KH>
struct PcgCouple {
    static constexpr int CP = 4 * CQ;
    static constexpr int HS = 32 / CQ;
    T acc[KH][4];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int k = 0; k < KH; ++k)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[k][i] = T(0);
    }
    __device__ __forceinline__ void row(const T* crow, const T* prow, int SG, int hs, int q4) {
        T pv[4];
        lds4<T>(prow + 4 * q4, pv);
#pragma unroll
        for (int k = 0; k < KH; ++k) {
            const int h = hs + HS * k;
            const T c = h < SG ? crow[h] : T(0);
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[k][i] = fma(c, pv[i], acc[k][i]);
        }
    }
};
// C_fy[row] p_small for a column quad of xs (rows of CP), level after level
template <typename T, int CP>
__device__ __forceinline__ void couple_dot(const T* crow, const T* xs, int SGP, T (&cs)[4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) cs[i] = T(0);
#pragma unroll 2
    for (int h = 0; h < SGP; h += 4) {
        T c4[4];
        lds4<T>(crow + h, c4);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            T xr[4];
            lds4<T>(xs + (h + u) * CP, xr);
#pragma unroll
            for (int i = 0; i < 4; ++i) cs[i] = fma(c4[u], xr[i], cs[i]);
        }
    }
}

// CLUSTER: the whole grid is one thread-block cluster and meets at the
// hardware cluster barrier; otherwise a cooperative launch of one CTA per SM.
// KH: levels of the small dim per lane (PcgCouple); 0 without coupling.
//
// C_fy' p_f is summed in the solve precision over a.lists lists (list v: the
// first chunks of long rows among chunks v, v + lists, ..., then steps
// v, v + lists, ... of 32 / CQ short rows in row order), the lists' sums in
// FP64; a warp takes whole lists.  C_fy's rows cancel (a balanced row sums to
// zero over the levels), so the rounding of these FP32 sums shows in badly
// identified rows of the answer: the lists follow from the number of SMs
// (kPcgListsPerSm each), and neither they nor the level order of C_fy p_small
// depend on whether the launch is a cluster or the grid, so that the answer
// depends on that only through FP64 rounding.
template <typename T, int CQ, int KH, bool CLUSTER>
__global__ void __launch_bounds__(pcg_threads<T>(), 1) pcg_persistent_kernel(const PcgArgs<T> a) {
    constexpr unsigned kFull = 0xffffffffu;
    constexpr bool coupled = KH > 0;
    constexpr bool LISTS = coupled && CLUSTER && sizeof(T) == 4;  // a warp takes several lists
    constexpr int NT = pcg_threads<T>();
    constexpr int NW = NT / 32;
    constexpr int CP = 4 * CQ;
    static_assert(sizeof(T) != 4 || NW == kPcgListsPerSm, "one list per warp of the FP32 grid");
    constexpr int RW = kPcgRowsPerWarp;
    constexpr int LPR = 32 / RW;  // lanes per short row
    constexpr int SR = 32 / CQ;   // short rows per coupling step
    constexpr int J = LPR / CQ;   // of which this many share a column quad
    constexpr int U = sizeof(T) == 4 ? 8 : 4;  // gathers in flight per lane
    __shared__ double red_q[2][NW][CP], red_c[2][NW][CP], red_s[2][NW][CP];
    __shared__ double s_alpha[CP], s_beta[CP], s_rz[CP];
    __shared__ int s_active[CP], s_iters[CP];
    __shared__ int s_any, s_ok;
    __shared__ double s_cyy[coupled ? kPcgOwnRows : 1][kPcgMaxSG], s_yq[kPcgOwnRows][CP];  // this CTA's small rows
    extern __shared__ __align__(16) unsigned char pcg_smem_raw[];
    T* s_xs = reinterpret_cast<T*>(pcg_smem_raw);  // [kPcgMaxSG][CP] small rows of p
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;
    const int NB = gridDim.x;
    const int b = blockIdx.x;
    const int64_t GR = a.Gf + a.SG;
    const int PS = a.part_stride;
    const int SG = a.SG, SGP = a.SGP;
    double* mypart = a.cta_part + static_cast<int64_t>(b) * PS;
    const PcgSlab<T> sl(CP, SG, SGP, a.cbuf);
    unsigned char* s_slabs = pcg_smem_raw + align16(static_cast<size_t>(kPcgMaxSG) * CP * sizeof(T));
    unsigned char* slab = s_slabs + static_cast<size_t>(warp) * sl.bytes;  // this warp's staging
    // contiguous row range owned by this CTA (updates, directions)
    const int64_t r0 = GR * b / NB, r1 = GR * (b + 1) / NB;
    const int c_of_t = tid % CP;  // column of this thread where a thread owns one column
    const int tq = tid % CQ;      // column quad of this thread where it owns four
    // lane (gw, jl, q4): row gw of a tile, every J-th of its nonzeros from jl on,
    // column quad q4; once the J shares have met, the lane owns columns
    // oc .. oc + CQ of the row.  With the row in the low bits, lanes of one
    // quad share the address of a row of p_small or p in shared memory.
    const int gw = lane & (RW - 1);
    const int q4 = (lane / RW) % CQ;
    const int jl = lane / (RW * CQ);
    const int oc = 4 * q4 + jl * CQ;
    const int hs = gw + RW * jl;
    const int npairs = SG * CP;
    unsigned int epoch = 0;

    // CTA sums of K values: v[k][i] of column 4 (lane % CQ) + i, and w[k] of
    // column lane % CP; thread c < CP stores the sum of column c at
    // mypart[off[k] + c], then the grid meets.  Everything the CTA wrote
    // before is visible to the CTAs that have passed the barrier.
    auto publish = [&](auto& v, auto& w, const int (&off)[2], int K) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            if (k >= K) break;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                double t = v[k][i];
#pragma unroll
                for (int o = 16; o >= CQ; o >>= 1) t += __shfl_xor_sync(kFull, t, o);
                if (lane < CQ) red_q[k][warp][4 * lane + i] = t;
            }
            double t = w[k];
#pragma unroll
            for (int o = 16; o >= CP; o >>= 1) t += __shfl_xor_sync(kFull, t, o);
            if (lane < CP) red_c[k][warp][lane] = t;
        }
        __syncthreads();
        if (tid < CP) {
            for (int k = 0; k < K; ++k) {
                double s = 0.0;
#pragma unroll
                for (int j = 0; j < NW; ++j) s += red_q[k][j][tid] + red_c[k][j][tid];
                mypart[off[k] + tid] = s;
            }
        }
    };
    // the same for p'q: dot of columns oc .. in the lanes gw = 0, w of column lane % CP
    auto publish_own = [&](const double (&dot)[CQ], const double (&w)[2]) {
        if (gw == 0) {
#pragma unroll
            for (int i = 0; i < CQ; ++i) red_q[0][warp][oc + i] = dot[i];
        }
        double t = w[0];
#pragma unroll
        for (int o = 16; o >= CP; o >>= 1) t += __shfl_xor_sync(kFull, t, o);
        if (lane < CP) red_c[0][warp][lane] = t;
        __syncthreads();
        if (tid < CP) {
            double s = 0.0;
#pragma unroll
            for (int j = 0; j < NW; ++j) s += red_q[0][j][tid] + red_c[0][j][tid];
            mypart[tid] = s;
        }
    };
    auto meet = [&]() -> bool {
        if (CLUSTER) {
            asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
            return true;
        }
        ++epoch;
        if (warp == 0) {
            __syncwarp();
            if (lane == 0) {
                int ok = 1;
                const unsigned int target = epoch * static_cast<unsigned int>(NB);
                __threadfence();
                asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(a.bar) : "memory");
                unsigned int seen;
                long long t0 = 0;
                for (unsigned int spin = 1;; ++spin) {
                    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(a.bar) : "memory");
                    if (seen >= target) break;
                    if ((spin & 255u) == 0) {  // now and then: has the wait run out, here or elsewhere
                        const long long t = clock64();
                        if (t0 == 0) t0 = t;
                        if (*reinterpret_cast<volatile int*>(a.status) != 0 || t - t0 > kBarrierCycles) {
                            atomicOr(a.status, 2);
                            ok = 0;
                            break;
                        }
                    }
                }
                s_ok = ok;
            }
        }
        __syncthreads();
        return s_ok != 0;
    };
    // sum over CTAs of part[cta * stride + off[k] + c]: returned to threads
    // c < CP (fixed order: a thread's slice, a shuffle tree, the warps in order)
    auto col_sums = [&](const double* part, int nparts, int stride, int off0, int off1, int K, double (&out)[2]) {
        double s[2] = {0.0, 0.0};
        for (int i = tid / CP; i < nparts; i += NT / CP) {
            const double* src = part + static_cast<int64_t>(i) * stride + c_of_t;
            s[0] += __ldcg(src + off0);
            if (K > 1) s[1] += __ldcg(src + off1);
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            if (k >= K) break;
#pragma unroll
            for (int o = 16; o >= CP; o >>= 1) s[k] += __shfl_xor_sync(kFull, s[k], o);
            if (lane < CP) red_s[k][warp][lane] = s[k];
        }
        __syncthreads();
        out[0] = out[1] = 0.0;
        if (tid < CP) {
            for (int k = 0; k < K; ++k) {
                double t = 0.0;
#pragma unroll
                for (int j = 0; j < NW; ++j) t += red_s[k][j][tid];
                out[k] = t;
            }
        }
    };
    const int off_rr[2] = {CP * (1 + SG), CP * (2 + SG)};

    if (coupled)
        for (int i = tid; i < kPcgOwnRows * SG; i += NT) {
            const int k = i / SG, h = b + k * NB;
            if (h < SG) s_cyy[k][i - k * SG] = __ldg(a.cyy + h * SG + i - k * SG);
        }

    // ---- init: x = 0, p = z = dinv r; partials of r'z, r'r ----
    // (streaming loops: a thread owns column quad tq of rows in its CTA's
    // range, two quads in flight, every load issued before the stores)
    {
        double v[2][4] = {}, w[2] = {0.0, 0.0};
        const int64_t e1 = r1 * CQ;
        for (int64_t e = r0 * CQ + tid; e < e1; e += NT) {
            V4<T> rv, zv, xz;
            v4_load_cg(a.r + 4 * e, rv);
            const T dv = __ldg(a.dinv + e / CQ);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const double ri = static_cast<double>(rv.v[i]);
                zv.v[i] = precond(dv, rv.v[i]);
                xz.v[i] = T(0);
                v[0][i] = fma(ri, static_cast<double>(zv.v[i]), v[0][i]);
                v[1][i] = fma(ri, ri, v[1][i]);
            }
            v4_store(a.x + 4 * e, xz);
            v4_store(a.p + 4 * e, zv);
        }
        publish(v, w, off_rr, 2);
    }
    if (!meet()) return;
    {
        double s[2];
        col_sums(a.cta_part, NB, PS, off_rr[0], off_rr[1], 2, s);
        if (warp == 0) {
            int act = 0;
            if (lane < CP) {
                s_rz[lane] = s[0];
                s_iters[lane] = 0;
                act = (a.thr[lane] > 0.0 && s[1] > a.thr[lane] && s[0] > 0.0) ? 1 : 0;
                s_active[lane] = act;
            }
            const int any = __any_sync(kFull, act);
            if (lane == 0) s_any = any;
        }
        __syncthreads();
    }

    const int64_t nwarps = static_cast<int64_t>(NB) * NW;
    // warps of different CTAs get neighbouring work items, so that few items
    // spread over many SMs
    const int64_t wid = static_cast<int64_t>(warp) * NB + b;
    int it = 0;
    while (s_any && it < a.max_iter) {
        // ================= A: q = S p, C_fy' p_f, dots =================
        if (coupled) {
            for (int i = tid; i < SGP * CP; i += NT) s_xs[i] = i < npairs ? __ldcg(a.p + a.Gf * CP + i) : T(0);
            __syncthreads();
        }
        double w[2] = {0.0, 0.0}, dot[CQ] = {};  // dot: the lane's own columns
        // C_fy' p_f of the warp's current list, and of its lists before (an FP32
        // grid has one list per warp, an FP64 sum needs no lists)
        PcgCouple<T, CQ, coupled ? KH : 1> cpl;
        cpl.zero();
        double cdot[LISTS ? KH : 1][4] = {};
        // own columns of a quad's sums
        auto own = [&](const Acc4& acc, double (&o)[CQ]) {
#pragma unroll
            for (int i = 0; i < CQ; ++i) {
                o[i] = acc.v[i];
#pragma unroll
                for (int j = 1; j < J; ++j)
                    if (jl == j) o[i] = acc.v[j * CQ + i];
            }
        };
        // rows of a coupling step: lane (sr, sq) stages and owns quad sq of row sr
        const int sr = lane % SR, sq = lane / SR;
        const int64_t nsteps = coupled ? (a.nshort + SR - 1) / SR : 0;
        const int64_t lists = coupled ? a.lists : nwarps;
        for (int64_t v = wid; v < lists; v += nwarps) {
            if (coupled && v >= a.nlchunks && v >= nsteps) break;  // this list and the later ones are empty
            T* srow = reinterpret_cast<T*>(slab + sl.row);
            // ---- long-row chunks: a warp each, lane groups interleave the
            // nonzeros; the next chunk's record is loaded one chunk ahead
            int4 lm = v < a.nlchunks ? __ldg(a.lchunk_meta + v) : make_int4(0, 0, 0, 0);
            // the first rows of the coupling do not depend on the chunks
            int64_t st = v;
            auto short_row = [&](int64_t step) {
                const int64_t i = step * SR + sr;
                return step < nsteps && i < a.nshort ? __ldg(a.short_rows + i) : -1;
            };
            int32_t g = coupled ? short_row(st) : -1;
            auto stage_step = [&](int k) {
                T* d = reinterpret_cast<T*>(slab + sl.step + k * sl.step_bytes);
                constexpr int VT = 16 / sizeof(T);  // elements per 16-byte copy
                if (g >= 0) {
#pragma unroll
                    for (int i = 0; i < 4 / VT; ++i)
                        cp_async16(d + sr * CP + 4 * sq + i * VT, a.p + static_cast<int64_t>(g) * CP + 4 * sq + i * VT);
                    T* c = d + SR * CP + sr * SGP;
                    const T* src = a.cfy + static_cast<int64_t>(g) * SGP;
                    for (int i = sq; i < SGP / VT; i += CQ) cp_async16(c + i * VT, src + i * VT);
                }
                cp_async_commit();
            };
            if (coupled) stage_step(0);
            for (int64_t ch = v; ch < a.nlchunks; ch += lists) {
                const int32_t row = lm.x, jb = lm.y, je = lm.z;
                const bool first = lm.w != 0;
                if (ch + lists < a.nlchunks) lm = __ldg(a.lchunk_meta + ch + lists);
                T pv[CQ], cs[4] = {};
#pragma unroll
                for (int i = 0; i < CQ; ++i) pv[i] = __ldcg(a.p + static_cast<int64_t>(row) * CP + oc + i);
                if (coupled && first) {  // the row's first chunk carries its products with C_fy
                    for (int h = lane; h < SGP; h += 32)
                        srow[CP + h] = __ldg(a.cfy + static_cast<int64_t>(row) * SGP + h);
                    if (gw == 0) {
#pragma unroll
                        for (int i = 0; i < CQ; ++i) srow[oc + i] = pv[i];
                    }
                    __syncwarp();
                    couple_dot<T, CP>(srow + CP, s_xs + 4 * q4, SGP, cs);
                    cpl.row(srow + CP, srow, SG, sr, sq);
                    __syncwarp();
                }
                Acc4 acc;
                acc_zero(acc);
                gather_rows<T, CP, U>(a.col, a.val, a.p, jb + hs, je, 32 / CQ, q4, acc);
                // lane groups of the warp combined by a butterfly
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    if (o >= RW && o < RW * CQ) continue;  // the lane bits of the column quad
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc.v[i] += __shfl_xor_sync(kFull, acc.v[i], o);
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) acc.v[i] += static_cast<double>(cs[i]);
                double qo[CQ];
                own(acc, qo);
                if (gw == 0) {
                    double* dst = a.lpart + ch * CP + oc;
#pragma unroll
                    for (int i = 0; i < CQ; ++i) {
                        dst[i] = qo[i];
                        dot[i] = fma(static_cast<double>(pv[i]), qo[i], dot[i]);
                    }
                }
            }
            // ---- the list's short rows in order, SR per step: C_fy p_small into
            // q (completed below by this warp) and C_fy' p_f
            if (coupled) {
                for (int k = 0; st < nsteps; st += lists) {
                    const int32_t gc = g;
                    const unsigned rows = __ballot_sync(kFull, sq == 0 && gc >= 0);
                    g = short_row(st + lists);
                    cp_async_wait_all();
                    __syncwarp();
                    const T* d = reinterpret_cast<const T*>(slab + sl.step + k * sl.step_bytes);
                    if (a.cbuf == 2) stage_step(k ^= 1);
                    if (gc >= 0) {
                        T cs[4];
                        couple_dot<T, CP>(d + SR * CP + sr * SGP, s_xs + 4 * sq, SGP, cs);
                        V4<T> o;
#pragma unroll
                        for (int i = 0; i < 4; ++i) o.v[i] = cs[i];
                        v4_store(a.q + static_cast<int64_t>(gc) * CP + 4 * sq, o);
                    }
                    // rows of a step are a prefix of it
                    const int nr = __popc(rows);
#pragma unroll 8
                    for (int r = 0; r < nr; ++r) cpl.row(d + SR * CP + r * SGP, d + r * CP, SG, sr, sq);
                    __syncwarp();
                    if (a.cbuf == 1) stage_step(0);
                }
                cp_async_wait_all();
                if constexpr (LISTS) {
#pragma unroll
                    for (int k = 0; k < KH; ++k)
#pragma unroll
                        for (int i = 0; i < 4; ++i) cdot[k][i] += static_cast<double>(cpl.acc[k][i]);
                    cpl.zero();
                }
                __syncwarp();
            }
            // ---- the same rows (without coupling: any) in tiles of about equal length
            int64_t t = v, te = a.ntiles;
            const int64_t ts = coupled ? 1 : nwarps;
            if (coupled) {
                const int64_t full = nsteps / lists, rest = nsteps - full * lists;
                t = (v * full + min(v, rest)) * (SR / RW);
                te = ((v + 1) * full + min(v + 1, rest)) * (SR / RW);
            }
            int2 tm = t < te ? __ldg(a.tile_meta + t) : make_int2(0, 0);
            int2 row = t < te ? __ldg(a.tile_rows + t * RW + gw) : make_int2(-1, 0);
            auto stage_tile = [&](int k) {
                unsigned char* d = slab + k * sl.buf;
                const unsigned char* c = reinterpret_cast<const unsigned char*>(a.tile_col + 4 * static_cast<int64_t>(tm.x));
                const unsigned char* x = reinterpret_cast<const unsigned char*>(a.tile_val + 4 * static_cast<int64_t>(tm.x));
                const int n16 = (tm.y + 3) >> 2;  // 16-byte pieces of the columns
                for (int i = lane; i < n16; i += 32) cp_async16(d + 16 * i, c + 16 * i);
                for (int i = lane; i < n16 * static_cast<int>(sizeof(T) / 4); i += 32)
                    cp_async16(d + sl.val + 16 * i, x + 16 * i);
                cp_async_commit();
            };
            stage_tile(0);
            for (int k = 0; t < te; t += ts, k ^= 1) {
                const int32_t gr = row.x;
                const int e0 = row.y & 0xffff, len = row.y >> 16;
                const int longest = __reduce_max_sync(kFull, len);
                T pv[CQ], cs[CQ] = {};
                if (gr >= 0) {
#pragma unroll
                    for (int i = 0; i < CQ; ++i) {
                        pv[i] = __ldcg(a.p + static_cast<int64_t>(gr) * CP + oc + i);
                        if (coupled) cs[i] = __ldcg(a.q + static_cast<int64_t>(gr) * CP + oc + i);
                    }
                }
                tm = t + ts < te ? __ldg(a.tile_meta + t + ts) : make_int2(0, 0);
                row = t + ts < te ? __ldg(a.tile_rows + (t + ts) * RW + gw) : make_int2(-1, 0);
                cp_async_wait_all();
                __syncwarp();
                const unsigned char* d = slab + k * sl.buf;
                const int32_t* tc = reinterpret_cast<const int32_t*>(d) + e0;
                const T* tv = reinterpret_cast<const T*>(d + sl.val) + e0;
                Acc4 acc;
                acc_zero(acc);
                bool staged = false;
                for (int jb = jl; jb < longest || !staged; jb += J * U) {
                    V4<T> xv[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int j = jb + u * J;
                        if (j < len) v4_load_cg(a.p + static_cast<int64_t>(tc[j]) * CP + 4 * q4, xv[u]);
                        else v4_zero(xv[u]);
                    }
                    if (!staged) {  // behind the first gathers: the next tile's copies
                        stage_tile(k ^ 1);
                        staged = true;
                    }
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int j = jb + u * J;
                        const double vj = j < len ? static_cast<double>(tv[j]) * unscale64<T>() : 0.0;
#pragma unroll
                        for (int i = 0; i < 4; ++i) acc.v[i] = fma(vj, scaled64(xv[u].v[i]), acc.v[i]);
                    }
                }
                __syncwarp();
#pragma unroll
                for (int o = RW * CQ; o < 32; o <<= 1)
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc.v[i] += __shfl_xor_sync(kFull, acc.v[i], o);
                double qo[CQ];
                own(acc, qo);
                if (gr >= 0) {
#pragma unroll
                    for (int i = 0; i < CQ; ++i) {
                        const T qs = static_cast<T>(qo[i] + static_cast<double>(cs[i]));
                        a.q[static_cast<int64_t>(gr) * CP + oc + i] = qs;
                        // dot with the stored (rounded) value
                        dot[i] = fma(static_cast<double>(pv[i]), static_cast<double>(qs), dot[i]);
                    }
                }
            }
            cp_async_wait_all();
            __syncwarp();
        }
        // this CTA's C_fy' p_f, and its share of p'q: the row dots above plus
        // p_small . (C_fy' p_f partial), plus p_small' C_yy p_small dealt over
        // the CTAs by level
        if (coupled) {
            double* dump = reinterpret_cast<double*>(slab);  // [SG][CP]
#pragma unroll
            for (int k = 0; k < KH; ++k) {
                const int h = sr + SR * k;
                if (h < SG) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if constexpr (LISTS) dump[h * CP + 4 * sq + i] = cdot[k][i];
                        else dump[h * CP + 4 * sq + i] = static_cast<double>(cpl.acc[k][i]);
                    }
                }
            }
            __syncthreads();
            for (int pr = tid; pr < npairs; pr += NT) {
                double cp = 0.0;  // pr % CP == c_of_t
#pragma unroll
                for (int k = 0; k < NW; ++k) cp += reinterpret_cast<const double*>(s_slabs + k * sl.bytes)[pr];
                mypart[CP + pr] = cp;
                w[0] = fma(static_cast<double>(s_xs[pr]), cp, w[0]);
            }
            // rows b, b + NB, ... of C_yy p_small, by CP threads each from the last warp down
            const int k = (NT - 1 - tid) / CP, h = b + k * NB;
            if (k < kPcgOwnRows && h < SG) {
                double yq = 0.0;
                for (int h2 = 0; h2 < SG; ++h2)
                    yq = fma(s_cyy[k][h2], static_cast<double>(s_xs[h2 * CP + c_of_t]), yq);
                s_yq[k][c_of_t] = yq;
                w[0] = fma(static_cast<double>(s_xs[h * CP + c_of_t]), yq, w[0]);
            }
        }
        // own columns into the quads' order: lane (0, jl, q4) holds columns oc ..
#pragma unroll
        for (int i = 0; i < CQ; ++i) {
#pragma unroll
            for (int o = RW / 2; o > 0; o >>= 1) dot[i] += __shfl_xor_sync(kFull, dot[i], o);
        }
        publish_own(dot, w);
        if (!meet()) return;

        // ================= B: alpha, finish long and small rows, r -= alpha q =================
        {
            double s[2];
            col_sums(a.cta_part, NB, PS, 0, 0, 1, s);
            if (tid < CP) s_alpha[tid] = (s_active[tid] && s[0] > 0.0) ? s_rz[tid] / s[0] : 0.0;
            __syncthreads();
        }
        // entry (row, c) of r = ri, whose q is finished here; its share of r'z and r'r
        double rzp = 0.0, rrp = 0.0;  // column c_of_t
        auto finish = [&](int64_t row, int c, T ri, T dv, double qv) {
            const double al = s_alpha[c];
            if (al != 0.0) {
                ri = static_cast<T>(static_cast<double>(ri) - al * static_cast<double>(static_cast<T>(qv)));
                a.r[row * CP + c] = ri;
            }
            const double rd = static_cast<double>(ri);
            rzp = fma(rd, static_cast<double>(precond(dv, ri)), rzp);
            rrp = fma(rd, rd, rrp);
        };
        // long rows of at most kHugeChunks chunks: CP lanes each, lane c sums
        // column c of the row's chunk partials in chunk order
        {
            constexpr int RPW = 32 / CP;  // rows per warp
            const int64_t step = nwarps * RPW;
            int64_t li = wid * RPW + lane / CP;
            int4 m = li < a.nlong ? __ldg(a.long_meta + li) : make_int4(0, 0, 0, 0);
            for (; li < a.nlong; li += step) {
                const int4 cur = m;
                if (li + step < a.nlong) m = __ldg(a.long_meta + li + step);
                if (cur.z - cur.y > kHugeChunks) continue;
                const T ri = __ldcg(a.r + static_cast<int64_t>(cur.x) * CP + c_of_t);
                const T dv = __ldg(a.dinv + cur.x);
                double qv = 0.0;
                for (int32_t k = cur.y; k < cur.z; k += 8) {
                    double u[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        u[j] = k + j < cur.z ? __ldcg(a.lpart + static_cast<int64_t>(k + j) * CP + c_of_t) : 0.0;
#pragma unroll
                    for (int j = 0; j < 8; ++j) qv += u[j];
                }
                finish(cur.x, c_of_t, ri, dv, qv);
            }
        }
        // small rows b, b + NB, ... and huge long rows (dealt from the last CTA
        // down): the CTA sums the row's partials in a fixed order, thread
        // c < CP updates column c
        if (coupled) {
            for (int h = b, k = 0; h < SG; h += NB, ++k) {
                const int64_t row = a.Gf + h;
                const T ri = tid < CP ? __ldcg(a.r + row * CP + tid) : T(0);
                double s[2];
                col_sums(a.cta_part, NB, PS, CP + h * CP, 0, 1, s);
                if (tid < CP) finish(row, tid, ri, __ldg(a.dinv + row), s[0] + s_yq[k][tid]);
                __syncthreads();  // red_s is free again
            }
        }
        for (int64_t sI = NB - 1 - b; sI < a.nhuge; sI += NB) {
            const int4 m = __ldg(a.long_meta + __ldg(a.huge_li + sI));
            double s[2];
            col_sums(a.lpart + static_cast<int64_t>(m.y) * CP, m.z - m.y, CP, 0, 0, 1, s);
            if (tid < CP)
                finish(m.x, tid, __ldcg(a.r + static_cast<int64_t>(m.x) * CP + tid), __ldg(a.dinv + m.x), s[0]);
            __syncthreads();
        }
        // this CTA's short rows (contiguous range; long and small rows skipped)
        {
            double vb[2][4] = {}, wb[2];
            double al4[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) al4[i] = s_alpha[4 * tq + i];
            const bool any_al = al4[0] != 0.0 || al4[1] != 0.0 || al4[2] != 0.0 || al4[3] != 0.0;
            const int64_t e1 = min(r1, a.Gf) * CQ;
            for (int64_t e = r0 * CQ + tid; e < e1; e += 2 * NT) {
                const int64_t ev[2] = {e, e + NT};
                bool use[2];
                V4<T> rv[2], qv[2];
                T dv[2];
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    use[k] = ev[k] < e1;
                    if (use[k]) {
                        const int64_t row = ev[k] / CQ;
                        v4_load_cg(a.r + 4 * ev[k], rv[k]);
                        dv[k] = __ldg(a.dinv + row);
                        if (any_al) v4_load_cg(a.q + 4 * ev[k], qv[k]);
                        use[k] = __ldg(a.row_off + row + 1) - __ldg(a.row_off + row) <= kShortNnz;
                    }
                }
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    if (!use[k]) continue;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        double ri = static_cast<double>(rv[k].v[i]);
                        if (al4[i] != 0.0) {
                            ri -= al4[i] * static_cast<double>(qv[k].v[i]);
                            rv[k].v[i] = static_cast<T>(ri);
                            ri = static_cast<double>(rv[k].v[i]);
                        }
                        const T zi = precond(dv[k], rv[k].v[i]);
                        vb[0][i] = fma(ri, static_cast<double>(zi), vb[0][i]);
                        vb[1][i] = fma(ri, ri, vb[1][i]);
                    }
                    if (any_al) v4_store(a.r + 4 * ev[k], rv[k]);
                }
            }
            wb[0] = rzp;
            wb[1] = rrp;
            publish(vb, wb, off_rr, 2);
        }
        if (!meet()) return;

        // ================= C: beta, masks; x += alpha p, p = z + beta p =================
        {
            double s[2];
            col_sums(a.cta_part, NB, PS, off_rr[0], off_rr[1], 2, s);
            if (warp == 0) {
                int act = 0;
                if (lane < CP) {
                    s_beta[lane] = 0.0;
                    if (s_active[lane]) {
                        const double old = s_rz[lane];
                        s_beta[lane] = old > 0.0 ? s[0] / old : 0.0;
                        s_rz[lane] = s[0];
                        s_iters[lane] += 1;
                        act = ((s[1] > a.thr[lane]) && (s[0] > 0.0)) ? 1 : 0;
                        s_active[lane] = act;
                    }
                }
                const int any = __any_sync(kFull, act);
                if (lane == 0) s_any = any;
            }
            __syncthreads();
        }
        {
            // a column that just stopped keeps p (its x and r no longer move)
            bool act4[4];
            double be4[4], al4[4];
            bool work = false;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                act4[i] = s_active[4 * tq + i] != 0;
                be4[i] = s_beta[4 * tq + i];
                al4[i] = s_alpha[4 * tq + i];
                work = work || act4[i] || al4[i] != 0.0;
            }
            if (work) {
                const int64_t e1 = r1 * CQ;
                for (int64_t e = r0 * CQ + tid; e < e1; e += 2 * NT) {
                    const int64_t eb = e + NT;
                    const bool vb = eb < e1;
                    V4<T> rv[2], pv[2], xv[2];
                    T dv[2];
                    v4_load_cg(a.r + 4 * e, rv[0]);
                    v4_load_cg(a.p + 4 * e, pv[0]);
                    v4_load_cg(a.x + 4 * e, xv[0]);
                    dv[0] = __ldg(a.dinv + e / CQ);
                    if (vb) {
                        v4_load_cg(a.r + 4 * eb, rv[1]);
                        v4_load_cg(a.p + 4 * eb, pv[1]);
                        v4_load_cg(a.x + 4 * eb, xv[1]);
                        dv[1] = __ldg(a.dinv + eb / CQ);
                    }
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        if (k == 1 && !vb) break;
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const double pi = static_cast<double>(pv[k].v[i]);
                            if (al4[i] != 0.0)
                                xv[k].v[i] = static_cast<T>(static_cast<double>(xv[k].v[i]) + al4[i] * pi);
                            if (act4[i]) {
                                const T zi = precond(dv[k], rv[k].v[i]);
                                pv[k].v[i] = static_cast<T>(static_cast<double>(zi) + be4[i] * pi);
                            }
                        }
                        v4_store(a.x + 4 * (k ? eb : e), xv[k]);
                        v4_store(a.p + 4 * (k ? eb : e), pv[k]);
                    }
                }
            }
        }
        ++it;
        if (!CLUSTER) __syncthreads();  // every store of the CTA precedes the arrival
        if (!meet()) return;
    }
    if (b == 0 && tid < CP) {
        a.rz_out[tid] = s_rz[tid];
        a.iters_out[tid] = s_iters[tid];
        if (tid == 0) *a.loops_out = it;
    }
}

}  // namespace b200fe

namespace b200fe {

// Work lists of pcg_persistent_kernel over the CSR rows of S_ff.  Per row g:
// is_short[g] (<= kShortNnz nonzeros), is_long[g], its number of kLongChunk
// chunks, is_huge[g].
__global__ void pcg_lists_count_kernel(const int32_t* __restrict__ row_off, int32_t G,
                                       int32_t* __restrict__ is_short, int32_t* __restrict__ is_long,
                                       int32_t* __restrict__ nchunks, int32_t* __restrict__ is_huge) {
    for (int64_t g = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; g < G;
         g += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int32_t len = row_off[g + 1] - row_off[g];
        const bool sh = len <= kShortNnz;
        const int32_t nc = sh ? 0 : (len + kLongChunk - 1) / kLongChunk;
        is_short[g] = sh ? 1 : 0;
        is_long[g] = sh ? 0 : 1;
        nchunks[g] = nc;
        is_huge[g] = nc > kHugeChunks ? 1 : 0;
    }
}

// Fills the lists from the exclusive scans of the counts (short rows ascending).
__global__ void pcg_lists_fill_kernel(const int32_t* __restrict__ row_off, int32_t G,
                                      const int32_t* __restrict__ is_short,
                                      const int32_t* __restrict__ short_idx,
                                      const int32_t* __restrict__ long_idx,
                                      const int32_t* __restrict__ chunk_off, int32_t* __restrict__ short_row,
                                      int4* __restrict__ long_meta, int4* __restrict__ lchunk_meta,
                                      const int32_t* __restrict__ huge_idx, int32_t* __restrict__ huge_li) {
    for (int64_t g = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; g < G;
         g += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        if (is_short[g]) {
            short_row[short_idx[g]] = static_cast<int32_t>(g);
            continue;
        }
        const int32_t li = long_idx[g];
        const int32_t c0 = chunk_off[g], c1 = chunk_off[g + 1];
        long_meta[li] = make_int4(static_cast<int32_t>(g), c0, c1, 0);
        if (c1 - c0 > kHugeChunks) huge_li[huge_idx[g]] = li;
        const int32_t b = row_off[g], e = row_off[g + 1];
        for (int32_t c = c0; c < c1; ++c) {
            const int32_t cb = b + (c - c0) * kLongChunk;
            lchunk_meta[c] = make_int4(static_cast<int32_t>(g), cb, min(e, cb + kLongChunk), c == c0 ? 1 : 0);
        }
    }
}

// PcgTiles: tiles of kPcgRowsPerWarp short rows of about equal length, their
// nonzeros one row after the other, each tile from a multiple of four entries
// on (16-byte copies).  Rows are sorted by falling length within their
// summation list (lists > 0: steps of sr rows dealt to the lists) or all
// together; padded with row -1 to npad = a multiple of sr.
__global__ void pcg_tile_key_kernel(const int32_t* __restrict__ row_off, const int32_t* __restrict__ srow,
                                    int64_t nshort, int64_t npad, int sr, int lists, int32_t* __restrict__ key,
                                    int32_t* __restrict__ row) {
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < npad;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int32_t g = i < nshort ? srow[i] : -1;
        const int32_t len = g >= 0 ? row_off[g + 1] - row_off[g] : 0;
        const int32_t list = lists > 0 ? static_cast<int32_t>((i / sr) % lists) : 0;
        key[i] = list * (kShortNnz + 2) + (g >= 0 ? kShortNnz - len : kShortNnz + 1);
        row[i] = g;
    }
}
// len[t]: entries / 4 of tile t, rounded up
__global__ void pcg_tile_len_kernel(const int32_t* __restrict__ row_off, const int32_t* __restrict__ srow,
                                    int64_t ntiles, int32_t* __restrict__ len) {
    for (int64_t t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; t <= ntiles;
         t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        int32_t n = 0;
        for (int64_t k = t * kPcgRowsPerWarp; t < ntiles && k < (t + 1) * kPcgRowsPerWarp; ++k)
            if (srow[k] >= 0) n += row_off[srow[k] + 1] - row_off[srow[k]];
        len[t] = (n + 3) / 4;
    }
}
// One warp per tile: lanes take (row, every fourth nonzero).
template <typename T>
__global__ void pcg_tile_fill_kernel(const int32_t* __restrict__ row_off, const int32_t* __restrict__ col,
                                     const double* __restrict__ val, const int32_t* __restrict__ srow,
                                     int64_t ntiles, const int32_t* __restrict__ off,
                                     int2* __restrict__ meta, int2* __restrict__ rows,
                                     int32_t* __restrict__ tcol, T* __restrict__ tval) {
    constexpr int RW = kPcgRowsPerWarp;
    const int lane = threadIdx.x & 31, r = lane % RW;
    const int64_t nw = static_cast<int64_t>(gridDim.x) * (blockDim.x / 32);
    for (int64_t t = static_cast<int64_t>(blockIdx.x) * (blockDim.x / 32) + threadIdx.x / 32; t < ntiles; t += nw) {
        const int64_t k = t * RW + r;
        const int32_t g = srow[k];
        const int32_t b = g >= 0 ? row_off[g] : 0;
        const int32_t n = g >= 0 ? row_off[g + 1] - b : 0;
        int32_t e0 = 0, total = 0;
        for (int i = 0; i < RW; ++i) {
            const int32_t ni = __shfl_sync(0xffffffffu, n, i);
            if (i < r) e0 += ni;
            total += ni;
        }
        const int32_t o = off[t];
        if (lane < RW) rows[k] = make_int2(g, e0 | (n << 16));
        if (lane == 0) meta[t] = make_int2(o, total);
        const int64_t d = 4 * static_cast<int64_t>(o) + e0;
        for (int j = lane / RW; j < n; j += 32 / RW) {
            tcol[d + j] = col[b + j];
            tval[d + j] = static_cast<T>(val[b + j]);
        }
    }
}

}  // namespace b200fe
