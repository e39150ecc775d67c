// el_solve.cu -- conjugate-gradient pressure solves on the grid-shaped ghost-fluid matrix.
//
// Replaces the Eigen ConjugateGradient<..., Lower, IncompleteCholesky<double>> call of
// src/project/3d/eulerian_liquid/simulator.cpp:102-109 (x0 = 0, stop on |r|^2 < tol^2 |b|^2 of
// the recursively updated residual, iteration cap) with three GPU solvers:
//
//   EL_SOLVER_JACOBI_FP64  plain FP64 PCG, Jacobi preconditioner (the correctness baseline;
//                          jacobi_dir_kernel / jacobi_update_kernel)
//   EL_SOLVER_MG_FP64      FP64 PCG with a multigrid V-cycle preconditioner
//   EL_SOLVER_MIXED        FP64 iterative refinement: r = b - A x in FP64, the correction
//                          solved by FP32 multigrid PCG on the FP32 operator, x += |r| e in FP64
//
// Work distribution: every level keeps an ordered list of its active row segments (32 cells
// of one (j, k) row holding at least one cell with a positive diagonal).  Kernels run one
// warp per listed segment with a fixed grid, so cells that are air or solid cost nothing,
// all loads of a cell are issued before any is used, and the partial sums of the dot
// products are formed in a fixed order (deterministic).  Vector entries outside the active
// segments are never written; they stay finite and always meet a zero coupling.
//
// Operators are stored as per-cell records {diagonal, coupling with +x, +y, +z}: float4 for
// the FP32 PCG operator, Rec64 for the FP64 multigrid, and half4 for the level-0 operator the
// FP32 multigrid smooths with (diagonal rounded up, couplings rounded towards zero, so the
// record operator stays diagonally dominant, hence SPD).
//
// Multigrid: coarse operators by aggregation of 2x2x2 blocks scaled by 1/2
// (A_c = 1/2 P^T A P, piecewise-constant P; it reproduces the rediscretised Laplacian for
// constant coefficients and carries the ghost-fluid Dirichlet terms down by summation),
// restriction R = P^T, two Jacobi sweeps before and two after with Chebyshev weights (see
// kSweep1 / kSweep2), and 30 damped-Jacobi sweeps on the coarsest level (at most 8 cells per
// axis) in one block's shared memory.  The same polynomial smoother on both legs and R = P^T
// make the V-cycle symmetric, as PCG needs.
//
// Per PCG iteration:  K1  p = z + beta p ; Ap = A p ; alpha = rz / p.Ap
//                     K2  x += alpha p ; r -= alpha Ap ; rr = r.r (; z = D^-1 r, rz = r.z for Jacobi)
//                     V   z = M^-1 r ; rz = r.z ; beta            (multigrid solvers)
// Scalars live in device memory; once converged the remaining launched kernels return at
// entry, so the host polls only every `check_every` iterations.
#include <cuda_fp16.h>

#include <climits>
#include <type_traits>

#include "el_df.cuh"
#include "el_internal.cuh"

namespace el {

// Damped Jacobi on the coarsest level (a solve): the damping that balances the 3-D 7-point
// Laplacian's high-frequency error reduction.
constexpr double kOmega = 6.0 / 7.0;
// The smoother's sweep weights kSweep1 / kSweep2 are defined in el_internal.cuh.
constexpr int kCoarsestSweeps = 30;
constexpr int kCoarsestMaxDim = 8;
constexpr int kCoarsestMaxCells = 512;
constexpr int kSegThreads = 256;
// Block size of the PCG kernels that end in a dot product: few, large blocks, because each block's
// reduction occupies the FP64 pipe (block_sum) -- one block an SM in FP64.
template <typename V>
constexpr int kDotThreads = sizeof(V) == 8 ? 1024 : 512;

__device__ __forceinline__ bool finite_d(double v) { return isfinite(v); }

__device__ __forceinline__ bool positive(float v) { return v > 0.f; }
__device__ __forceinline__ bool positive(double v) { return d_positive(v); }  // on the integer pipe

// The reciprocal of a row's diagonal, 0 on an empty row.  A diagonal below 2^-1000 takes that scale
// instead: its reciprocal could overflow, and a smaller one only leaves that row to the Krylov method.
__device__ __forceinline__ double row_inverse(double d) { return positive(d) ? 1.0 / fmax(d, 0x1p-1000) : 0.0; }

// ---------------------------------------------------------------------------------------
// coefficient records

template <typename V>
struct Co {
    V d, x, y, z;
};

__device__ __forceinline__ Co<float> ldrec(const float4* r, long long c) {
    const float4 v = __ldg(r + c);
    return {v.x, v.y, v.z, v.w};
}
__device__ __forceinline__ Co<float> ldrec(const ushort4* r, long long c) {
    const ushort4 v = __ldg(r + c);
    return {__half2float(__ushort_as_half(v.x)), __half2float(__ushort_as_half(v.y)),
            __half2float(__ushort_as_half(v.z)), __half2float(__ushort_as_half(v.w))};
}
__device__ __forceinline__ Co<double> ldrec(const Rec64* r, long long c) {
    const double2* p = reinterpret_cast<const double2*>(r + c);
    const double2 a = __ldg(p), b = __ldg(p + 1);
    return {a.x, a.y, b.x, b.y};
}

// The FP64 operator of the context: diag64 plus three coupling arrays of the field type.
template <typename OT>
struct SplitOp {
    const double* __restrict__ d;
    const OT* __restrict__ x;
    const OT* __restrict__ y;
    const OT* __restrict__ z;
};

// ---------------------------------------------------------------------------------------
// segment geometry

struct LGeom {
    int n0, n1, n2, nsr;
    int s1, s2;  // strides of j and k (every grid holds fewer than 2^31 cells)
};

inline LGeom make_geom(int n0, int n1, int n2) {
    return LGeom{n0, n1, n2, (n0 + 31) / 32, n0, n0 * n1};
}

__device__ __forceinline__ void seg_cell(int id, const LGeom& g, int lane, int& i, int& j, int& k) {
    const int row = id / g.nsr;
    i = (id - row * g.nsr) * 32 + lane;
    j = row % g.n1;
    k = row / g.n1;
}

struct SegArg {
    const int4* __restrict__ desc;  // {first cell index, i0, j, k}
    const int* __restrict__ count;
};

// Walks the active segments, one warp per segment; defines lane, i, j, k, c (cell index, int:
// every grid holds fewer than 2^31 cells) and live (i < n0).  Lanes past the row end stay in
// the loop (live = false) so that warp shuffles see all 32 lanes.
#define SEG_LOOP_ALL_BEGIN(seg, g)                                                \
    const int lane = threadIdx.x & 31;                                            \
    const int warp_global = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;         \
    const int nwarps = (gridDim.x * blockDim.x) >> 5;                             \
    const int nseg = *(seg).count;                                                \
    for (int qs = warp_global; qs < nseg; qs += nwarps) {                         \
        const int4 sd = (seg).desc[qs];                                           \
        const int i = sd.y + lane, j = sd.z, k = sd.w;                            \
        const int c = sd.x + lane;                                                \
        const bool live = i < (g).n0;

// the same, with the next segment's descriptor loaded while the current one is processed (for
// the kernels whose registers leave room for it)
#define SEG_LOOP_ALL_PF_BEGIN(seg, g)                                             \
    const int lane = threadIdx.x & 31;                                            \
    const int warp_global = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;         \
    const int nwarps = (gridDim.x * blockDim.x) >> 5;                             \
    const int nseg = *(seg).count;                                                \
    int4 sd_next = warp_global < nseg ? (seg).desc[warp_global] : make_int4(0, 0, 0, 0); \
    for (int qs = warp_global; qs < nseg; qs += nwarps) {                         \
        const int4 sd = sd_next;                                                  \
        if (qs + nwarps < nseg) sd_next = (seg).desc[qs + nwarps];                \
        const int i = sd.y + lane, j = sd.z, k = sd.w;                            \
        const int c = sd.x + lane;                                                \
        const bool live = i < (g).n0;

#define SEG_LOOP_BEGIN(seg, g) \
    SEG_LOOP_ALL_PF_BEGIN(seg, g) \
    if (!live) continue;

#define SEG_LOOP_END }

constexpr unsigned kFull = 0xffffffffu;

// ---------------------------------------------------------------------------------------
// segment lists: per-segment activity flag (seg_flags_diag_kernel, coarsen_kernel), then an ordered
// compaction.  Each launch costs two to three microseconds whatever its size, so a list of up to
// kSegDirect segments is one: a block of seg_write_kernel adds up the flags before its own; a longer one
// has its chunks counted first.  Flags, counts, a scan of the counts and the list in four launches a
// level took 11 us a level, five levels and more a solve; coarse levels now take one launch, the finest
// two or three (75 x 62 x 53: 0.90 -> 0.87 ms a solve, 151 x 97 x 133 1.61 -> 1.56).

constexpr int kSegChunk = 1024;
constexpr long long kSegDirect = 16 * kSegChunk;

__global__ void seg_flags_diag_kernel(LGeom g, const double* __restrict__ diag, long long total,
                                      uint8_t* __restrict__ flags) {
    // a warp per row (j, k): one index division a row, not one a segment, and up to eight of
    // the row's segments in flight together; segment id = row * nsr + segment of the row
    (void)total;
    const int lane = threadIdx.x & 31;
    const long long w0 = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
    const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
    const long long nrows = (long long)g.n1 * g.n2;
    constexpr int U = 8;
    for (long long row = w0; row < nrows; row += nw) {
        const int j = (int)(row % g.n1), k = (int)(row / g.n1);
        const double* drow = diag + (long long)g.s1 * j + (long long)g.s2 * k;
        for (int s0 = 0; s0 < g.nsr; s0 += U) {
            bool act[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int i = (s0 + u) * 32 + lane;
                act[u] = s0 + u < g.nsr && i < g.n0 && d_positive(drow[i]);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const unsigned m = __ballot_sync(0xffffffffu, act[u]);
                if (lane == 0 && s0 + u < g.nsr) flags[row * g.nsr + s0 + u] = m ? 1 : 0;
            }
        }
    }
}

__global__ void seg_count_kernel(const uint8_t* __restrict__ flags, long long total, int* __restrict__ chunk) {
    __shared__ int sh[8];
    pdl_wait();
    pdl_trigger();
    const long long base = (long long)blockIdx.x * kSegChunk;
    int cnt = 0;
    for (int q = threadIdx.x; q < kSegChunk; q += blockDim.x) {
        const long long id = base + q;
        if (id < total && flags[id]) ++cnt;
    }
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_down_sync(0xffffffffu, cnt, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = cnt;
    __syncthreads();
    if (threadIdx.x == 0) {
        int t = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += sh[w];
        chunk[blockIdx.x] = t;
    }
}

// The descriptors of a chunk's active segments, in order: each warp of the block takes an equal
// run of the chunk's flags, counts its active ones, and writes them after the counts of the
// warps before it and of the chunks before this one (chunk: their counts; null: from the flags).
// The last block leaves the list's length.
__global__ void seg_write_kernel(LGeom g, const uint8_t* __restrict__ flags, long long total,
                                 const int* __restrict__ chunk, int4* __restrict__ desc, int* __restrict__ count) {
    __shared__ int wcount[32], before[32];
    pdl_wait();
    pdl_trigger();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int span = kSegChunk / nw;
    const long long wb = (long long)blockIdx.x * kSegChunk + (long long)w * span;
    int pre = 0, cnt = 0;
    if (chunk) {
        for (int q = threadIdx.x; q < (int)blockIdx.x; q += blockDim.x) pre += chunk[q];
    } else {
        const uint4* f4 = reinterpret_cast<const uint4*>(flags);
        for (int q = threadIdx.x; q < (int)blockIdx.x * (kSegChunk / 16); q += blockDim.x) {
            const uint4 f = f4[q];  // sixteen flags, each 0 or 1
            pre += __popc(f.x) + __popc(f.y) + __popc(f.z) + __popc(f.w);
        }
    }
    for (int q = 0; q < span; q += 32) {
        const long long id = wb + q + lane;
        cnt += __popc(__ballot_sync(kFull, id < total && flags[id]));
    }
    for (int o = 16; o > 0; o >>= 1) pre += __shfl_down_sync(kFull, pre, o);
    if (lane == 0) {
        wcount[w] = cnt;
        before[w] = pre;
    }
    __syncthreads();
    int run = 0;
    for (int v = 0; v < nw; ++v) run += before[v];
    if (threadIdx.x == 0 && blockIdx.x == gridDim.x - 1) {
        int all = run;
        for (int v = 0; v < nw; ++v) all += wcount[v];
        *count = all;
    }
    for (int v = 0; v < w; ++v) run += wcount[v];
    for (int q = 0; q < span; q += 32) {
        const long long id = wb + q + lane;
        const bool f = id < total && flags[id];
        const unsigned m = __ballot_sync(kFull, f);
        if (f) {
            int i0, j, k;
            seg_cell((int)id, g, 0, i0, j, k);
            desc[run + __popc(m & ((1u << lane) - 1u))] = make_int4((int)(i0 + g.s1 * j + g.s2 * k), i0, j, k);
        }
        run += __popc(m);
    }
}

// ---------------------------------------------------------------------------------------
// operator packing (once per solve)

// float4 PCG records and half4 multigrid records of the FP32 inner system.
template <typename OT>
__global__ void pack32_kernel(long long n, const double* __restrict__ d, const OT* __restrict__ ox,
                              const OT* __restrict__ oy, const OT* __restrict__ oz, float4* __restrict__ a32,
                              ushort4* __restrict__ a16) {
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x) {
        const float4 r = make_float4((float)d[c], (float)ox[c], (float)oy[c], (float)oz[c]);
        a32[c] = r;
        // diagonal rounded up, (non-positive) couplings rounded towards zero: the half record
        // operator keeps diag >= sum |couplings| row by row
        a16[c] = make_ushort4(__half_as_ushort(__float2half_ru(r.x)), __half_as_ushort(__float2half_rz(r.y)),
                              __half_as_ushort(__float2half_rz(r.z)), __half_as_ushort(__float2half_rz(r.w)));
    }
}

template <typename OT>
__global__ void pack64_kernel(long long n, const double* __restrict__ d, const OT* __restrict__ ox,
                              const OT* __restrict__ oy, const OT* __restrict__ oz, Rec64* __restrict__ a,
                              double* __restrict__ rd) {
    for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < n; c += (long long)gridDim.x * blockDim.x) {
        const double dc = d[c];
        a[c] = Rec64{dc, (double)ox[c], (double)oy[c], (double)oz[c]};
        rd[c] = row_inverse(dc);
    }
}

// Coarse records A_c = 1/2 P^T A P over 2x2x2 blocks.  The FP32 hierarchy (float4 coarse
// records, built from half4 or float4 records) sums in FP32 -- the eight children's values
// carry at most 24 significant bits, and FP64 arithmetic runs at a small fraction of the FP32
// rate on this GPU -- the FP64 hierarchy in FP64.  A warp's 32 coarse cells are a row segment, whose
// activity flag it writes.
template <typename RF, typename RC>
__global__ void coarsen_kernel(LGeom F, const RF* __restrict__ fr, LGeom C, RC* __restrict__ cr,
                               double* __restrict__ rd, uint8_t* __restrict__ flags) {
    pdl_wait();
    pdl_trigger();
    using A = typename std::conditional<sizeof(RC) == sizeof(float4), float, double>::type;
    const int I = blockIdx.x * blockDim.x + threadIdx.x;
    const int J = blockIdx.y * blockDim.y + threadIdx.y;
    const int K = blockIdx.z;
    if (J >= C.n1) return;  // a warp is a row's segment
    A d = 0, sx = 0, sy = 0, sz = 0, inner = 0;
    for (int kk = 0; kk < 2; ++kk)
        for (int jj = 0; jj < 2; ++jj)
            for (int ii = 0; ii < 2; ++ii) {
                const int i = 2 * I + ii, j = 2 * J + jj, k = 2 * K + kk;
                if (i >= F.n0 || j >= F.n1 || k >= F.n2) continue;
                const auto r = ldrec(fr, i + F.s1 * j + F.s2 * k);
                d += r.d;
                if (ii == 0) inner += r.x; else sx += r.x;
                if (jj == 0) inner += r.y; else sy += r.y;
                if (kk == 0) inner += r.z; else sz += r.z;
            }
    A dc = A(0.5) * (d + A(2) * inner);
    // an aggregate coupled to nothing outside it (an enclosed Neumann pocket) has a zero row
    // sum; its diagonal is raised to half the children's, which keeps the operator SPD
    if (d > A(0) && !(dc > A(1e-6) * d)) dc = A(0.5) * d;
    const unsigned active = __ballot_sync(kFull, I < C.n0 && dc > A(0));
    if (threadIdx.x == 0) flags[((long long)K * C.n1 + J) * C.nsr + blockIdx.x] = active ? 1 : 0;
    if (I >= C.n0) return;
    const long long q = I + C.s1 * J + C.s2 * K;
    if constexpr (sizeof(RC) == sizeof(float4))
        cr[q] = make_float4(dc, A(0.5) * sx, A(0.5) * sy, A(0.5) * sz);
    else {
        cr[q] = Rec64{dc, 0.5 * sx, 0.5 * sy, 0.5 * sz};
        rd[q] = row_inverse(dc);
    }
}

// ---------------------------------------------------------------------------------------
// The 7-point stencil around each lane's cell.  recf(q) loads a cell's record (diagonal and
// +x/+y/+z couplings), rawf(q, qi, qj, qk) loads the vector data of a cell and valf(raw, rec)
// turns it into the value the stencil applies to.  Every load of the stencil (including the
// cells just outside the segment, fetched by lanes 0 and 31) is issued before any value is
// formed, so a lane waits for memory once; the i-neighbours of the other lanes come by shuffle.
// ALL: every neighbour's record is needed (for its diagonal); else only those carrying a
// coupling (-x, -y, -z) are loaded.  Must be called by all 32 lanes.
// Per-thread partial sums of a dot product: FP32 for the FP32 solver (a thread sums a few
// dozen products; FP64 arithmetic runs at a small fraction of the FP32 rate on this GPU), FP64
// otherwise; the grid reduction is FP64 either way.
template <typename V>
using DotAcc = typename std::conditional<sizeof(V) == 4, float, double>::type;

template <typename V>
struct St7 {
    V v0, vxm, vxp, vym, vyp, vzm, vzp;  // values at the centre and the six neighbours
    V d, cxm, cxp, cym, cyp, czm, czp;   // diagonal and couplings
};

// which of the stencil's cells exist, and the cell just outside the segment (of lane 0 or of lane
// 31: one load and one value serve both)
struct Near7 {
    bool iym, iyp, izm, izp, ixm, ixp, xp_in;
    int ce, ie;
};

__device__ __forceinline__ Near7 near7(const LGeom& g, int c, int i, int j, int k, bool live, int lane) {
    Near7 n;
    n.iym = live && j > 0;
    n.iyp = live && j < g.n1 - 1;
    n.izm = live && k > 0;
    n.izp = live && k < g.n2 - 1;
    n.ixm = lane == 0 && live && i > 0;
    n.xp_in = live && i + 1 < g.n0;
    n.ixp = lane == 31 && n.xp_in;
    n.ce = n.ixm ? c - 1 : c + 1;
    n.ie = n.ixm ? i - 1 : i + 1;
    return n;
}

template <typename V>
struct Rec7 {
    Co<V> r0, ym, yp, zm, zp, xe;
};

template <typename V, bool ALL, typename RF>
__device__ __forceinline__ Rec7<V> load_rec7(const LGeom& g, const Near7& n, int c, bool live, RF&& recf) {
    const Co<V> z4{V(0), V(0), V(0), V(0)};
    Rec7<V> r;
    r.r0 = live ? recf(c) : z4;
    r.ym = n.iym ? recf(c - g.s1) : z4;
    r.yp = (ALL && n.iyp) ? recf(c + g.s1) : z4;
    r.zm = n.izm ? recf(c - g.s2) : z4;
    r.zp = (ALL && n.izp) ? recf(c + g.s2) : z4;
    r.xe = (n.ixm || (ALL && n.ixp)) ? recf(n.ce) : z4;
    return r;
}

template <typename Raw>
struct Raw7 {
    Raw a0, ym, yp, zm, zp, xe;
};

template <typename LF>
__device__ __forceinline__ auto load_raw7(const LGeom& g, const Near7& n, int c, int i, int j, int k, bool live,
                                          LF&& rawf) {
    using Raw = decltype(rawf(0, 0, 0, 0));
    Raw7<Raw> a;
    a.a0 = live ? rawf(c, i, j, k) : Raw{};
    a.ym = n.iym ? rawf(c - g.s1, i, j - 1, k) : Raw{};
    a.yp = n.iyp ? rawf(c + g.s1, i, j + 1, k) : Raw{};
    a.zm = n.izm ? rawf(c - g.s2, i, j, k - 1) : Raw{};
    a.zp = n.izp ? rawf(c + g.s2, i, j, k + 1) : Raw{};
    a.xe = (n.ixm || n.ixp) ? rawf(n.ce, n.ie, j, k) : Raw{};
    return a;
}

template <typename V, typename Raw, typename VF>
__device__ __forceinline__ St7<V> value7(const Near7& n, const Rec7<V>& r, const Raw7<Raw>& a, bool live, int lane,
                                         VF&& valf) {
    St7<V> st;
    st.d = r.r0.d;
    st.cxp = r.r0.x;
    st.cyp = r.r0.y;
    st.czp = r.r0.z;
    st.cym = r.ym.y;
    st.czm = r.zm.z;
    st.v0 = live ? valf(a.a0, r.r0) : V(0);
    st.vym = n.iym ? valf(a.ym, r.ym) : V(0);
    st.vyp = n.iyp ? valf(a.yp, r.yp) : V(0);
    st.vzm = n.izm ? valf(a.zm, r.zm) : V(0);
    st.vzp = n.izp ? valf(a.zp, r.zp) : V(0);
    const V sxm = __shfl_up_sync(kFull, st.v0, 1);
    const V sxp = __shfl_down_sync(kFull, st.v0, 1);
    const V scm = __shfl_up_sync(kFull, r.r0.x, 1);
    const V vxe = (n.ixm || n.ixp) ? valf(a.xe, r.xe) : V(0);
    st.vxm = lane == 0 ? vxe : sxm;
    st.cxm = lane == 0 ? r.xe.x : scm;
    st.vxp = n.xp_in ? (lane == 31 ? vxe : sxp) : V(0);
    return st;
}

template <typename V, bool ALL, typename RF, typename LF, typename VF>
__device__ __forceinline__ St7<V> gather7(const LGeom& g, int c, int i, int j, int k, bool live, int lane, RF&& recf,
                                          LF&& rawf, VF&& valf) {
    const Near7 n = near7(g, c, i, j, k, live, lane);
    const Rec7<V> r = load_rec7<V, ALL>(g, n, c, live, recf);
    const auto a = load_raw7(g, n, c, i, j, k, live, rawf);
    return value7<V>(n, r, a, live, lane, valf);
}

template <typename V>
__device__ __forceinline__ V apply7(const St7<V>& st) {
    return stencil7(st.d, st.v0, st.cxm, st.vxm, st.cxp, st.vxp, st.cym, st.vym, st.cyp, st.vyp, st.czm, st.vzm,
                    st.czp, st.vzp);
}

template <typename V, typename R>
struct RecLoad {
    const R* __restrict__ a;
    __device__ __forceinline__ Co<V> operator()(int q) const {
        const auto r = ldrec(a, q);
        return Co<V>{(V)r.d, (V)r.x, (V)r.y, (V)r.z};
    }
};

template <typename OT>
struct SplitLoad {
    SplitOp<OT> a;
    __device__ __forceinline__ Co<double> operator()(int q) const {
        return Co<double>{a.d[q], f2d(a.x[q]), f2d(a.y[q]), f2d(a.z[q])};
    }
};


// K1: new direction fused with A p and p.Ap over the active segments (record operator: FP32 inner
// system, FP64 multigrid).
template <typename V, typename R>
__global__ void __launch_bounds__(kDotThreads<V>) dir_spmv_rec_kernel(LGeom g, SegArg seg, const R* __restrict__ A,
                                                                      const V* __restrict__ z,
                                                                      const V* __restrict__ p_in,
                                                                      V* __restrict__ p_out, V* __restrict__ ap,
                                                                      Scalars* s, int first, double* partials,
                                                                      unsigned* counter) {
    const RecLoad<V, R> recf{A};
    const int lane = threadIdx.x & 31;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    int qs = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nseg = *seg.count;
    int4 sd = qs < nseg ? seg.desc[qs] : make_int4(0, g.n0, 0, 0);
    Near7 nb = near7(g, sd.x + lane, sd.y + lane, sd.z, sd.w, sd.y + lane < g.n0, lane);
    Rec7<V> rec = load_rec7<V, false>(g, nb, sd.x + lane, sd.y + lane < g.n0, recf);
    pdl_wait();
    pdl_trigger();
    if (s->done) return;
    const V beta = first ? V(0) : (V)s->beta;
    DotAcc<V> part = 0;
    auto rawf = [&](int q, int, int, int) -> V { return first ? z[q] : z[q] + beta * p_in[q]; };
    auto valf = [](V raw, const Co<V>&) -> V { return raw; };
    while (qs < nseg) {
        const bool live = sd.y + lane < g.n0;
        const int c = sd.x + lane;
        const auto raw = load_raw7(g, nb, c, 0, 0, 0, live, rawf);
        const St7<V> st = value7<V>(nb, rec, raw, live, lane, valf);
        qs += nwarps;
        if (qs < nseg) sd = seg.desc[qs];
        if (live) {
            V pc = V(0), apc = V(0);
            if (positive(st.d)) {
                pc = st.v0;
                apc = apply7(st);
            }
            p_out[c] = pc;
            ap[c] = apc;
            part += (DotAcc<V>)pc * (DotAcc<V>)apc;
        }
        if (qs >= nseg) break;
        nb = near7(g, sd.x + lane, sd.y + lane, sd.z, sd.w, sd.y + lane < g.n0, lane);
        rec = load_rec7<V, false>(g, nb, sd.x + lane, sd.y + lane < g.n0, recf);
    }
    double acc[1] = {(double)part};
    double tot[1];
    if (grid_sum<1, kDotThreads<V>>(acc, partials, counter, tot)) {
        const double alpha = s->rz / tot[0];
        s->alpha = alpha;
        if (!finite_d(alpha)) {
            s->bad = 1;
            s->done = 1;
        }
    }
}

// the end of an update: |r|^2 from the threads' shares, and whether it is small enough
template <typename V>
__device__ __forceinline__ void update_done(DotAcc<V> part, Scalars* s, double* partials, unsigned* counter) {
    double acc[1] = {(double)part};
    double tot[1];
    if (grid_sum<1, kDotThreads<V>>(acc, partials, counter, tot)) {
        s->rr = tot[0];
        const int iter = s->iter + 1;
        s->iter = iter;
        if (!finite_d(tot[0])) {
            s->bad = 1;
            s->done = 1;
        } else if (tot[0] < s->thresh || iter >= s->iter_limit) {
            s->done = 1;
        }
    }
}

// K2: x += alpha p ; r -= alpha Ap ; |r|^2; FP64 also t = the V-cycle's first sweep from zero.
template <typename V>
__global__ void __launch_bounds__(kDotThreads<V>) update_kernel(LGeom g, SegArg seg, V* __restrict__ x,
                                                                V* __restrict__ r, const V* __restrict__ p,
                                                                const V* __restrict__ ap, V* __restrict__ t,
                                                                const V* __restrict__ rd, Scalars* s,
                                                                double* partials, unsigned* counter) {
    // two segments per warp and iteration, all eight loads issued before any use: the kernel is
    // pure streaming and bound by the loads in flight
    const int lane = threadIdx.x & 31;
    const int warp_global = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    const int nseg = *seg.count;
    const int qe = warp_global + nwarps;
    int4 sa = warp_global < nseg ? seg.desc[warp_global] : make_int4(0, 0, 0, 0);
    int4 sb = qe < nseg ? seg.desc[qe] : sa;
    pdl_wait();
    pdl_trigger();
    if (s->done) return;
    const V alpha = (V)s->alpha;
    DotAcc<V> part = 0;
    auto finish = [&](int c, V pc, V apc, V xc, V rc0) {
        const V rc = rc0 - alpha * apc;
        x[c] = xc + alpha * pc;
        r[c] = rc;
        if (sizeof(V) == 8) t[c] = rn_mul(rn_mul(V(kSweep1), rc), rd[c]);
        part += (DotAcc<V>)rc * (DotAcc<V>)rc;
    };
    for (int qs = warp_global; qs < nseg; qs += 2 * nwarps) {
        const int q2 = qs + nwarps;
        if (qs != warp_global) {
            sa = seg.desc[qs];
            sb = q2 < nseg ? seg.desc[q2] : sa;
        }
        const bool la = sa.y + lane < g.n0, lb = q2 < nseg && sb.y + lane < g.n0;
        const int ca = sa.x + lane, cb = sb.x + lane;
        V pa = V(0), apa = V(0), xa = V(0), ra = V(0), pb = V(0), apb = V(0), xb = V(0), rb = V(0);
        if (la) {
            pa = p[ca];
            apa = ap[ca];
            xa = x[ca];
            ra = r[ca];
        }
        if (lb) {
            pb = p[cb];
            apb = ap[cb];
            xb = x[cb];
            rb = r[cb];
        }
        if (la) finish(ca, pa, apa, xa, ra);
        if (lb) finish(cb, pb, apb, xb, rb);
    }
    update_done<V>(part, s, partials, counter);
}

// ---------------------------------------------------------------------------------------
// Plain FP64 PCG with the Jacobi preconditioner: two kernels an iteration.
//
// Bound by the FP64 pipe (2 lanes a clock per SM; a division costs nine of its operations) on a
// large scene, by the chain of latencies on a small one.  So
//   - the update stores z = D^-1 r, formed with reciprocals of the diagonal taken once a solve, and
//     the direction reads z: 14 FP64 operations a cell in K1 where r / d at every point of the
//     stencil took about 80, 5 in K2;
//   - a kernel leaves its dot products as one partial sum a block, and the next kernel's blocks
//     each sum those (at most one block an SM) while their own loads are in flight: no fence, ticket
//     and last block at the end of a launch;
//   - what no kernel of the iteration writes (segments, coefficients) is loaded before the wait for
//     the kernel before.
// Dam break, FP64, both kernels of an iteration: 128^3 115.6 -> 32.1 us, 64^3 38.6 -> 13.9 us.
//
// rz of iteration t (0, 1, ...) lives in rz2[t & 1]: K1's blocks read the old one while block 0
// stores the new one.
constexpr int kJacThreads = 512;
constexpr int kJacMaxBlocks = 256;  // at most one block an SM

struct JacPart {
    double* pap;  // [blocks]      p.Ap   (K1)
    double* rr;   // [blocks][2]   r.r, r.z   (K2)
    int blocks;
};

// The totals of NV values over the blocks' partials, in every thread (a barrier): warp q sums
// value q, in the same order in every block.
template <int NV>
__device__ __forceinline__ void sum_partials(const double* __restrict__ part, int blocks, double (&out)[NV]) {
    __shared__ double tot[NV];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < NV) {
        double t[kJacMaxBlocks / 32];
#pragma unroll
        for (int m = 0; m < kJacMaxBlocks / 32; ++m) {
            const int b = lane + 32 * m;
            t[m] = b < blocks ? __ldcg(part + (size_t)b * NV + warp) : 0.0;
        }
        double v = t[0];
#pragma unroll
        for (int m = 1; m < kJacMaxBlocks / 32; ++m)
            if (32 * m < blocks) v += t[m];
        v = warp_sum(v);
        if (lane == 0) tot[warp] = v;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NV; ++q) out[q] = tot[q];
}

// |r|^2 and r.z after an update: the stopping test, and beta for the next direction
struct JacNext {
    double rr, rz, beta;
    bool bad, done;
};
__device__ __forceinline__ JacNext jacobi_next(const double (&t)[2], double rz_old, double thresh) {
    JacNext n;
    n.rr = t[0];
    n.rz = t[1];
    n.beta = t[1] / rz_old;
    n.bad = !finite_d(t[0]);
    n.done = n.bad || t[0] < thresh;
    return n;
}
__device__ __forceinline__ void jacobi_store(Scalars* s, const JacNext& n, int slot_new) {
    s->rr = n.rr;
    s->iter += 1;
    s->beta = n.beta;
    s->rz2[slot_new] = n.rz;
    if (n.bad) s->bad = 1;
    if (n.done) s->done = 1;
}

// K1 of iteration t (slot = t & 1).  pending: the update before left its dot products as partials
// (else s->beta holds the result).
template <typename OT>
__global__ void __launch_bounds__(kJacThreads, 1) jacobi_dir_kernel(LGeom g, SegArg seg, SplitOp<OT> A,
                                                                    const double* __restrict__ z,
                                                                    const double* __restrict__ p_in,
                                                                    double* __restrict__ p_out,
                                                                    double* __restrict__ ap, Scalars* s, int first,
                                                                    int pending, int slot, JacPart part) {
    __shared__ SumScratch<1, kJacThreads> sh;
    const SplitLoad<OT> recf{A};
    const int lane = threadIdx.x & 31;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    int qs = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nseg = *seg.count;
    int4 sd = qs < nseg ? seg.desc[qs] : make_int4(0, g.n0, 0, 0);
    Near7 nb = near7(g, sd.x + lane, sd.y + lane, sd.z, sd.w, sd.y + lane < g.n0, lane);
    Rec7<double> rec = load_rec7<double, false>(g, nb, sd.x + lane, sd.y + lane < g.n0, recf);
    pdl_wait();
    pdl_trigger();
    auto rawf = [&](int q, int, int, int) -> double2 { return make_double2(z[q], first ? 0.0 : p_in[q]); };
    auto raw = load_raw7(g, nb, sd.x + lane, 0, 0, 0, sd.y + lane < g.n0, rawf);
    const int done = s->done;
    double beta = first ? 0.0 : s->beta;
    if (pending) {
        const double rz_old = s->rz2[slot ^ 1], thresh = s->thresh;
        double t[2];
        sum_partials(part.rr, part.blocks, t);
        if (done) return;
        const JacNext n = jacobi_next(t, rz_old, thresh);
        if (blockIdx.x == 0 && threadIdx.x == 0) jacobi_store(s, n, slot);
        if (n.done) return;
        beta = n.beta;
    } else if (done) {
        return;
    }
    auto valf = [&](double2 v, const Co<double>&) -> double { return first ? v.x : v.x + beta * v.y; };
    double acc[1] = {0.0};
    while (true) {
        const bool live = sd.y + lane < g.n0;
        const int c = sd.x + lane;
        const St7<double> st = value7<double>(nb, rec, raw, live, lane, valf);
        if (live) {
            double pc = 0.0, apc = 0.0;
            if (positive(st.d)) {
                pc = st.v0;
                apc = apply7(st);
            }
            p_out[c] = pc;
            ap[c] = apc;
            acc[0] += pc * apc;
        }
        qs += nwarps;
        if (qs >= nseg) break;
        sd = seg.desc[qs];
        nb = near7(g, sd.x + lane, sd.y + lane, sd.z, sd.w, sd.y + lane < g.n0, lane);
        rec = load_rec7<double, false>(g, nb, sd.x + lane, sd.y + lane < g.n0, recf);
        raw = load_raw7(g, nb, sd.x + lane, 0, 0, 0, sd.y + lane < g.n0, rawf);
    }
    block_sum<1, kJacThreads, kJacThreads>(acc, sh, 0);
    if (threadIdx.x == 0) part.pap[blockIdx.x] = acc[0];
}

// K2 of iteration t: alpha = rz / p.Ap; x += alpha p; r -= alpha Ap; z = D^-1 r; r.r and r.z
__global__ void __launch_bounds__(kJacThreads, 1) jacobi_update_kernel(LGeom g, SegArg seg,
                                                                       const double* __restrict__ inv_diag,
                                                                       double* __restrict__ x, double* __restrict__ r,
                                                                       double* __restrict__ z,
                                                                       const double* __restrict__ p,
                                                                       const double* __restrict__ ap, Scalars* s,
                                                                       int slot, JacPart part) {
    __shared__ SumScratch<2, kJacThreads> sh;
    const int lane = threadIdx.x & 31;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    const int nseg = *seg.count;
    constexpr int U = 2;  // segments in flight a warp
    int qs = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    int c[U];
    bool live[U];
    double ic[U], pc[U], apc[U], xc[U], rc[U];
    auto cells = [&]() {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int q = qs + u * nwarps;
            const int4 sd = q < nseg ? seg.desc[q] : make_int4(0, g.n0, 0, 0);
            live[u] = sd.y + lane < g.n0;
            c[u] = sd.x + lane;
            ic[u] = live[u] ? inv_diag[c[u]] : 0.0;
        }
    };
    auto load = [&]() {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            pc[u] = live[u] ? p[c[u]] : 0.0;
            apc[u] = live[u] ? ap[c[u]] : 0.0;
            xc[u] = live[u] ? x[c[u]] : 0.0;
            rc[u] = live[u] ? r[c[u]] : 0.0;
        }
    };
    cells();
    pdl_wait();
    pdl_trigger();
    load();
    const int done = s->done;
    const double rz = s->rz2[slot];
    double t[1];
    sum_partials(part.pap, part.blocks, t);
    if (done) return;
    const double alpha = rz / t[0];
    if (!finite_d(alpha)) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            s->bad = 1;
            s->done = 1;
        }
        return;
    }
    double acc[2] = {0.0, 0.0};
    while (true) {
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (live[u]) {
                const double rn = rc[u] - alpha * apc[u];
                const double zn = rn * ic[u];
                x[c[u]] = xc[u] + alpha * pc[u];
                r[c[u]] = rn;
                z[c[u]] = zn;
                acc[0] += rn * rn;
                acc[1] += rn * zn;
            }
        qs += U * nwarps;
        if (qs >= nseg) break;
        cells();
        load();
    }
    block_sum<2, kJacThreads, kJacThreads>(acc, sh, 0);
    if (threadIdx.x == 0) {
        part.rr[2 * blockIdx.x] = acc[0];
        part.rr[2 * blockIdx.x + 1] = acc[1];
    }
}

// After the last iteration of a batch: its dot products into the scalars (the host polls them)
__global__ void jacobi_check_kernel(Scalars* s, int slot, JacPart part) {
    pdl_wait();
    pdl_trigger();
    const int done = s->done;
    const double rz_old = s->rz2[slot], thresh = s->thresh;
    double t[2];
    sum_partials(part.rr, part.blocks, t);
    if (done || threadIdx.x != 0) return;
    jacobi_store(s, jacobi_next(t, rz_old, thresh), slot ^ 1);
}

// Jacobi start: the reciprocal diagonal (0 on empty rows), z = D^-1 r and rz = r . z
__global__ void jacobi_start_kernel(LGeom g, SegArg seg, const double* __restrict__ diag, const double* __restrict__ r,
                                    double* __restrict__ inv_diag, double* __restrict__ z, Scalars* s,
                                    double* partials, unsigned* counter) {
    double acc[1] = {0.0};
    SEG_LOOP_BEGIN(seg, g)
    const double ic = row_inverse(diag[c]);
    const double rc = r[c];
    const double zc = rc * ic;
    inv_diag[c] = ic;
    z[c] = zc;
    acc[0] += rc * zc;
    SEG_LOOP_END
    double tot[1];
    if (grid_sum<1>(acc, partials, counter, tot)) s->rz2[0] = tot[0];
}

// The iterate as a float pair for the double-float residual (el_df.cuh), written with x by the
// kernels that change it (xs: null where no double-float residual reads it), shifted by the
// solve's power of two 2^df_shift (set from |b| by solve_init_kernel), which keeps the pairs
// of the whole system near 1 whatever its scale.  Beyond the pairs'
// range (|x| >= 2^128, an iterate no FP32 field can hold) the pair is infinite, so that the
// residual turns non-finite and the solve reports it.
__device__ __forceinline__ float2 x_pair(double x, int shift) {
    const double xs = d_shift(x, shift);
    bool ok = true;
    const F2 p = df_split(xs, ok);
    return ok ? make_float2(p.h, p.l) : make_float2(d2f(xs), 0.f);
}

// solve start (outer / plain): x = 0, r = b on the active segments, thresholds.
__global__ void solve_init_kernel(LGeom g, SegArg seg, const double* __restrict__ b, double* __restrict__ x,
                                  float2* __restrict__ xs, double* __restrict__ r, Scalars* s, double tol) {
    SEG_LOOP_BEGIN(seg, g)
    x[c] = 0.0;
    if (xs) xs[c] = make_float2(0.f, 0.f);
    r[c] = b[c];
    SEG_LOOP_END
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        const double bb = s->bb;
        // 2^df_shift |b| in [1, 2): the exponent of |b|^2 halved (0 for a zero or non-finite b)
        const unsigned long long bbits = (unsigned long long)__double_as_longlong(bb);
        const int eb = (int)((bbits >> 52) & 0x7ffu);
        s->df_shift = (eb == 0 || eb == 0x7ff) ? 0 : -((eb - 1023) >> 1);
        s->thresh = tol * tol * bb;
        s->rr = bb;
        s->iter = 0;
        s->bad = finite_d(bb) ? 0 : 1;
        s->done = (bb == 0.0 || bb < s->thresh || s->bad) ? 1 : 0;
        s->beta = 0.0;
        s->outer = 0;
        s->inner_total = 0;
        s->inner_passes = 0;
        s->iter_limit = INT_MAX;
        s->fault = 0;
    }
}

// the FP64 V-cycle's first sweep from zero for the first residual (later ones: update_kernel)
__global__ void first_sweep_kernel(LGeom g, SegArg seg, const double* __restrict__ r, const double* __restrict__ rd,
                                   double* __restrict__ t) {
    SEG_LOOP_BEGIN(seg, g)
    t[c] = rn_mul(rn_mul(kSweep1, r[c]), rd[c]);
    SEG_LOOP_END
}

// ---- warm start: x0 = alpha g with g the pressure grid as it stands --------------------
// x = g on fluid cells (0 elsewhere); the residual kernel then gives r0 = b - A g.
template <typename T>
__global__ void guess_load_kernel(LGeom g, SegArg seg, const T* __restrict__ guess, const double* __restrict__ diag,
                                  double* __restrict__ x) {
    SEG_LOOP_BEGIN(seg, g)
    x[c] = diag[c] > 0.0 ? (double)guess[c] : 0.0;
    SEG_LOOP_END
}

// alpha = (g.b) / (g.A g) with A g = b - r0: the scaling of g that minimises |x - x*|_A, so the
// scaled guess is never further from the solution in that norm than zero is.
__global__ void guess_alpha_kernel(LGeom g, SegArg seg, const double* __restrict__ x, const double* __restrict__ b,
                                   const double* __restrict__ r, Scalars* s, double* partials, unsigned* counter) {
    double acc[2] = {0.0, 0.0};
    SEG_LOOP_BEGIN(seg, g)
    const double xc = x[c];
    acc[0] += xc * b[c];
    acc[1] += xc * (b[c] - r[c]);
    SEG_LOOP_END
    double tot[2];
    if (grid_sum<2>(acc, partials, counter, tot)) {
        const double a = (tot[1] > 0.0 && finite_d(tot[0]) && finite_d(tot[1])) ? tot[0] / tot[1] : 0.0;
        s->aux = a;
    }
}

// x = alpha g, r = b - alpha A g = (1 - alpha) b + alpha r0, |r|^2 and the stopping test.
__global__ void guess_scale_kernel(LGeom g, SegArg seg, double* __restrict__ x, float2* __restrict__ xs,
                                   const double* __restrict__ b, double* __restrict__ r, Scalars* s,
                                   double* partials, unsigned* counter) {
    const double a = s->aux;
    double acc[1] = {0.0};
    SEG_LOOP_BEGIN(seg, g)
    // a == 0 (a useless or non-finite guess): exactly the zero start, whatever g held
    const double xc = a != 0.0 ? a * x[c] : 0.0;
    x[c] = xc;
    if (xs) xs[c] = x_pair(xc, s->df_shift);
    const double rc = a != 0.0 ? (1.0 - a) * b[c] + a * r[c] : b[c];
    r[c] = rc;
    acc[0] += rc * rc;
    SEG_LOOP_END
    double tot[1];
    if (grid_sum<1>(acc, partials, counter, tot)) {
        s->rr = tot[0];
        if (!finite_d(tot[0])) {
            s->bad = 1;
            s->done = 1;
        } else {
            s->done = (s->bb == 0.0 || tot[0] < s->thresh) ? 1 : 0;
        }
    }
}

// FP64 paths taken by few cells, kept out of line: the compiler would otherwise predicate them
// into the common path, where each FP64 instruction costs an issue slot of the FP64 pipe (the
// bound of these kernels) on every cell, switched off or not.
__device__ __noinline__ float scale_fp64(double r, double inv) { return (float)(r * inv); }

// |r| and 1 / |r| from |r|^2
__device__ __noinline__ double2 scale_from_norm(double rr) {
    const double norm = sqrt(rr);
    return make_double2(norm, norm > 0.0 ? 1.0 / norm : 0.0);
}

__device__ __noinline__ double residual_cell_fp64(double bc, double d, double x0, float cxm, double vxm, float cxp,
                                                  double vxp, float cym, double xym, float cyp, double xyp,
                                                  float czm, double xzm, float czp, double xzp) {
    return bc - stencil7(d, x0, f2d(cxm), vxm, f2d(cxp), vxp, f2d(cym), xym, f2d(cyp), xyp, f2d(czm), xzm, f2d(czp),
                         xzp);
}

// mixed solver: inner system r32 = r64 2^-k with 2^k the power of two at or below |r64| (the
// scaling is exact both ways, and |r32| lies in [1, 2)), x32 = 0, inner thresholds.  The scale
// comes from the exponent bits of |r|^2: square roots and divisions in FP64 by every thread cost
// more FP64 issue than the cells' own work.  A cell's value is shifted by the exponent field and
// rounded to float by integer arithmetic (d_shift, d2f): the inner system of a system scaled by
// a power of two is the same floats.  A zero, subnormal or non-finite |r|^2 takes the scale
// 1 / |r| in FP64.  The inner relative tolerance is what the outer one still needs,
// halved, kept within [floor, 1/2] (FP32 cannot go much below 1e-4 reliably):
// tau = clamp(0.5 tol |b| / |r|, floor, 0.5).
__global__ void inner_init_kernel(LGeom g, SegArg seg, const double* __restrict__ r64, float* __restrict__ r32,
                                  float* __restrict__ x32, const Scalars* so, Scalars* si, double tol,
                                  double tau_floor, int max_iter, double* partials, unsigned* counter) {
    const double rr = so->rr;
    const unsigned long long rb = (unsigned long long)__double_as_longlong(rr);
    const int erb = (int)((rb >> 52) & 0x7ffu);
    const int k = (erb - 1023) >> 1;
    // every positive normal |r|^2 gives a shift within the doubles' range (|k| <= 511)
    const bool pow2 = rb != 0ull && (rb >> 63) == 0ull && erb != 0 && erb != 0x7ff;
    double norm, inv;
    if (pow2) {
        norm = __longlong_as_double((long long)(1023 + k) << 52);
        inv = 0.0;
    } else {
        const double2 ni = scale_from_norm(rr);
        norm = ni.x;
        inv = ni.y;
    }
    float part = 0.f;
    // four segments a warp per pass, their loads in flight together (one load a cell)
    const int lane = threadIdx.x & 31;
    const int wg = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    const int nseg = *seg.count;
    constexpr int U = 4;
    for (int q0 = wg; q0 < nseg; q0 += U * nw) {
        int cc[U];
        bool lv[U];
        double rc[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int qs = q0 + u * nw;
            const int4 sd = qs < nseg ? seg.desc[qs] : make_int4(0, g.n0, 0, 0);
            cc[u] = sd.x + lane;
            lv[u] = qs < nseg && sd.y + lane < g.n0;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) rc[u] = lv[u] ? r64[cc[u]] : 0.0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (!lv[u]) continue;
            // r 2^-k by the exponent field, then rounded to float: exact scaling, integer pipe
            const float v = pow2 ? d2f(d_shift(rc[u], -k)) : scale_fp64(rc[u], inv);
            r32[cc[u]] = v;
            x32[cc[u]] = 0.0f;
            part += v * v;
        }
    }
    double acc[1] = {(double)part};
    double tot[1];
    if (grid_sum<1>(acc, partials, counter, tot)) {
        const double want = rr > 0.0 ? 0.5 * tol * sqrt(so->bb / rr) : 0.5;
        const double tau = fmin(0.5, fmax(tau_floor, want));
        si->bb = tot[0];
        si->rr = tot[0];
        si->thresh = tau * tau * tot[0];
        si->norm = norm;
        si->iter = 0;
        si->iter_limit = max_iter - so->inner_total;  // so->inner_total: by the device-driven loop
        si->bad = 0;
        si->fault = 0;
        si->beta = 0.0;
        si->done = (tot[0] == 0.0 || tot[0] < si->thresh) ? 1 : 0;
    }
}

// mixed solver: x64 += |r| * x32 (and its float pair)
__global__ void accumulate_kernel(LGeom g, SegArg seg, double* __restrict__ x64, float2* __restrict__ xs,
                                  const float* __restrict__ x32, const Scalars* si, const Scalars* so) {
    const double norm = si->norm;
    const int shift = so->df_shift;
    SEG_LOOP_BEGIN(seg, g)
    const double xn = __fma_rn(norm, f2d(x32[c]), x64[c]);
    x64[c] = xn;
    if (xs) xs[c] = x_pair(xn, shift);
    SEG_LOOP_END
}

// |r|^2 of a refinement residual into the scalars and the stopping test
__device__ __forceinline__ void residual_done(Scalars* s, double rr) {
    s->rr = rr;
    if (!finite_d(rr)) {
        s->bad = 1;
        s->done = 1;
    } else if (rr < s->thresh) {
        s->done = 1;
    }
}

// FP64 residual r = b - A x and |r|^2 (outer refinement step).
template <typename OT>
__global__ void __launch_bounds__(kSegThreads) residual_kernel(LGeom g, SegArg seg, SplitOp<OT> A,
                                                               const double* __restrict__ b,
                                                               const double* __restrict__ x, double* __restrict__ r,
                                                               Scalars* s, double* partials, unsigned* counter) {
    double acc[1] = {0.0};
    const SplitLoad<OT> recf{A};
    auto rawf = [&](int q, int, int, int) -> double { return x[q]; };
    auto valf = [](double raw, const Co<double>&) -> double { return raw; };
    SEG_LOOP_ALL_BEGIN(seg, g)
    const St7<double> st = gather7<double, false>(g, c, i, j, k, live, lane, recf, rawf, valf);
    if (live) {
        const double rc = d_positive(st.d) ? b[c] - apply7(st) : 0.0;
        r[c] = rc;
        acc[0] += rc * rc;
    }
    SEG_LOOP_END
    double tot[1];
    if (grid_sum<1>(acc, partials, counter, tot)) residual_done(s, tot[0]);
}

// The mixed solver's refinement residual r = b - A x and |r|^2 for FP32 fields, whose couplings
// are exact floats: double-float arithmetic on the FP32 pipe (el_df.cuh) in place of the FP64
// operations, which bound the FP64 kernel above (nine a cell, its FP64 pipe 86 % busy).  The
// iterate comes as float pairs (xs, written with x); b and the diagonal are split into pairs by
// integer arithmetic, b and the iterate shifted by the solve's power of two 2^df_shift (|b| near
// 1: the pairs' exponent range then holds the system at any scale, and the shift is undone
// exactly on r and |r|^2); the pair of r is
// within 2^-41 of the sum of its row's term magnitudes, and is stored as a double.  A warp in
// which any operand lies outside the pairs' exponent range (el_df.cuh) takes the FP64
// arithmetic of the kernel above for all its lanes (the splits of b and the diagonal decide).  |r|^2 is summed in FP32 per thread (each
// takes a few dozen cells; SqAcc keeps every square in range) and in FP64 over the grid.
__global__ void __launch_bounds__(kSegThreads, 4) residual_df_kernel(LGeom g, SegArg seg, SplitOp<float> A,
                                                                  const double* __restrict__ b,
                                                                  const double* __restrict__ x,
                                                                  const float2* __restrict__ xs,
                                                                  double* __restrict__ r, Scalars* s,
                                                                  double* partials, unsigned* counter) {
    SqAcc acc2;
    // the pairs hold b and x times 2^k (x_pair); the residual pair is r 2^k, shifted back
    const int sk = s->df_shift;
    SEG_LOOP_ALL_BEGIN(seg, g)
    const bool iym = live && j > 0, iyp = live && j < g.n1 - 1;
    const bool izm = live && k > 0, izp = live && k < g.n2 - 1;
    const bool ixm = lane == 0 && live && i > 0;
    const bool ixp = lane == 31 && live && i + 1 < g.n0;
    // loads, all issued before any value is formed
    const double d = live ? A.d[c] : 0.0;
    const double bc = live ? b[c] : 0.0;
    const float cxp = live ? A.x[c] : 0.f, cyp = live ? A.y[c] : 0.f, czp = live ? A.z[c] : 0.f;
    const float cym = iym ? A.y[c - g.s1] : 0.f, czm = izm ? A.z[c - g.s2] : 0.f;
    const float cxm_e = ixm ? A.x[c - 1] : 0.f;
    const float2 z2 = make_float2(0.f, 0.f);
    const float2 q0 = live ? xs[c] : z2;
    const float2 qym = iym ? xs[c - g.s1] : z2, qyp = iyp ? xs[c + g.s1] : z2;
    const float2 qzm = izm ? xs[c - g.s2] : z2, qzp = izp ? xs[c + g.s2] : z2;
    const float2 qxm_e = ixm ? xs[c - 1] : z2, qxp_e = ixp ? xs[c + 1] : z2;
    const bool act = live && d_positive(d);
    const bool xp_in = live && i + 1 < g.n0;
    const float cxm_s = __shfl_up_sync(kFull, cxp, 1);
    const float cxm = lane == 0 ? cxm_e : cxm_s;
    const F2 p0{q0.x, q0.y}, pym{qym.x, qym.y}, pyp{qyp.x, qyp.y}, pzm{qzm.x, qzm.y}, pzp{qzp.x, qzp.y};
    const F2 pxm_e{qxm_e.x, qxm_e.y}, pxp_e{qxp_e.x, qxp_e.y};
    bool ok = true;
    const F2 pd = df_split(d, ok), pb = df_split(d_shift(bc, sk), ok);
    F2 pxm, pxp;
    pxm.h = __shfl_up_sync(kFull, p0.h, 1);
    pxm.l = __shfl_up_sync(kFull, p0.l, 1);
    pxp.h = __shfl_down_sync(kFull, p0.h, 1);
    pxp.l = __shfl_down_sync(kFull, p0.l, 1);
    if (lane == 0) pxm = pxm_e;
    if (lane == 31) pxp = pxp_e;
    if (!xp_in) pxp = F2{0.f, 0.f};
    if (__all_sync(kFull, ok)) {
        if (act) {
            const F2 q = df_residual7(pb, pd, p0, cxm, pxm, cxp, pxp, cym, pym, cyp, pyp, czm, pzm, czp, pzp);
            r[c] = d_shift(__dadd_rn(f2d(q.h), f2d(q.l)), -sk);
            acc2.add(q.h);
        } else if (live) {
            r[c] = 0.0;
        }
    } else {
        // the FP64 arithmetic of residual_kernel, for every lane of the warp, on the double iterate
        const double x0 = live ? x[c] : 0.0;
        const double xym = iym ? x[c - g.s1] : 0.0, xyp = iyp ? x[c + g.s1] : 0.0;
        const double xzm = izm ? x[c - g.s2] : 0.0, xzp = izp ? x[c + g.s2] : 0.0;
        const double xxm_e = ixm ? x[c - 1] : 0.0, xxp_e = ixp ? x[c + 1] : 0.0;
        const double sxm = __shfl_up_sync(kFull, x0, 1), sxp = __shfl_down_sync(kFull, x0, 1);
        if (live) {
            const double vxm = lane == 0 ? xxm_e : sxm;
            const double vxp = xp_in ? (lane == 31 ? xxp_e : sxp) : 0.0;
            const double rc = act ? residual_cell_fp64(bc, d, x0, cxm, vxm, cxp, vxp, cym, xym, cyp, xyp, czm, xzm,
                                                       czp, xzp)
                                  : 0.0;
            r[c] = rc;
            acc2.add(d2f(d_shift(rc, sk)));
        }
    }
    SEG_LOOP_END
    double acc[1] = {acc2.value()};
    double tot[1];
    if (grid_sum<1>(acc, partials, counter, tot)) residual_done(s, d_shift(tot[0], -2 * sk));
}


// ---------------------------------------------------------------------------------------
// multigrid smoothing over the active segments of one level
//
// MODE 0: two sweeps from x = 0 (the first, omega b / D, formed on the fly; FP32)
// MODE 1: one sweep from x_in + P e (e = coarse correction, formed on the fly)
// MODE 2: one sweep from x_in.   DOT (finest level, last sweep): rz = b . x_out and beta.
//
// In FP64 these kernels are bound by the FP64 pipe (2 lanes a clock per SM; a division costs about nine
// of its operations, a comparison one), so nothing in a sweep divides or compares there: the
// reciprocals of the diagonal are taken once a solve (rd), the sign of a diagonal is read as an
// integer, and the first sweep from zero is stored by the kernel that forms b (update_kernel on the
// finest level, the restrictions below), not divided out at every point of the second sweep's stencil.
// 128^3 pool, finest level: second sweep from zero 97 -> 17 us (reads t), prolongation sweep 40 -> 23,
// last sweep 38 -> 21.
enum { SM_ZERO2 = 0, SM_PROLONG = 1, SM_PLAIN = 2 };

// a / d inside the FP32 multigrid preconditioner: the fast division (within 2 ulp; the preconditioner
// only has to be a fixed symmetric operator, not correctly rounded)
__device__ __forceinline__ float mg_div(float a, float d) { return __fdividef(a, d); }
enum { DOT_NONE = 0, DOT_INIT = 1, DOT_BETA = 2 };

// A value of an iterate or right-hand side.  COH: through L2 only (ld.global.cg), for arrays
// that other CTAs of the same launch wrote (the fused coarse cycle); a read-only-cache load
// would not see those writes.
template <bool COH, typename V>
__device__ __forceinline__ V ldv(const V* p, int q) {
    if constexpr (COH)
        return __ldcg(p + q);
    else
        return p[q];
}

// One smoothing sweep over the active segments of a level, warp wg of nw warps taking segments
// wg, wg + nw, ...; returns the thread's share of b.x when DOT is set.
// ZERO2: first sweep (formed on the fly) w1, this sweep w2; PROLONG: w1; PLAIN: w2.  start() is called
// once the first segment's list entry and records, which no kernel of an iteration writes, are on
// their way, and before anything else is read; false ends the call.
template <typename V, typename R, int MODE, int DOT, bool COH = false, typename Start>
__device__ __forceinline__ DotAcc<V> smooth_segments(const LGeom& g, const SegArg& seg, const R* __restrict__ A,
                                                     const V* __restrict__ b, const V* __restrict__ x_in,
                                                     const LGeom& gc, const V* __restrict__ e, V* __restrict__ x_out,
                                                     const V* __restrict__ rd, int wg, int nw, Start&& start) {
    static_assert(sizeof(V) == 4 || MODE != SM_ZERO2, "FP64 stores the first sweep");
    [[maybe_unused]] const V w_first = V(kSweep1);
    const V omega = V(MODE == SM_PROLONG ? kSweep1 : kSweep2);
    DotAcc<V> part = 0;
    const RecLoad<V, R> recf{A};
    auto rawf = [&](int q, int qi, int qj, int qk) -> V {
        if (MODE == SM_ZERO2) return ldv<COH>(b, q);
        V v = ldv<COH>(x_in, q);
        if (MODE == SM_PROLONG) v += ldv<COH>(e, (qi >> 1) + gc.s1 * (qj >> 1) + gc.s2 * (qk >> 1));
        return v;
    };
    // the current iterate at a cell.  A stored value is read as it is: it is finite everywhere, and a
    // coupling with a cell outside the system is zero; so the records of the +y and +z neighbours are
    // not read for their diagonals (two of five records a cell: last sweep of 151 x 97 x 133 12.3 -> 11.0
    // us, of a 128^3 level 8.0 -> 7.0)
    auto valf = [&](V raw, [[maybe_unused]] const Co<V>& rec) -> V {
        if constexpr (MODE == SM_ZERO2) return positive(rec.d) ? mg_div(rn_mul(w_first, raw), rec.d) : V(0);
        return raw;
    };
    const int lane = threadIdx.x & 31;
    int qs = wg;
    const int nseg = *seg.count;
    int4 sd = qs < nseg ? seg.desc[qs] : make_int4(0, g.n0, 0, 0);
    Near7 nb = near7(g, sd.x + lane, sd.y + lane, sd.z, sd.w, sd.y + lane < g.n0, lane);
    Rec7<V> rec = load_rec7<V, MODE == SM_ZERO2>(g, nb, sd.x + lane, sd.y + lane < g.n0, recf);
    if (!start()) return part;
    while (qs < nseg) {
        const bool live = sd.y + lane < g.n0;
        const int c = sd.x + lane;
        const auto raw = load_raw7(g, nb, c, sd.y + lane, sd.z, sd.w, live, rawf);
        const V bc = live ? ldv<COH>(b, c) : V(0), rc = sizeof(V) == 8 && live ? rd[c] : V(0);
        const St7<V> st = value7<V>(nb, rec, raw, live, lane, valf);
        if (live) {
            V xo = V(0);
            if (positive(st.d)) {
                const V q = rn_mul(omega, rn_sub(bc, apply7(st)));
                if constexpr (sizeof(V) == 8)
                    xo = rn_fma(q, rc, st.v0);
                else
                    xo = rn_add(st.v0, mg_div(q, st.d));
            }
            if (EL_IN(c, (long long)g.s2 * g.n2, 30)) x_out[c] = xo;
            if (DOT != DOT_NONE) part += (DotAcc<V>)bc * (DotAcc<V>)xo;
        }
        qs += nw;
        if (qs >= nseg) break;
        sd = seg.desc[qs];
        nb = near7(g, sd.x + lane, sd.y + lane, sd.z, sd.w, sd.y + lane < g.n0, lane);
        rec = load_rec7<V, MODE == SM_ZERO2>(g, nb, sd.x + lane, sd.y + lane < g.n0, recf);
    }
    return part;
}

// K2 of the FP32 solver and the V-cycle's first kernel in one: x += alpha p, r_out = r - alpha Ap, |r|^2,
// and z = two sweeps from zero on r_out, which is formed again at the points of the stencil (so r_out
// is another buffer).  The two are bound by launch and load latency on the scenes that do not take the
// tile kernels (which do the same).  Mixed solve of 75 x 62 x 53 cells 0.96 -> 0.90 ms, 48^3 0.67 -> 0.64;
// up to two waves of warps: 96^3 1.06 -> 1.03, 110 x 127 x 118 and 151 x 97 x 133 the same, and twelve
// scenes at once 8.95 -> 9.05 ms, where its second reading of r and Ap is not hidden.
template <typename R>
__global__ void __launch_bounds__(kDotThreads<float>) update_smooth_kernel(LGeom g, SegArg seg, const R* __restrict__ A,
                                                                          float* __restrict__ x,
                                                                          const float* __restrict__ r,
                                                                          float* __restrict__ r_out,
                                                                          const float* __restrict__ p,
                                                                          const float* __restrict__ ap,
                                                                          float* __restrict__ z, Scalars* s,
                                                                          double* partials, unsigned* counter) {
    const RecLoad<float, R> recf{A};
    const int lane = threadIdx.x & 31;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    int qs = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nseg = *seg.count;
    int4 sd = qs < nseg ? seg.desc[qs] : make_int4(0, g.n0, 0, 0);
    Near7 nb = near7(g, sd.x + lane, sd.y + lane, sd.z, sd.w, sd.y + lane < g.n0, lane);
    Rec7<float> rec = load_rec7<float, true>(g, nb, sd.x + lane, sd.y + lane < g.n0, recf);
    pdl_wait();
    pdl_trigger();
    if (s->done) return;
    const float alpha = (float)s->alpha, w1 = (float)kSweep1, w2 = (float)kSweep2;
    float part = 0.f;
    auto rawf = [&](int q, int, int, int) -> float2 { return make_float2(r[q], ap[q]); };
    auto residual = [&](float2 v) -> float { return v.x - alpha * v.y; };
    auto valf = [&](float2 v, const Co<float>& c) -> float {
        return positive(c.d) ? mg_div(rn_mul(w1, residual(v)), c.d) : 0.f;
    };
    while (qs < nseg) {
        const bool live = sd.y + lane < g.n0;
        const int c = sd.x + lane;
        const auto raw = load_raw7(g, nb, c, 0, 0, 0, live, rawf);
        const float xc = live ? x[c] : 0.f, pc = live ? p[c] : 0.f;
        const St7<float> st = value7<float>(nb, rec, raw, live, lane, valf);
        if (live) {
            const float rc = residual(raw.a0);
            float zc = 0.f;
            if (positive(st.d)) zc = rn_add(st.v0, mg_div(rn_mul(w2, rn_sub(rc, apply7(st))), st.d));
            x[c] = xc + alpha * pc;
            r_out[c] = rc;
            z[c] = zc;
            part += rc * rc;
        }
        qs += nwarps;
        if (qs >= nseg) break;
        sd = seg.desc[qs];
        nb = near7(g, sd.x + lane, sd.y + lane, sd.z, sd.w, sd.y + lane < g.n0, lane);
        rec = load_rec7<float, true>(g, nb, sd.x + lane, sd.y + lane < g.n0, recf);
    }
    update_done<float>(part, s, partials, counter);
}

// (the sweeps with a dot product keep eight blocks an SM: the grid is part of the sum's order)
template <typename V, typename R, int MODE, int DOT>
__global__ void __launch_bounds__(kSegThreads, DOT != DOT_NONE && sizeof(V) == 4 ? 8 : 1) smooth_kernel(LGeom g, SegArg seg, const R* __restrict__ A,
                                                             const V* __restrict__ b, const V* __restrict__ x_in,
                                                             LGeom gc, const V* __restrict__ e,
                                                             V* __restrict__ x_out, const V* __restrict__ rd,
                                                             Scalars* s, double* partials, unsigned* counter) {
    bool go = false;
    auto start = [&] {
        pdl_wait();
        pdl_trigger();
        return go = !s->done;
    };
    const DotAcc<V> part = smooth_segments<V, R, MODE, DOT>(g, seg, A, b, x_in, gc, e, x_out, rd,
                                                            (blockIdx.x * blockDim.x + threadIdx.x) >> 5,
                                                            (gridDim.x * blockDim.x) >> 5, start);
    if (!go) return;
    if (DOT != DOT_NONE) {
        double acc[1] = {(double)part};
        double tot[1];
        if (grid_sum<1>(acc, partials, counter, tot)) {
            if (DOT == DOT_BETA) s->beta = tot[0] / s->rz;
            s->rz = tot[0];
            if (!finite_d(tot[0])) {
                s->bad = 1;
                s->done = 1;
            }
        }
    }
}

// Residual of a level summed onto the coarse right-hand side (R = P^T): a quad of four
// warps takes one active coarse segment: warp (kk, jj) of the quad walks the fine row
// (2J + jj, 2K + kk) under it, 64 fine cells as two 32-cell halves (one fine cell per lane,
// coalesced); the quad then adds its four rows in a fixed order through shared memory
// (deterministic).  Four rows in flight per coarse segment: the kernel is bound by the latency of
// the gathers.  The finest level (FINEST) sums a cell's column over the rows before the i-pairs, the
// other levels the pairs of a row first.  A warp a coarse segment, eight gathers in sequence, was as
// fast on the finest level of 150 cells an axis and slower below: solve of 75 x 62 x 53 1.02 -> 0.96 ms,
// of 48^3 0.72 -> 0.67 (finest level: 10 -> 4 us a launch).
constexpr int kQuadsPerBlock = kSegThreads / 128;

// The quads' walk: quad `quad` of `nquads`, the block's quad quad_b (named barrier 1 + quad_b),
// row `sub` of it; part = the block's [quads][4][2][16] sums in shared memory; start() as for
// smooth_segments.
template <typename V, typename R, bool FINEST, bool COH = false, typename Start>
__device__ __forceinline__ void restrict_quad_segments(const LGeom& g, const R* __restrict__ A,
                                                       const V* __restrict__ b, const V* __restrict__ x,
                                                       const LGeom& gc, const SegArg& cseg, V* __restrict__ bc,
                                                       V* __restrict__ tc, const V* __restrict__ rdc,
                                                       V (*part)[4][2][FINEST ? 32 : 16], int quad, int nquads, int quad_b,
                                                       int sub, Start&& start) {
    const RecLoad<V, R> recf{A};
    auto rawf = [&](int q, int, int, int) -> V { return ldv<COH>(x, q); };
    auto valf = [](V raw, const Co<V>&) -> V { return raw; };
    const int lane = threadIdx.x & 31;
    const int kk = sub >> 1, jj = sub & 1;
    int qs = quad;
    const int nseg = *cseg.count;
    int4 sd = qs < nseg ? cseg.desc[qs] : make_int4(0, g.n0, 0, 0);
    // half h of the quad's row under a coarse segment: its fine cell at this lane, and that cell's
    // records (the row exists for all lanes of the warp or for none)
    Near7 nb[2];
    Rec7<V> rec[2];
    auto cell = [&](int h, int& c, int& i, int& j, int& k) -> bool {
        i = 2 * sd.y + 32 * h + lane;
        j = 2 * sd.z + jj;
        k = 2 * sd.w + kk;
        c = i + g.s1 * j + g.s2 * k;
        return i < g.n0 && j < g.n1 && k < g.n2;
    };
    auto records = [&] {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            int c, i, j, k;
            const bool live = cell(h, c, i, j, k);
            nb[h] = near7(g, c, i, j, k, live, lane);
            rec[h] = load_rec7<V, false>(g, nb[h], c, live, recf);
        }
    };
    records();
    if (!start()) return;
    while (qs < nseg) {
        const int I0 = sd.y, J = sd.z, K = sd.w;
        V sum[2] = {V(0), V(0)};  // fine i in [2*I0, 2*I0+32) and [2*I0+32, 2*I0+64)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            int c, i, j, k;
            const bool live = cell(h, c, i, j, k);
            const auto raw = load_raw7(g, nb[h], c, i, j, k, live, rawf);
            const V bv = live ? ldv<COH>(b, c) : V(0);
            const St7<V> st = value7<V>(nb[h], rec[h], raw, live, lane, valf);
            if (live && positive(st.d)) sum[h] = rn_sub(bv, apply7(st));
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if constexpr (FINEST) {
                part[quad_b][sub][h][lane] = sum[h];
            } else {
                const V pair = sum[h] + __shfl_down_sync(kFull, sum[h], 1);
                if ((lane & 1) == 0) part[quad_b][sub][h][lane >> 1] = pair;
            }
        }
        // the quad's four warps meet on their own named barrier (1 + quad in the block)
        asm volatile("bar.sync %0, %1;" ::"r"(1 + quad_b), "r"(128) : "memory");
        if (sub == 0) {
            const int h = lane >> 4, q = lane & 15;
            auto rows = [&](int n) {
                return ((part[quad_b][0][h][n] + part[quad_b][1][h][n]) + part[quad_b][2][h][n]) +
                       part[quad_b][3][h][n];
            };
            const V tot = FINEST ? rows(2 * q) + rows(2 * q + 1) : rows(q);
            const int I = I0 + 16 * h + q;
            const int o = I + gc.s1 * J + gc.s2 * K;
            if (I < gc.n0 && EL_IN(o, (long long)gc.s2 * gc.n2, 32)) {
                bc[o] = tot;
                if (sizeof(V) == 8) tc[o] = rn_mul(rn_mul(V(kSweep1), tot), rdc[o]);
            }
        }
        asm volatile("bar.sync %0, %1;" ::"r"(1 + quad_b), "r"(128) : "memory");
        qs += nquads;
        if (qs >= nseg) break;
        sd = cseg.desc[qs];
        records();
    }
}

template <typename V, typename R, bool FINEST>
__global__ void __launch_bounds__(kSegThreads, 4) restrict_quad_kernel(LGeom g, const R* __restrict__ A,
                                                                    const V* __restrict__ b, const V* __restrict__ x,
                                                                    LGeom gc, SegArg cseg, V* __restrict__ bc,
                                                                    V* __restrict__ tc, const V* __restrict__ rdc,
                                                                    const Scalars* s) {
    __shared__ V part[kQuadsPerBlock][4][2][FINEST ? 32 : 16];
    const int wb = threadIdx.x >> 5;                  // warp in the block
    const int quad_b = wb >> 2, sub = wb & 3;         // quad in the block, row of the quad
    restrict_quad_segments<V, R, FINEST>(g, A, b, x, gc, cseg, bc, tc, rdc, part, blockIdx.x * kQuadsPerBlock + quad_b,
                                 gridDim.x * kQuadsPerBlock, quad_b, sub, [&] {
                                     pdl_wait();
                                     pdl_trigger();
                                     return !s->done;
                                 });
}


// Coarsest level: omega-Jacobi sweeps from zero in one block's shared memory, a thread a cell, its
// row in registers.  In FP64 the row is scaled by omega / D beforehand, which leaves a sweep seven
// multiply-adds (the FP64 pipe of one SM bounds it): 512 cells 38 -> 21 us
template <typename V, typename R>
__global__ void __launch_bounds__(kCoarsestMaxCells) coarsest_kernel(LGeom g, const R* __restrict__ A,
                                                                     const V* __restrict__ b, V* __restrict__ x,
                                                                     const V* __restrict__ rd, int sweeps,
                                                                     const Scalars* s) {
    __shared__ V xs[2][kCoarsestMaxCells];
    const int n = g.n0 * g.n1 * g.n2;
    const int c = threadIdx.x;
    const V omega = V(kOmega);
    const int i = c % g.n0, j = (c / g.n0) % g.n1, k = c / (g.n0 * g.n1);
    const int s1 = g.n0, s2 = g.n0 * g.n1;
    const Co<V> z4{V(0), V(0), V(0), V(0)};
    auto rec = [&](bool in, int q) -> Co<V> {
        if (!in) return z4;
        const auto r = ldrec(A, q);
        return Co<V>{(V)r.d, (V)r.x, (V)r.y, (V)r.z};
    };
    const bool in = c < n;
    const Co<V> r0 = rec(in, c);
    const bool act = positive(r0.d);
    const bool hxm = act && i > 0, hxp = act && i < g.n0 - 1, hym = act && j > 0, hyp = act && j < g.n1 - 1;
    const bool hzm = act && k > 0, hzp = act && k < g.n2 - 1;
    V cxm = rec(hxm, c - 1).x, cym = rec(hym, c - s1).y, czm = rec(hzm, c - s2).z;
    V cxp = hxp ? r0.x : V(0), cyp = hyp ? r0.y : V(0), czp = hzp ? r0.z : V(0);
    // an absent neighbour: coefficient 0 at the cell itself
    const int qxm = hxm ? c - 1 : c, qxp = hxp ? c + 1 : c, qym = hym ? c - s1 : c, qyp = hyp ? c + s1 : c;
    const int qzm = hzm ? c - s2 : c, qzp = hzp ? c + s2 : c;
    [[maybe_unused]] const V w = sizeof(V) == 8 && act ? rn_mul(omega, rd[c]) : V(0);
    pdl_wait();
    pdl_trigger();
    if (s->done) return;
    V bc = in ? b[c] : V(0);
    V x0 = V(0);
    if constexpr (sizeof(V) == 8) {
        cxm = rn_mul(cxm, -w);
        cxp = rn_mul(cxp, -w);
        cym = rn_mul(cym, -w);
        cyp = rn_mul(cyp, -w);
        czm = rn_mul(czm, -w);
        czp = rn_mul(czp, -w);
        x0 = bc = rn_mul(bc, w);
    } else {
        if (act) x0 = mg_div(rn_mul(omega, bc), r0.d);
    }
    xs[0][c] = x0;
    __syncthreads();
    for (int it = 1; it < sweeps; ++it) {
        const V* cur = xs[(it - 1) & 1];
        if (act) {
            if constexpr (sizeof(V) == 8) {
                V a = rn_fma(V(1.0 - kOmega), x0, bc);
                a = rn_fma(cxm, cur[qxm], a);
                a = rn_fma(cxp, cur[qxp], a);
                a = rn_fma(cym, cur[qym], a);
                a = rn_fma(cyp, cur[qyp], a);
                a = rn_fma(czm, cur[qzm], a);
                x0 = rn_fma(czp, cur[qzp], a);
            } else {
                V a = rn_mul(r0.d, x0);
                if (hxm) a = rn_fma(cxm, cur[qxm], a);
                if (hxp) a = rn_fma(cxp, cur[qxp], a);
                if (hym) a = rn_fma(cym, cur[qym], a);
                if (hyp) a = rn_fma(cyp, cur[qyp], a);
                if (hzm) a = rn_fma(czm, cur[qzm], a);
                if (hzp) a = rn_fma(czp, cur[qzp], a);
                x0 = rn_add(x0, mg_div(rn_mul(omega, rn_sub(bc, a)), r0.d));
            }
        }
        xs[it & 1][c] = x0;
        __syncthreads();
    }
    if (in) x[c] = x0;
}

// ---------------------------------------------------------------------------------------
// The bottom of the FP32 V-cycle in one CTA.  Coarsening stops once the largest dimension is
// at most 8, so the level above the coarsest holds at most 16^3 cells: one launch of 1024 threads
// does what the segment kernels do in five: the two sweeps from zero, the restriction, the coarsest
// level's solve, the prolongation sweep and the last sweep, over the dense level (cells with no
// diagonal come out 0, as they contribute nothing to their neighbours), with barriers between the
// passes instead of kernel boundaries.  Only the level's final x goes back to global memory (the
// finer level's prolongation reads it).
//
// One SM's shared memory bounds the passes: a float4 record a neighbour, read in every pass, was 23
// wavefronts a warp and cell.  So a thread owns C cells in a row along z, (t mod 16, t / 16 mod 16,
// C (t / 256) + m), with their couplings, right-hand side and values in registers, and reads only the
// neighbours' values in x and y and above and below its own; the couplings are loaded before the wait
// for the kernel before.  512 threads of eight cells: 1024 of four (the fused coarse cycle's) leave
// a thread 64 registers, which the coarsest level's rows do not fit beside the level's.
// 16^3 and 8^3: 17.5 -> 13.4 us, of which 1.6 may pass before the kernel before ends; 12^3 and 6^3
// 14.0 -> 11.7.  The coarsest level's 30 sweeps are bound by the latency of a sweep (a barrier, the
// neighbours' values, seven dependent multiply-adds): with a cell a thread 0.13 us each, with two 0.16,
// with four 0.31.
constexpr int kBottomThreads = 512;   // of mg_bottom_kernel
constexpr int kCycleThreads = 1024;   // of mg_coarse_cycle_kernel
constexpr int kBottomDim = 16;        // the level's cells are (i, j, k) at i + 16 j + 256 k in shared memory
// the coarsest level's cells are at i + 8 j + 64 k; kBottomCoarseThreads threads own them
constexpr int kBottomCoarseThreads = 512;

struct BottomSmem {
    float v[2][kBottomDim * kBottomDim * kBottomDim];
    float4 rec[kCoarsestMaxCells];  // the coarsest level's
    float c[2][kCoarsestMaxCells];
};

// C cells along z, (i, j, k0 + m), of a dense level of at most N cells an axis, stored with pitches N and
// N * N: couplings (0 towards cells outside), and the places of the neighbours outside the C (the cell
// itself where there is none)
template <int C, int N>
struct Column {
    static constexpr int PY = N, PZ = N * N;
    float d[C], cxm[C], cxp[C], cym[C], cyp[C], cz[C + 1];  // cz[m]: between k0 + m - 1 and k0 + m
    int at, xm, xp, ym, yp, zm, zp;
    bool live[C];
    template <typename RF>
    __device__ __forceinline__ void load(int i, int j, int k0, int n0, int n1, int n2, RF&& recf) {
        at = i + PY * j + PZ * k0;
        xm = i > 0 ? -1 : 0;
        xp = i + 1 < N ? 1 : 0;
        ym = j > 0 ? -PY : 0;
        yp = j + 1 < N ? PY : 0;
        zm = k0 > 0 ? -PZ : 0;
        zp = k0 + C < N ? C * PZ : (C - 1) * PZ;
        const bool row = i < n0 && j < n1;
        const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
        cz[0] = row && k0 > 0 && k0 < n2 ? recf(i, j, k0 - 1).w : 0.f;
#pragma unroll
        for (int m = 0; m < C; ++m) {
            live[m] = row && k0 + m < n2;
            const float4 r = live[m] ? recf(i, j, k0 + m) : z4;
            d[m] = r.x;
            cxp[m] = i + 1 < n0 ? r.y : 0.f;
            cyp[m] = j + 1 < n1 ? r.z : 0.f;
            cz[m + 1] = k0 + m + 1 < n2 ? r.w : 0.f;
            cxm[m] = live[m] && i > 0 ? recf(i - 1, j, k0 + m).y : 0.f;
            cym[m] = live[m] && j > 0 ? recf(i, j - 1, k0 + m).z : 0.f;
        }
    }
    // A x at the four cells, x also in v[] (of every cell of the level)
    __device__ __forceinline__ void apply(const float* v, const float (&x)[C], float (&ax)[C]) const {
        const float* q = v + at;
        const float below = q[zm], above = q[zp];
#pragma unroll
        for (int m = 0; m < C; ++m) {
            const float* c = q + m * PZ;
            ax[m] = stencil7(d[m], x[m], cxm[m], c[xm], cxp[m], c[xp], cym[m], c[ym], cyp[m], c[yp], cz[m],
                             m ? x[m - 1] : below, cz[m + 1], m + 1 < C ? x[m + 1] : above);
        }
    }
};

// The coarsest level (right-hand side in sm.c[0], the result too): damped Jacobi from zero as
// coarsest_kernel, by kBottomCoarseThreads threads on named barrier 15.
__device__ __forceinline__ void coarsest_solve(BottomSmem& sm, int tid, const LGeom& gc) {
    constexpr int C = kCoarsestMaxCells / kBottomCoarseThreads;
    const float omega = (float)kOmega;
    Column<C, 8> A;
    A.load(tid & 7, (tid >> 3) & 7, C * (tid >> 6), gc.n0, gc.n1, gc.n2,
           [&](int i, int j, int k) { return sm.rec[i + 8 * j + 64 * k]; });
    float b[C], x[C], t[C];
#pragma unroll
    for (int m = 0; m < C; ++m) {
        b[m] = sm.c[0][A.at + 64 * m];
        x[m] = A.d[m] > 0.f ? mg_div(rn_mul(omega, b[m]), A.d[m]) : 0.f;
    }
    auto put = [&](float* v) {
#pragma unroll
        for (int m = 0; m < C; ++m) v[A.at + 64 * m] = x[m];
        asm volatile("bar.sync 15, %0;" ::"r"(kBottomCoarseThreads) : "memory");
    };
    static_assert(kCoarsestSweeps % 2 == 0, "the last sweep's values go to sm.c[0]");
#pragma unroll 2
    for (int it = 1; it < kCoarsestSweeps; ++it) {
        float* v = sm.c[it & 1];
        put(v);
        A.apply(v, x, t);
#pragma unroll
        for (int m = 0; m < C; ++m)
            x[m] = A.d[m] > 0.f ? rn_add(x[m], mg_div(rn_mul(omega, rn_sub(b[m], t[m])), A.d[m])) : 0.f;
    }
    put(sm.c[0]);
}

// the bottom's passes by one CTA of 4096 / C threads
template <int C, typename Start>
__device__ __forceinline__ void bottom_cycle(const LGeom& gf, const float4* __restrict__ recf,
                                             const float* __restrict__ bf, float* __restrict__ xf, const LGeom& gc,
                                             const float4* __restrict__ recc, unsigned char* bottom_smem,
                                             Start&& start) {
    BottomSmem& sm = *reinterpret_cast<BottomSmem*>(bottom_smem);
    const float w1 = (float)kSweep1, w2 = (float)kSweep2;
    const int tid = threadIdx.x;
    const int fi = tid & 15, fj = (tid >> 4) & 15, k0 = C * (tid >> 8);
    Column<C, 16> A;
    A.load(fi, fj, k0, gf.n0, gf.n1, gf.n2,
           [&](int i, int j, int k) { return recf[i + gf.s1 * j + gf.s2 * k]; });
    if (tid < kCoarsestMaxCells) {
        const int ci = tid & 7, cj = (tid >> 3) & 7, ck = tid >> 6;
        sm.rec[tid] = ci < gc.n0 && cj < gc.n1 && ck < gc.n2 ? recc[ci + gc.s1 * cj + gc.s2 * ck]
                                                             : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (!start()) return;
    float b[C], x[C], t[C];
#pragma unroll
    for (int m = 0; m < C; ++m)  // (b may have been written by other CTAs of the fused coarse cycle)
        b[m] = A.live[m] ? __ldcg(bf + fi + gf.s1 * fj + gf.s2 * (k0 + m)) : 0.f;
    auto put = [&](float* v) {
#pragma unroll
        for (int m = 0; m < C; ++m) v[A.at + 256 * m] = x[m];
        __syncthreads();
    };
    auto sweep = [&](const float* v, float w) {
        A.apply(v, x, t);
#pragma unroll
        for (int m = 0; m < C; ++m)
            x[m] = A.d[m] > 0.f ? rn_add(x[m], mg_div(rn_mul(w, rn_sub(b[m], t[m])), A.d[m])) : 0.f;
    };
    // two sweeps from zero: the first is pointwise
#pragma unroll
    for (int m = 0; m < C; ++m) x[m] = A.d[m] > 0.f ? mg_div(rn_mul(w1, b[m]), A.d[m]) : 0.f;
    put(sm.v[0]);
    sweep(sm.v[0], w2);
    put(sm.v[1]);
    // residual, then its 2 x 2 x 2 sums onto the coarsest level (order of the segment kernels:
    // i-pairs of the rows (jj, kk) = (0,0), (1,0), (0,1), (1,1), summed in that order); a warp holds
    // 16 cells in x of two rows in y
    A.apply(sm.v[1], x, t);
    {
        float p[C], q[C];
#pragma unroll
        for (int m = 0; m < C; ++m) {
            const float r = A.d[m] > 0.f ? rn_sub(b[m], t[m]) : 0.f;
            p[m] = r + __shfl_down_sync(kFull, r, 1);
            q[m] = __shfl_down_sync(kFull, p[m], 16);
        }
        if (!(tid & 17)) {
            float* c = sm.c[0] + (fi >> 1) + 8 * (fj >> 1) + 64 * (k0 >> 1);
#pragma unroll
            for (int h = 0; h < C / 2; ++h) c[64 * h] = ((p[2 * h] + q[2 * h]) + p[2 * h + 1]) + q[2 * h + 1];
        }
    }
    __syncthreads();
    if (tid < kBottomCoarseThreads) coarsest_solve(sm, tid, gc);
    __syncthreads();
    // prolongation (x + P e) and a sweep, then the last sweep into global memory
    {
        const float* e = sm.c[0] + (fi >> 1) + 8 * (fj >> 1) + 64 * (k0 >> 1);
#pragma unroll
        for (int m = 0; m < C; ++m) x[m] = A.live[m] ? x[m] + e[64 * (m / 2)] : 0.f;
    }
    put(sm.v[0]);
    sweep(sm.v[0], w1);
    put(sm.v[1]);
    sweep(sm.v[1], w2);
#pragma unroll
    for (int m = 0; m < C; ++m)
        if (A.live[m]) xf[fi + gf.s1 * fj + gf.s2 * (k0 + m)] = x[m];
}

__global__ void __launch_bounds__(kBottomThreads) mg_bottom_kernel(LGeom gf, const float4* __restrict__ recf,
                                                                   const float* __restrict__ bf,
                                                                   float* __restrict__ xf, LGeom gc,
                                                                   const float4* __restrict__ recc,
                                                                   const Scalars* s) {
    extern __shared__ __align__(16) unsigned char bottom_smem[];
    bottom_cycle<8>(gf, recf, bf, xf, gc, recc, bottom_smem, [&] {
        pdl_wait();
        pdl_trigger();
        return !s->done;
    });
}

// ---------------------------------------------------------------------------------------
// The coarse levels of one FP32 V-cycle in one cooperative launch.  Below the finest level the
// segment kernels are launches of a few microseconds each (about 13 per V-cycle at 256^3:
// two sweeps from zero and the restriction per level going down, the bottom, the prolongation
// sweep and the last sweep per level coming up), so the V-cycle's coarse part was bound by
// launch latency.  Here one launch of 1024-thread CTAs, all resident at once (a cooperative
// launch), runs the same passes -- the same device functions, so the same expressions in the
// same order and bit-identical results -- separated by grid barriers; the bottom pair (<= 16^3
// and the coarsest level) runs in CTA 0's shared memory while the others wait at the next
// barrier.  Arrays written by one pass and read by another are loaded through L2
// (ld.global.cg).  Every barrier wait is bounded: a CTA that gives up marks the solve as failed
// (fault, bad, done) and leaves; the other CTAs' waits then run out too.
constexpr int kCoarseMaxLevels = 16;
constexpr int kCoopQuads = kCycleThreads / 128;  // restriction quads per CTA
constexpr long long kBarrierPolls = 1ll << 21;    // past the first 4096, each poll sleeps ~100 ns: ~0.2 s

struct CoarseLevel {
    LGeom g;
    const float4* rec;
    float* b;
    float* x;
    float* t;
    SegArg seg;
};

struct CoarseCycle {
    CoarseLevel lv[kCoarseMaxLevels];  // by hierarchy level
    int from, pre_end;                 // levels [from, pre_end) go down and up; pre_end, pre_end + 1: bottom
    int sweeps;                        // coarsest-level sweeps
    unsigned* bar;                     // grid barrier: arrivals, generation (arrivals 0 before a launch)
};

__device__ __forceinline__ unsigned ld_acquire_gpu(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// all CTAs of the launch meet; false when this CTA's wait ran out
__device__ __forceinline__ bool coarse_grid_barrier(unsigned* bar, unsigned nblocks) {
    __shared__ int ok_s;
    __syncthreads();
    if (threadIdx.x == 0) {
        int ok = 1;
        const unsigned gen = ld_acquire_gpu(bar + 1);  // cannot advance before this CTA arrives
        __threadfence();
        if (atomicAdd(bar, 1u) == nblocks - 1) {
            atomicExch(bar, 0u);
            __threadfence();
            atomicAdd(bar + 1, 1u);
        } else {
            long long n = 0;
            while (ld_acquire_gpu(bar + 1) == gen) {
                if (++n > kBarrierPolls) {
                    ok = 0;
                    break;
                }
                if (n > 4096) __nanosleep(100);  // a tight poll first: the others are usually close
            }
        }
        __threadfence();
        ok_s = ok;
    }
    __syncthreads();
    return ok_s != 0;
}

__global__ void __launch_bounds__(kCycleThreads, 1) mg_coarse_cycle_kernel(const __grid_constant__ CoarseCycle a,
                                                                            Scalars* s) {
    if (s->done) return;  // read by every CTA before any can change it: all leave, or none
    extern __shared__ __align__(16) unsigned char bottom_smem[];
    __shared__ float part[kCoopQuads][4][2][16];
    const unsigned nblk = gridDim.x;
    const int wg = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    const int wb = threadIdx.x >> 5, quad_b = wb >> 2, sub = wb & 3;
    const int quad = blockIdx.x * kCoopQuads + quad_b, nquads = gridDim.x * kCoopQuads;
    auto now = [] { return true; };
    auto fail = [&]() {
        if (threadIdx.x == 0) {
            s->fault = 1;
            s->bad = 1;
            s->done = 1;
        }
    };
    for (int l = a.from; l < a.pre_end; ++l) {
        const CoarseLevel& F = a.lv[l];
        const CoarseLevel& C = a.lv[l + 1];
        smooth_segments<float, float4, SM_ZERO2, DOT_NONE, true>(F.g, F.seg, F.rec, F.b, nullptr, F.g, nullptr, F.x, nullptr,
                                                                 wg, nw, now);
        if (!coarse_grid_barrier(a.bar, nblk)) return fail();
        restrict_quad_segments<float, float4, false, true>(F.g, F.rec, F.b, F.x, C.g, C.seg, C.b, nullptr, nullptr, part, quad, nquads,
                                                    quad_b, sub, now);
        if (!coarse_grid_barrier(a.bar, nblk)) return fail();
    }
    if (blockIdx.x == 0) {
        const CoarseLevel& F = a.lv[a.pre_end];
        const CoarseLevel& C = a.lv[a.pre_end + 1];
        bottom_cycle<4>(F.g, F.rec, F.b, F.x, C.g, C.rec, bottom_smem, now);
    }
    for (int l = a.pre_end - 1; l >= a.from; --l) {
        const CoarseLevel& F = a.lv[l];
        const CoarseLevel& C = a.lv[l + 1];
        if (!coarse_grid_barrier(a.bar, nblk)) return fail();
        smooth_segments<float, float4, SM_PROLONG, DOT_NONE, true>(F.g, F.seg, F.rec, F.b, F.x, C.g, C.x, F.t, nullptr, wg,
                                                                   nw, now);
        if (!coarse_grid_barrier(a.bar, nblk)) return fail();
        smooth_segments<float, float4, SM_PLAIN, DOT_NONE, true>(F.g, F.seg, F.rec, F.b, F.t, F.g, nullptr, F.x, nullptr, wg,
                                                                 nw, now);
    }
}

// ---------------------------------------------------------------------------------------
// host side

static int seg_blocks(el_ctx* ctx, long long total_segments) {
    const long long warps = (long long)ctx->num_sms * ctx->seg_per_sm * (kSegThreads / 32);
    const long long need = std::max<long long>(1, std::min<long long>(total_segments, warps));
    return (int)((need * 32 + kSegThreads - 1) / kSegThreads);
}

// Blocks of a PCG kernel of kDotThreads<V>: one wave at most, and the tuned warps per SM.
template <typename V, typename... KArgs>
static int dot_blocks(el_ctx* ctx, void (*kernel)(KArgs...), long long total_segments) {
    const long long warps = (long long)ctx->num_sms * ctx->seg_per_sm * (kSegThreads / 32);
    const long long need = std::max<long long>(1, std::min<long long>(total_segments, warps));
    return one_wave(ctx, kernel, kDotThreads<V>, (int)((need * 32 + kDotThreads<V> - 1) / kDotThreads<V>));
}

static SegArg seg_arg(const SegList& l) { return SegArg{l.desc, l.count}; }

// Cells a segment kernel of multigrid level `level` visits (for the byte counts of profiled
// launches): the active segments' cells, as read back by record_active(), else `full`.
static double active_cells(const el_ctx* ctx, int level, double full) {
    if (level >= 0 && level < (int)ctx->prof_active.size() && ctx->prof_active[level] >= 0)
        return ctx->prof_active[level];
    return full;
}

// While profiling, reads back the active segment counts of the finest level (seg0) and of the
// coarse levels (one synchronisation per solve; not used outside profiling).
template <typename V>
static int record_active(el_ctx* ctx, const SegList& seg0, int n0, const std::vector<MGLevel<V>>* mg) {
    ctx->prof_active.clear();
    if (!ctx->prof_mask) return EL_OK;
    const size_t levels = mg ? mg->size() : 1;
    std::vector<int> counts(levels, 0);
    for (size_t l = 0; l < levels; ++l) {
        const int* c = l == 0 ? seg0.count : (*mg)[l].seg.count;
        EL_CUDA_TRY(ctx, cudaMemcpyAsync(&counts[l], c, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    }
    EL_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    for (size_t l = 0; l < levels; ++l) {
        const int w = l == 0 ? n0 : (*mg)[l].n0;
        ctx->prof_active.push_back((double)counts[l] * std::min(32, w));
    }
    return EL_OK;
}

static int alloc_seglist(el_ctx* ctx, SegList& l, int n0, int n1, int n2) {
    l.nsr = (n0 + 31) / 32;
    l.total = (long long)l.nsr * n1 * n2;
    const long long nchunks = (l.total + kSegChunk - 1) / kSegChunk;
    l.desc = (int4*)ctx_alloc(ctx, l.total * sizeof(int4));
    l.flags = (uint8_t*)ctx_alloc(ctx, l.total);
    l.chunk = (int*)ctx_alloc(ctx, (nchunks + 1) * sizeof(int));
    l.count = l.chunk + nchunks;
    return (l.desc && l.flags && l.chunk) ? EL_OK : set_error(ctx, EL_ERR_OUT_OF_MEMORY, "segment lists");
}

// compaction of the flags into the ordered id list
static int enqueue_compact(el_ctx* ctx, SegList& l, const LGeom& g) {
    const int nchunks = (int)((l.total + kSegChunk - 1) / kSegChunk);
    const bool direct = l.total <= kSegDirect;
    if (!direct)
        launch_dependent(ctx, seg_count_kernel, dim3(nchunks), dim3(256), 0, (const uint8_t*)l.flags, l.total, l.chunk);
    launch_dependent(ctx, seg_write_kernel, dim3(nchunks), dim3(256), 0, g, (const uint8_t*)l.flags, l.total,
                     direct ? (const int*)nullptr : (const int*)l.chunk, l.desc, l.count);
    return direct ? 1 : 2;
}

static int grid1d(el_ctx* ctx, long long n) {
    return (int)std::max<long long>(1, std::min<long long>((n + 255) / 256, (long long)ctx->num_sms * ctx->stencil_per_sm));
}

// Hierarchy below the finest level (allocated once per context and solver precision).
template <typename V>
static int build_hierarchy(el_ctx* ctx, std::vector<MGLevel<V>>& mg, size_t coarse_rec_bytes) {
    mg.clear();
    MGLevel<V> L0;
    L0.n0 = ctx->ni;
    L0.n1 = ctx->nj;
    L0.n2 = ctx->nk;
    const long long n = (long long)ctx->ni * ctx->nj * ctx->nk;
    L0.t = (V*)ctx_alloc(ctx, n * sizeof(V));
    if (sizeof(V) == 8) L0.rd = (V*)ctx_alloc(ctx, n * sizeof(V));
    if (!L0.t || (sizeof(V) == 8 && !L0.rd)) return set_error(ctx, EL_ERR_OUT_OF_MEMORY, "multigrid");
    mg.push_back(L0);
    while (std::max(mg.back().n0, std::max(mg.back().n1, mg.back().n2)) > kCoarsestMaxDim) {
        MGLevel<V> C;
        C.n0 = (mg.back().n0 + 1) / 2;
        C.n1 = (mg.back().n1 + 1) / 2;
        C.n2 = (mg.back().n2 + 1) / 2;
        const long long m = (long long)C.n0 * C.n1 * C.n2;
        C.rec = ctx_alloc(ctx, m * coarse_rec_bytes);
        C.b = (V*)ctx_alloc(ctx, m * sizeof(V));
        C.x = (V*)ctx_alloc(ctx, m * sizeof(V));
        C.t = (V*)ctx_alloc(ctx, m * sizeof(V));
        if (sizeof(V) == 8) C.rd = (V*)ctx_alloc(ctx, m * sizeof(V));
        if (!C.rec || !C.b || !C.x || !C.t || (sizeof(V) == 8 && !C.rd)) return set_error(ctx, EL_ERR_OUT_OF_MEMORY, "multigrid");
        int rc = alloc_seglist(ctx, C.seg, C.n0, C.n1, C.n2);
        if (rc != EL_OK) return rc;
        mg.push_back(C);
    }
    return EL_OK;
}

// Coarse records and segment lists of every level below the finest.
template <typename V, typename R0, typename RC>
static int enqueue_coarsen(el_ctx* ctx, std::vector<MGLevel<V>>& mg) {
    int launched = 0;
    for (size_t l = 0; l + 1 < mg.size(); ++l) {
        const MGLevel<V>& F = mg[l];
        MGLevel<V>& C = mg[l + 1];
        const LGeom gf = make_geom(F.n0, F.n1, F.n2), gc = make_geom(C.n0, C.n1, C.n2);
        dim3 block(32, 4, 1);
        dim3 grid((C.n0 + 31) / 32, (C.n1 + 3) / 4, C.n2);
        {
            ProfScope prof(ctx, EL_KC_MG_COARSE, (double)F.n0 * F.n1 * F.n2 * (l == 0 ? sizeof(R0) : sizeof(RC)) +
                                                     (double)C.n0 * C.n1 * C.n2 * sizeof(RC));
            if (l == 0)
                launch_dependent(ctx, coarsen_kernel<R0, RC>, grid, block, 0, gf, (const R0*)F.rec, gc, (RC*)C.rec,
                                 (double*)C.rd, C.seg.flags);
            else
                launch_dependent(ctx, coarsen_kernel<RC, RC>, grid, block, 0, gf, (const RC*)F.rec, gc, (RC*)C.rec,
                                 (double*)C.rd, C.seg.flags);
        }
        ProfScope prof(ctx, EL_KC_OTHER, (double)C.seg.total * 17);  // flags read, descriptors written
        launched += 1 + enqueue_compact(ctx, C.seg, gc);
    }
    return launched;
}

template <typename V, typename R, int MODE, int DOT>
static void launch_smooth(el_ctx* ctx, const MGLevel<V>& F, const SegList& seg, const V* x_in, const MGLevel<V>* C,
                          V* x_out, Scalars* s) {
    const LGeom g = make_geom(F.n0, F.n1, F.n2);
    const LGeom gc = C ? make_geom(C->n0, C->n1, C->n2) : g;
    const int blocks = one_wave(ctx, smooth_kernel<V, R, MODE, DOT>, kSegThreads, seg_blocks(ctx, seg.total));
    launch_dependent(ctx, smooth_kernel<V, R, MODE, DOT>, dim3(blocks), dim3(kSegThreads), 0, g,
                     seg_arg(seg), (const R*)F.rec, (const V*)F.b, x_in, gc, C ? (const V*)C->x : (const V*)nullptr,
                     x_out, (const V*)F.rd, s, ctx->partials, ctx->counter);
}

// The coarse part of an FP32 V-cycle, levels [from, pre_end) and the bottom pair, as one
// cooperative launch of mg_coarse_cycle_kernel; the grid is one CTA per 32 rows of level
// `from` (a warp per row segment), at most every resident CTA.
static bool coarse_fused_usable(const el_ctx* ctx, int L) {
    return ctx->coarse_fused && ctx->coarse_per_sm > 0 && ctx->coarse_bar && L <= kCoarseMaxLevels;
}

static int coarse_cycle_grid(const el_ctx* ctx, const SegList& seg_from) {
    const long long cap = (long long)ctx->num_sms * ctx->coarse_per_sm;
    const long long want = (seg_from.total + kCycleThreads / 32 - 1) / (kCycleThreads / 32);
    return (int)std::max<long long>(1, std::min(cap, want));
}

static int launch_coarse_cycle(el_ctx* ctx, std::vector<MGLevel<float>>& mg, int from, int pre_end, Scalars* s) {
    CoarseCycle a{};
    for (int l = from; l <= pre_end + 1; ++l) {
        const MGLevel<float>& X = mg[l];
        a.lv[l] = CoarseLevel{make_geom(X.n0, X.n1, X.n2), (const float4*)X.rec, X.b, X.x, X.t, seg_arg(X.seg)};
    }
    a.from = from;
    a.pre_end = pre_end;
    a.bar = ctx->coarse_bar;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(coarse_cycle_grid(ctx, mg[from].seg), 1, 1);
    cfg.blockDim = dim3(kCycleThreads, 1, 1);
    cfg.dynamicSmemBytes = (int)sizeof(BottomSmem);
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, mg_coarse_cycle_kernel, a, s);
    return 1;
}

// z = M^-1 r with r = mg[0].b and z = mg[0].x; dot = DOT_INIT or DOT_BETA.  R0 / RC are the
// record types of the finest / coarse levels.  from > 0: the levels below `from` only (level
// from - 1 restricted onto mg[from].b before, and prolonged from mg[from].x after, by the caller).
// smoothed: the finest level's two sweeps from zero are in mg[0].x already.
template <typename V, typename R0, typename RC>
static int enqueue_vcycle(el_ctx* ctx, std::vector<MGLevel<V>>& mg, const SegList& seg0, Scalars* s, int dot,
                          int from = 0, bool smoothed = false) {
    int launched = 0;
    const int L = (int)mg.size();
    auto segof = [&](int l) -> const SegList& { return l == 0 ? seg0 : mg[l].seg; };
    auto cells = [](const MGLevel<V>& X) { return (double)X.n0 * X.n1 * X.n2; };
    auto act = [&](int l, const MGLevel<V>& X) { return active_cells(ctx, l, cells(X)); };
    const double vs = sizeof(V);
    if (L == 1) {
        // too small to coarsen: the coarsest sweeps solve it, one more sweep gives the dot
        MGLevel<V>& C = mg[0];
        launch_dependent(ctx, coarsest_kernel<V, R0>, dim3(1), dim3(kCoarsestMaxCells), 0, make_geom(C.n0, C.n1, C.n2),
                         (const R0*)C.rec, (const V*)C.b, C.t, (const V*)C.rd, (int)kCoarsestSweeps, (const Scalars*)s);
        if (dot == DOT_INIT)
            launch_smooth<V, R0, SM_PLAIN, DOT_INIT>(ctx, C, seg0, C.t, nullptr, C.x, s);
        else
            launch_smooth<V, R0, SM_PLAIN, DOT_BETA>(ctx, C, seg0, C.t, nullptr, C.x, s);
        return 2;
    }
    // the FP32 hierarchy's last two levels in one CTA (mg_bottom_kernel)
    constexpr bool kBottomType = std::is_same<V, float>::value && std::is_same<RC, float4>::value;
    const bool fused_bottom = kBottomType && L >= 3 && mg[L - 2].n0 <= kBottomDim && mg[L - 2].n1 <= kBottomDim &&
                              mg[L - 2].n2 <= kBottomDim && mg[L - 1].n0 <= 8 && mg[L - 1].n1 <= 8 &&
                              mg[L - 1].n2 <= 8;
    const int pre_end = fused_bottom ? L - 2 : L - 1;  // levels smoothed and restricted by the loops
    // levels [coop_from, pre_end) and the bottom in one cooperative launch (the FP32 hierarchy)
    int coop_from = -1;
    if constexpr (kBottomType)
        if (fused_bottom && coarse_fused_usable(ctx, L)) {
            // coarse_fused = 1: every level below the finest; 2: from the second one on (the
            // first, the largest, keeps its launches)
            const int c = std::max(from, ctx->coarse_fused);
            if (c < pre_end) coop_from = c;
        }
    const int down_end = coop_from >= 0 ? coop_from : pre_end;  // levels by per-level launches
    for (int l = from; l < down_end; ++l) {
        MGLevel<V>& F = mg[l];
        MGLevel<V>& C = mg[l + 1];
        const double rb = l == 0 ? sizeof(R0) : sizeof(RC);
        if (l > 0 || !smoothed) {
            // reads b and records (FP64: t and rd); writes x
            ProfScope prof(ctx, l == 0 ? EL_KC_SMOOTH : EL_KC_MG_COARSE, act(l, F) * ((vs == 8 ? 4 : 2) * vs + rb));
            // the two sweeps from zero; FP64: the first is in t already
            constexpr int mode = sizeof(V) == 8 ? SM_PLAIN : SM_ZERO2;
            const V* first = sizeof(V) == 8 ? F.t : nullptr;
            if (l == 0)
                launch_smooth<V, R0, mode, DOT_NONE>(ctx, F, segof(l), first, nullptr, F.x, s);
            else
                launch_smooth<V, RC, mode, DOT_NONE>(ctx, F, segof(l), first, nullptr, F.x, s);
            ++launched;
        }
        {
            // reads b, x and records; writes the coarse b
            ProfScope prof(ctx, l == 0 ? EL_KC_RESTRICT : EL_KC_MG_COARSE, act(l, F) * (2 * vs + rb) + act(l + 1, C) * vs);
            const LGeom gf = make_geom(F.n0, F.n1, F.n2), gc = make_geom(C.n0, C.n1, C.n2);
            auto quads = [&](auto kernel, const auto* rec) {
                const int blocks = one_wave(ctx, kernel, kSegThreads, seg_blocks(ctx, 4 * C.seg.total));
                launch_dependent(ctx, kernel, dim3(blocks), dim3(kSegThreads), 0, gf, rec, (const V*)F.b, (const V*)F.x,
                                 gc, seg_arg(C.seg), C.b, C.t, (const V*)C.rd, (const Scalars*)s);
            };
            if (l > 0)
                quads(restrict_quad_kernel<V, RC, false>, (const RC*)F.rec);
            else
                quads(restrict_quad_kernel<V, R0, true>, (const R0*)F.rec);
        }
        ++launched;
    }
    if (coop_from >= 0) {
        if constexpr (kBottomType) {
            // reads and writes what the per-level launches and the bottom would
            double bytes = cells(mg[L - 2]) * (sizeof(RC) + 2 * vs) + cells(mg[L - 1]) * sizeof(RC);
            for (int l = coop_from; l < pre_end; ++l)
                bytes += act(l, mg[l]) * (2 * (2 * vs + sizeof(RC)) + 2 * (3 * vs + sizeof(RC))) +
                         act(l + 1, mg[l + 1]) * 2 * vs;
            ProfScope prof(ctx, EL_KC_MG_COARSE, bytes);
            launched += launch_coarse_cycle(ctx, mg, coop_from, pre_end, s);
        }
    } else if (fused_bottom) {
        if constexpr (kBottomType) {
            MGLevel<V>& F = mg[L - 2];
            MGLevel<V>& C = mg[L - 1];
            // reads the level's records and b and the coarsest records; writes the level's x
            ProfScope prof(ctx, EL_KC_MG_COARSE, cells(F) * (sizeof(RC) + 2 * vs) + cells(C) * sizeof(RC));
            launch_dependent(ctx, mg_bottom_kernel, dim3(1), dim3(kBottomThreads), (int)sizeof(BottomSmem),
                             make_geom(F.n0, F.n1, F.n2), (const float4*)F.rec, (const float*)F.b, F.x,
                             make_geom(C.n0, C.n1, C.n2), (const float4*)C.rec, (const Scalars*)s);
            ++launched;
        }
    } else {
        MGLevel<V>& C = mg[L - 1];
        ProfScope prof(ctx, EL_KC_MG_COARSE, cells(C) * (3 * vs + sizeof(RC)));
        launch_dependent(ctx, coarsest_kernel<V, RC>, dim3(1), dim3(kCoarsestMaxCells), 0, make_geom(C.n0, C.n1, C.n2),
                         (const RC*)C.rec, (const V*)C.b, C.x, (const V*)C.rd, (int)kCoarsestSweeps, (const Scalars*)s);
        ++launched;
    }
    for (int l = down_end - 1; l >= from; --l) {
        MGLevel<V>& F = mg[l];
        MGLevel<V>& C = mg[l + 1];
        const double rb = l == 0 ? sizeof(R0) : sizeof(RC);
        const int cls = l == 0 ? EL_KC_SMOOTH : EL_KC_MG_COARSE;
        {
            // prolongation sweep: b, x, records, coarse x read, t written
            ProfScope prof(ctx, cls, act(l, F) * (3 * vs + rb) + act(l + 1, C) * vs);
            if (l == 0)
                launch_smooth<V, R0, SM_PROLONG, DOT_NONE>(ctx, F, segof(l), F.x, &C, F.t, s);
            else
                launch_smooth<V, RC, SM_PROLONG, DOT_NONE>(ctx, F, segof(l), F.x, &C, F.t, s);
        }
        {
            // last sweep: b, t, records read, x written
            ProfScope prof(ctx, cls, act(l, F) * (3 * vs + rb));
            if (l == 0 && dot == DOT_INIT)
                launch_smooth<V, R0, SM_PLAIN, DOT_INIT>(ctx, F, segof(l), F.t, nullptr, F.x, s);
            else if (l == 0)
                launch_smooth<V, R0, SM_PLAIN, DOT_BETA>(ctx, F, segof(l), F.t, nullptr, F.x, s);
            else
                launch_smooth<V, RC, SM_PLAIN, DOT_NONE>(ctx, F, segof(l), F.t, nullptr, F.x, s);
        }
        launched += 2;
    }
    return launched;
}

// The finest level of the FP32 V-cycle by the tile kernels (el_march.cu), from the pre-smoothed
// level on: restriction, the coarse levels (the segment kernels), prolongation sweep, last sweep
// with the dot product (dot = DOT_INIT or DOT_BETA).
static int enqueue_march_vcycle_rest(el_ctx* ctx, std::vector<MGLevel<float>>& mg, Scalars* s, int dot) {
    MGLevel<float>& F = mg[0];
    MGLevel<float>& C = mg[1];
    const double na = active_cells(ctx, 0, (double)F.n0 * F.n1 * F.n2);
    const double nc = active_cells(ctx, 1, (double)C.n0 * C.n1 * C.n2);
    int n = 0;
    {
        // reads x, b and half4 records; writes the coarse b
        ProfScope prof(ctx, EL_KC_RESTRICT, na * 16 + nc * 4);
        n += march_restrict(ctx, F.x, F.b, C.b, s);
    }
    n += enqueue_vcycle<float, ushort4, float4>(ctx, mg, ctx->seg0, s, DOT_NONE, 1);
    {
        // reads x, b, records and the coarse x; writes t
        ProfScope prof(ctx, EL_KC_SMOOTH, na * 20 + nc * 4);
        n += march_prolong(ctx, F.x, F.b, F.t, s);
    }
    {
        // reads t, b, records; writes x
        ProfScope prof(ctx, EL_KC_SMOOTH, na * 20);
        n += march_last(ctx, F.t, F.b, F.x, s, dot);
    }
    return n;
}

// z = M^-1 r by the tile kernels on the finest level (the V-cycle that opens a refinement sweep)
static int enqueue_march_vcycle(el_ctx* ctx, std::vector<MGLevel<float>>& mg, Scalars* s, int dot) {
    const double na = active_cells(ctx, 0, (double)mg[0].n0 * mg[0].n1 * mg[0].n2);
    int n = 0;
    {
        // reads b and records; writes x
        ProfScope prof(ctx, EL_KC_SMOOTH, na * 16);
        n += march_zero2(ctx, mg[0].b, mg[0].x, s);
    }
    return n + enqueue_march_vcycle_rest(ctx, mg, s, dot);
}

// One PCG iteration of the mixed solver's inner system with the finest level on the tile
// kernels: K1 (direction, A p, alpha), then the update fused with the pre-smoother (x, r out of
// place, |r|^2, z's first two sweeps), then the rest of the V-cycle.  The direction and the
// residual each alternate between two buffers; mg[0].b follows r.
static int enqueue_march_iteration(el_ctx* ctx, float*& p, float*& p_alt, float*& r, float*& r_alt, Scalars* s,
                                   int first, std::vector<MGLevel<float>>& mg) {
    const double na = active_cells(ctx, 0, (double)ctx->ni * ctx->nj * ctx->nk);
    int n = 0;
    {
        // reads z, p (not on the first iteration), float4 records; writes p, Ap
        ProfScope prof(ctx, EL_KC_DIR_SPMV, na * (4.0 * (first ? 3 : 4) + 16));
        n += march_dir_spmv(ctx, ctx->z32, p, p_alt, ctx->ap32, s, first);
    }
    std::swap(p, p_alt);
    {
        // reads r, Ap, x, p, half4 records; writes x, r, z
        ProfScope prof(ctx, EL_KC_UPDATE, na * 36);
        n += march_update_smooth(ctx, ctx->x32, p, r, r_alt, ctx->ap32, ctx->z32, s);
    }
    std::swap(r, r_alt);
    mg[0].b = r;
    return n + enqueue_march_vcycle_rest(ctx, mg, s, DOT_BETA);
}

static int poll(el_ctx* ctx, Scalars* host_copy, int which) {
    EL_CUDA_TRY(ctx, cudaMemcpyAsync(host_copy, ctx->dscal + which, sizeof(Scalars), cudaMemcpyDeviceToHost,
                                     ctx->stream));
    EL_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
    return EL_OK;
}

// One PCG iteration of a multigrid-preconditioned solve (record operator A).  The direction alternates
// between two buffers, in FP32 the residual too (mg[0].b follows it).
template <typename V, typename RA, typename R0, typename RC>
static int enqueue_mg_iteration(el_ctx* ctx, const RA* A, V* x, V*& r, V*& r_alt, V* z, V*& p, V*& p_alt, V* ap,
                                Scalars* s, int first, std::vector<MGLevel<V>>& mg) {
    const LGeom g = make_geom(ctx->ni, ctx->nj, ctx->nk);
    const SegList& seg = ctx->seg0;
    const double N = active_cells(ctx, 0, (double)ctx->ni * ctx->nj * ctx->nk), vs = sizeof(V);
    {
        // reads z, p (not on the first iteration), records; writes p, Ap
        ProfScope prof(ctx, EL_KC_DIR_SPMV, N * (vs * (first ? 3 : 4) + sizeof(RA)));
        auto kernel = dir_spmv_rec_kernel<V, RA>;
        launch_dependent(ctx, kernel, dim3(dot_blocks<V>(ctx, kernel, seg.total)), dim3(kDotThreads<V>), 0, g,
                         seg_arg(seg), A, (const V*)z, (const V*)p, p_alt, ap, s, first, ctx->partials,
                         ctx->counter);
    }
    std::swap(p, p_alt);
    if constexpr (sizeof(V) == 4) {
        // (while kernel classes are timed, the update and the sweeps go as the kernels of their classes)
        if (mg.size() > 1 && seg.total <= 128ll * ctx->num_sms && ctx->prof_mask == 0) {
            auto kernel = update_smooth_kernel<R0>;
            launch_dependent(ctx, kernel, dim3(dot_blocks<V>(ctx, kernel, seg.total)), dim3(kDotThreads<V>), 0, g,
                             seg_arg(seg), (const R0*)mg[0].rec, x, (const V*)r, r_alt, (const V*)p, (const V*)ap, z, s,
                             ctx->partials, ctx->counter);
            std::swap(r, r_alt);
            mg[0].b = r;
            return 2 + enqueue_vcycle<V, R0, RC>(ctx, mg, seg, s, DOT_BETA, 0, true);
        }
    }
    {
        // reads x, r, p, Ap; writes x, r
        ProfScope prof(ctx, EL_KC_UPDATE, N * vs * 6);
        auto kernel = update_kernel<V>;
        launch_dependent(ctx, kernel, dim3(dot_blocks<V>(ctx, kernel, seg.total)), dim3(kDotThreads<V>), 0, g,
                         seg_arg(seg), x, r, (const V*)p, (const V*)ap, mg[0].t, (const V*)mg[0].rd, s, ctx->partials,
                         ctx->counter);
    }
    return 2 + enqueue_vcycle<V, R0, RC>(ctx, mg, seg, s, DOT_BETA);
}

// One iteration of the plain FP64 PCG.  pending: the update before it left its dot products as
// partials; last: they are summed after this one (the end of a batch).  The slot of rz follows the
// direction buffers, which alternate every iteration.
template <typename OT>
static int enqueue_jacobi_iteration(el_ctx* ctx, const SplitOp<OT>& A, double*& p, double*& p_alt, Scalars* s,
                                    int first, bool pending, bool last) {
    const LGeom g = make_geom(ctx->ni, ctx->nj, ctx->nk);
    const SegList& seg = ctx->seg0;
    const double N = active_cells(ctx, 0, (double)ctx->ni * ctx->nj * ctx->nk);
    const int slot = p == ctx->p64 ? 0 : 1;
    JacPart part;
    const long long want = (seg.total * 32 + kJacThreads - 1) / kJacThreads;  // a warp a segment
    part.blocks = (int)std::max<long long>(1, std::min<long long>(want, std::min(ctx->num_sms, kJacMaxBlocks)));
    part.pap = ctx->partials;
    part.rr = ctx->partials + kJacMaxBlocks;
    {
        // reads z, p (not on the first iteration), diag, 3 couplings; writes p, Ap
        ProfScope prof(ctx, EL_KC_DIR_SPMV, N * (8.0 * (first ? 4 : 5) + 3 * sizeof(OT)));
        launch_dependent(ctx, jacobi_dir_kernel<OT>, dim3(part.blocks), dim3(kJacThreads), 0, g, seg_arg(seg), A,
                         (const double*)ctx->z64, (const double*)p, p_alt, ctx->ap64, s, first, (int)pending, slot,
                         part);
    }
    std::swap(p, p_alt);
    {
        // reads x, r, p, Ap, the reciprocal diagonal; writes x, r, z
        ProfScope prof(ctx, EL_KC_UPDATE, N * 8.0 * 8);
        launch_dependent(ctx, jacobi_update_kernel, dim3(part.blocks), dim3(kJacThreads), 0, g, seg_arg(seg),
                         (const double*)ctx->inv64, ctx->x64, ctx->r64, ctx->z64, (const double*)p,
                         (const double*)ctx->ap64, s, slot, part);
    }
    if (!last) return 2;
    ProfScope prof(ctx, EL_KC_OTHER, 0);
    launch_dependent(ctx, jacobi_check_kernel, dim3(1), dim3(64), 0, s, slot, part);
    return 3;
}

// Launch PCG iterations (check_every per poll) until converged or `budget` are launched.
//
// The first iteration is launched directly; the following ones in batches of `check_every`
// (rounded up to even, so the two direction buffers are back in place after a batch).  A batch
// is captured once per context and solver as a CUDA graph and replayed afterwards: all its
// pointers and launch shapes are fixed per context, and the kernels read everything that
// changes (scalars, segment lists) from device memory.  While kernel classes are being
// profiled the batches are launched directly instead.
template <typename F>
static int run_iterations(el_ctx* ctx, int solver, int which, int budget, int check_every, Scalars* out,
                          F&& enqueue) {
    int launched_iters = 0;
    int st = poll(ctx, out, which);
    if (st != EL_OK) return st;
    if (out->done || budget <= 0) return EL_OK;
    // enqueue(first, position in the batch, last of the batch)
    ctx->launches += enqueue(1, 0, true);
    launched_iters = 1;
    const int batch = std::max(2, (check_every + 1) / 2 * 2);
    const bool graphs = ctx->use_graphs && ctx->prof_mask == 0;
    if (graphs && ctx->iter_graph[solver] && ctx->iter_graph_len[solver] != batch) {
        cudaGraphExecDestroy(ctx->iter_graph[solver]);
        ctx->iter_graph[solver] = nullptr;
    }
    st = poll(ctx, out, which);
    if (st != EL_OK) return st;
    while (!out->done && launched_iters < budget) {
        // a full batch may run past the budget by up to batch - 1 iterations only when the
        // budget is not a multiple of it; the iteration count reported is the device's
        if (graphs && budget - launched_iters >= batch) {
            if (!ctx->iter_graph[solver]) {
                cudaGraph_t graph = nullptr;
                EL_CUDA_TRY(ctx, cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
                int n = 0;
                for (int q = 0; q < batch; ++q) n += enqueue(0, q, q + 1 == batch);
                EL_CUDA_TRY(ctx, cudaStreamEndCapture(ctx->stream, &graph));
                const cudaError_t e = cudaGraphInstantiate(&ctx->iter_graph[solver], graph, 0);
                cudaGraphDestroy(graph);
                if (e != cudaSuccess) return set_error(ctx, EL_ERR_CUDA, std::string("graph: ") + cudaGetErrorString(e));
                ctx->iter_graph_len[solver] = batch;
                ctx->iter_graph_kernels[solver] = n;
            }
            EL_CUDA_TRY(ctx, cudaGraphLaunch(ctx->iter_graph[solver], ctx->stream));
            ctx->launches += ctx->iter_graph_kernels[solver];
            launched_iters += batch;
        } else {
            const int b = std::min(batch, budget - launched_iters);
            for (int q = 0; q < b; ++q) ctx->launches += enqueue(0, q, q + 1 == b);
            launched_iters += b;
        }
        st = check_launch(ctx, "pcg iteration");
        if (st != EL_OK) return st;
        st = poll(ctx, out, which);
        if (st != EL_OK) return st;
    }
    return EL_OK;
}

template <typename T>
static SplitOp<T> split_op(el_ctx* ctx) {
    return SplitOp<T>{ctx->diag64, (const T*)ctx->off[0], (const T*)ctx->off[1], (const T*)ctx->off[2]};
}

static void reset_vectors(el_ctx* ctx) {
    const size_t n = (size_t)ctx->ni * ctx->nj * ctx->nk;
    for (double* v : {ctx->x64, ctx->r64, ctx->z64, ctx->p64, ctx->p64b, ctx->ap64})
        if (v) cudaMemsetAsync(v, 0, n * 8, ctx->stream);
    for (float* v : {ctx->x32, ctx->r32, ctx->r32b, ctx->z32, ctx->p32, ctx->p32b, ctx->ap32})
        if (v) cudaMemsetAsync(v, 0, n * 4, ctx->stream);
    if (ctx->xs) cudaMemsetAsync(ctx->xs, 0, n * 8, ctx->stream);
    for (auto& L : ctx->mg32) {
        const size_t m = (size_t)L.n0 * L.n1 * L.n2 * 4;
        for (float* v : {L.t, L.rec ? L.b : nullptr, L.rec ? L.x : nullptr})
            if (v) cudaMemsetAsync(v, 0, m, ctx->stream);
    }
    for (auto& L : ctx->mg64) {
        const size_t m = (size_t)L.n0 * L.n1 * L.n2 * 8;
        for (double* v : {L.t, L.rec ? L.b : nullptr, L.rec ? L.x : nullptr})
            if (v) cudaMemsetAsync(v, 0, m, ctx->stream);
    }
}

// mg[0].b follows the residual buffer during a solve; between solves it is r32 again
static void mg_restore_pointers(el_ctx* ctx) {
    if (!ctx->mg32.empty()) ctx->mg32[0].b = ctx->r32;
}

// The float pair of the iterate, kept where the refinement residual is double-float: the mixed
// solver on FP32 fields (exact float couplings); null otherwise.
template <typename T>
static float2* iterate_pairs(el_ctx* ctx, int solver) {
    return (solver == EL_SOLVER_MIXED && std::is_same<T, float>::value) ? ctx->xs : nullptr;
}

// The mixed solver's refinement residual: double-float arithmetic for FP32 fields (exact float
// couplings), FP64 for FP64 fields.
template <typename T>
static void enqueue_refine_residual(el_ctx* ctx, const LGeom& g, const SplitOp<T>& A64, Scalars* s0) {
    const int nb = seg_blocks(ctx, ctx->seg0.total);
    if constexpr (std::is_same<T, float>::value)
        // the resident four CTAs per SM (its launch bounds) in one wave: 102 -> 94 us at 256^3
        residual_df_kernel<<<std::min(nb, ctx->num_sms * 4), kSegThreads, 0, ctx->stream>>>(
            g, seg_arg(ctx->seg0), A64, ctx->rhs64, ctx->x64, ctx->xs, ctx->r64, s0, ctx->partials, ctx->counter);
    else
        residual_kernel<T><<<nb, kSegThreads, 0, ctx->stream>>>(g, seg_arg(ctx->seg0), A64, ctx->rhs64, ctx->x64,
                                                                ctx->r64, s0, ctx->partials, ctx->counter);
}

// The end of a solve, from the scalars read back: residual, errors, status.
static int finish_solve(el_ctx* ctx, const Scalars* h, el_solve_stats* st) {
    st->relres = h->bb > 0 ? sqrt(h->rr / h->bb) : 0.0;
    if (h->bad) {
        // entries outside the active segments are never rewritten and must stay finite (they
        // meet zero couplings), so a failed solve leaves every solver vector cleared
        reset_vectors(ctx);
        if (h->fault) return set_error(ctx, EL_ERR_TIMEOUT, "a bounded wait of the pressure solve gave up");
        return set_error(ctx, EL_ERR_NAN, "non-finite value in the pressure solve");
    }
    st->status = h->done ? EL_OK : EL_ERR_NOT_CONVERGED;
    return EL_OK;
}

// Solve A x64 = rhs64 (matrix already built, s0.bb set).  Fills stats.
template <typename T>
static int solve_t(el_ctx* ctx, const el_solve_params& prm, el_solve_stats* st) {
    const long long n = (long long)ctx->ni * ctx->nj * ctx->nk;
    const LGeom g = make_geom(ctx->ni, ctx->nj, ctx->nk);
    const int check = std::max(1, prm.check_every);
    Scalars* s0 = ctx->dscal;
    Scalars* h = ctx->hscal;
    const SplitOp<T> A64 = split_op<T>(ctx);
    // active segments of the finest level
    {
        ProfScope prof(ctx, EL_KC_OTHER, (double)n * 8);
        seg_flags_diag_kernel<<<seg_blocks(ctx, ctx->seg0.total), kSegThreads, 0, ctx->stream>>>(
            g, ctx->diag64, ctx->seg0.total, ctx->seg0.flags);
    }
    ctx->launches += 1 + enqueue_compact(ctx, ctx->seg0, g);
    int rc = record_active<double>(ctx, ctx->seg0, ctx->ni, nullptr);
    if (rc != EL_OK) return rc;
    const double na = active_cells(ctx, 0, (double)n);
    {
        ProfScope prof(ctx, EL_KC_OTHER, na * 24);
        solve_init_kernel<<<seg_blocks(ctx, ctx->seg0.total), kSegThreads, 0, ctx->stream>>>(
            g, seg_arg(ctx->seg0), ctx->rhs64, ctx->x64, iterate_pairs<T>(ctx, prm.solver), ctx->r64, s0, prm.tol);
    }
    ctx->launches += 1;
    if (prm.initial_guess) {
        ProfScope prof(ctx, EL_KC_OTHER, na * 56);
        const int nb = seg_blocks(ctx, ctx->seg0.total);
        guess_load_kernel<T><<<nb, kSegThreads, 0, ctx->stream>>>(g, seg_arg(ctx->seg0),
                                                                  (const T*)ctx->field[EL_FIELD_PRESSURE], ctx->diag64,
                                                                  ctx->x64);
        residual_kernel<T><<<nb, kSegThreads, 0, ctx->stream>>>(g, seg_arg(ctx->seg0), A64, ctx->rhs64, ctx->x64,
                                                                ctx->r64, s0, ctx->partials, ctx->counter);
        guess_alpha_kernel<<<nb, kSegThreads, 0, ctx->stream>>>(g, seg_arg(ctx->seg0), ctx->x64, ctx->rhs64, ctx->r64,
                                                                s0, ctx->partials, ctx->counter);
        guess_scale_kernel<<<nb, kSegThreads, 0, ctx->stream>>>(g, seg_arg(ctx->seg0), ctx->x64,
                                                                iterate_pairs<T>(ctx, prm.solver), ctx->rhs64,
                                                                ctx->r64, s0, ctx->partials, ctx->counter);
        ctx->launches += 4;
    }
    st->outer_iterations = 1;
    if (prm.solver == EL_SOLVER_JACOBI_FP64) {
        jacobi_start_kernel<<<seg_blocks(ctx, ctx->seg0.total), kSegThreads, 0, ctx->stream>>>(
            g, seg_arg(ctx->seg0), ctx->diag64, ctx->r64, ctx->inv64, ctx->z64, s0, ctx->partials, ctx->counter);
        ctx->launches += 1;
        double* p = ctx->p64;
        double* p_alt = ctx->p64b;
        rc = run_iterations(ctx, EL_SOLVER_JACOBI_FP64, 0, prm.max_iter, check, h,
                            [&](int first, int pos, bool last) {
                                return enqueue_jacobi_iteration<T>(ctx, A64, p, p_alt, s0, first, pos > 0, last);
                            });
        st->iterations = h->iter;
    } else if (prm.solver == EL_SOLVER_MG_FP64) {
        auto& mg = ctx->mg64;
        mg[0].rec = ctx->A64rec;
        mg[0].b = ctx->r64;
        mg[0].x = ctx->z64;
        pack64_kernel<T><<<grid1d(ctx, n), 256, 0, ctx->stream>>>(n, ctx->diag64, A64.x, A64.y, A64.z, ctx->A64rec,
                                                                  mg[0].rd);
        ctx->launches += 1 + enqueue_coarsen<double, Rec64, Rec64>(ctx, mg);
        rc = record_active(ctx, ctx->seg0, ctx->ni, &mg);
        if (rc != EL_OK) return rc;
        first_sweep_kernel<<<seg_blocks(ctx, ctx->seg0.total), kSegThreads, 0, ctx->stream>>>(
            g, seg_arg(ctx->seg0), ctx->r64, mg[0].rd, mg[0].t);
        ctx->launches += 1 + enqueue_vcycle<double, Rec64, Rec64>(ctx, mg, ctx->seg0, s0, DOT_INIT);
        double* r = ctx->r64;
        double* p = ctx->p64;
        double* p_alt = ctx->p64b;
        rc = run_iterations(ctx, EL_SOLVER_MG_FP64, 0, prm.max_iter, check, h, [&](int first, int, bool) {
            return enqueue_mg_iteration<double, Rec64, Rec64, Rec64>(ctx, ctx->A64rec, ctx->x64, r, r, ctx->z64, p,
                                                                    p_alt, ctx->ap64, s0, first, mg);
        });
        st->iterations = h->iter;
    } else {
        // mixed: FP64 refinement around FP32 multigrid PCG
        auto& mg = ctx->mg32;
        mg[0].rec = ctx->A16;
        mg[0].b = ctx->r32;
        mg[0].x = ctx->z32;
        if (!ctx->records_fresh) {
            ProfScope prof(ctx, EL_KC_OTHER, (double)n * (8 + 3 * sizeof(T) + 24));
            pack32_kernel<T><<<grid1d(ctx, n), 256, 0, ctx->stream>>>(n, ctx->diag64, A64.x, A64.y, A64.z, ctx->A32,
                                                                      ctx->A16);
            ctx->launches += 1;
        }
        ctx->launches += enqueue_coarsen<float, ushort4, float4>(ctx, mg);
        const bool march = ctx->march.on && ctx->solver_tiles;
        if (march) {
            ProfScope prof(ctx, EL_KC_OTHER, (double)n * 8);
            ctx->launches += march_enqueue_items(ctx);
        }
        // the fused coarse cycle's barrier starts clear (a failed solve may have left arrivals)
        if (ctx->coarse_bar) EL_CUDA_TRY(ctx, cudaMemsetAsync(ctx->coarse_bar, 0, 8, ctx->stream));
        rc = record_active(ctx, ctx->seg0, ctx->ni, &mg);
        if (rc != EL_OK) return rc;
        Scalars* s1 = ctx->dscal + 1;
        Scalars hi;
        rc = poll(ctx, h, 0);
        int inner_total = 0, outer = 0;
        float *p = ctx->p32, *p_alt = ctx->p32b, *r = ctx->r32, *r_alt = ctx->r32b;
        while (rc == EL_OK && !h->done && outer < std::max(1, prm.max_outer) && inner_total < prm.max_iter) {
            // every sweep starts from the same buffer assignment, so that the captured iteration
            // batches (run_iterations) see the pointers they were captured with
            p = ctx->p32;
            p_alt = ctx->p32b;
            r = ctx->r32;
            r_alt = ctx->r32b;
            mg[0].b = ctx->r32;
            {
                ProfScope prof(ctx, EL_KC_OTHER, na * 16);
                inner_init_kernel<<<seg_blocks(ctx, ctx->seg0.total), kSegThreads, 0, ctx->stream>>>(
                    g, seg_arg(ctx->seg0), ctx->r64, ctx->r32, ctx->x32, s0, s1, prm.tol, prm.inner_floor,
                    prm.max_iter - inner_total, ctx->partials, ctx->counter);
            }
            ctx->launches += 1;
            if (march)
                ctx->launches += enqueue_march_vcycle(ctx, mg, s1, DOT_INIT);
            else
                ctx->launches += enqueue_vcycle<float, ushort4, float4>(ctx, mg, ctx->seg0, s1, DOT_INIT);
            rc = run_iterations(ctx, EL_SOLVER_MIXED, 1, prm.max_iter - inner_total, check, &hi, [&](int first, int, bool) {
                if (march) return enqueue_march_iteration(ctx, p, p_alt, r, r_alt, s1, first, mg);
                return enqueue_mg_iteration<float, float4, ushort4, float4>(ctx, ctx->A32, ctx->x32, r, r_alt, ctx->z32,
                                                                            p, p_alt, ctx->ap32, s1, first, mg);
            });
            if (rc != EL_OK) break;
            inner_total += hi.iter;
            if (hi.fault) h->fault = 1;
            if (hi.bad) {
                h->bad = 1;
                break;
            }
            {
                ProfScope prof(ctx, EL_KC_OTHER, na * 20);
                accumulate_kernel<<<seg_blocks(ctx, ctx->seg0.total), kSegThreads, 0, ctx->stream>>>(
                    g, seg_arg(ctx->seg0), ctx->x64, iterate_pairs<T>(ctx, prm.solver), ctx->x32, s1, s0);
            }
            {
                // reads x, b, diag (f64), 3 couplings; writes r (f64)
                ProfScope prof(ctx, EL_KC_RESIDUAL, na * (32 + 3 * sizeof(T)));
                enqueue_refine_residual(ctx, g, A64, s0);
            }
            ctx->launches += 2;
            ++outer;
            rc = poll(ctx, h, 0);
        }
        st->iterations = inner_total;
        st->outer_iterations = outer;
    }
    mg_restore_pointers(ctx);
    if (rc != EL_OK) return rc;
    return finish_solve(ctx, h, st);
}

// ---------------------------------------------------------------------------------------
// Capture-safe mixed solve: the same kernels, with the refinement sweeps and the PCG iterations
// driven on the device by conditional WHILE nodes of a CUDA graph (no host polling), for
// steps that are captured whole.  Must be enqueued on a stream that is being captured.

// Condition of the PCG loop: not converged and the inner iteration budget not spent.
__global__ void inner_cond_kernel(cudaGraphConditionalHandle h, Scalars* so, const Scalars* si, int max_iter,
                                  int count_pass) {
    if (count_pass) so->inner_passes += 1;
    cudaGraphSetConditional(h, (!si->done && si->iter + so->inner_total < max_iter) ? 1u : 0u);
}

// Condition of the refinement loop.  count_sweep: called after a sweep (adds its iterations);
// otherwise it sets the condition for the first sweep.
__global__ void outer_cond_kernel(cudaGraphConditionalHandle h, Scalars* so, const Scalars* si, int max_outer,
                                  int max_iter, int count_sweep) {
    if (count_sweep) {
        so->outer += 1;
        so->inner_total += si->iter;
        if (si->bad) so->bad = 1;
        if (si->fault) so->fault = 1;
    }
    const bool go = !so->done && !so->bad && so->outer < max_outer && so->inner_total < max_iter;
    cudaGraphSetConditional(h, go ? 1u : 0u);
}

// A conditional handle on the graph being captured on ctx->stream.
static int new_handle(el_ctx* ctx, cudaGraphConditionalHandle* handle) {
    cudaStreamCaptureStatus cs;
    cudaGraph_t graph = nullptr;
    EL_CUDA_TRY(ctx, cudaStreamGetCaptureInfo(ctx->stream, &cs, nullptr, &graph, nullptr, nullptr, nullptr));
    if (cs != cudaStreamCaptureStatusActive) return set_error(ctx, EL_ERR_INVALID_ARGUMENT, "stream is not capturing");
    EL_CUDA_TRY(ctx, cudaGraphConditionalHandleCreate(handle, graph, 0, cudaGraphCondAssignDefault));
    return EL_OK;
}

// Adds a WHILE node on `handle` after the work captured so far on ctx->stream and redirects
// ctx->stream to the capture of its body (ended by end_while).  The condition must have been
// set by a kernel captured before this call.
static int begin_while(el_ctx* ctx, int depth, cudaGraphConditionalHandle handle, cudaStream_t* parent) {
    cudaStreamCaptureStatus cs;
    cudaGraph_t graph = nullptr;
    const cudaGraphNode_t* deps = nullptr;
    const cudaGraphEdgeData* edges = nullptr;
    size_t ndeps = 0;
    EL_CUDA_TRY(ctx, cudaStreamGetCaptureInfo(ctx->stream, &cs, nullptr, &graph, &deps, &edges, &ndeps));
    if (cs != cudaStreamCaptureStatusActive) return set_error(ctx, EL_ERR_INVALID_ARGUMENT, "stream is not capturing");
    cudaGraphNodeParams prm = {};
    prm.type = cudaGraphNodeTypeConditional;
    prm.conditional.handle = handle;
    prm.conditional.type = cudaGraphCondTypeWhile;
    prm.conditional.size = 1;
    cudaGraphNode_t node;
    EL_CUDA_TRY(ctx, cudaGraphAddNode(&node, graph, deps, edges, ndeps, &prm));
    EL_CUDA_TRY(ctx, cudaStreamUpdateCaptureDependencies(ctx->stream, &node, nullptr, 1, cudaStreamSetCaptureDependencies));
    if (!ctx->body_stream[depth]) return set_error(ctx, EL_ERR_INVALID_ARGUMENT, "loop streams not prepared");
    EL_CUDA_TRY(ctx, cudaStreamBeginCaptureToGraph(ctx->body_stream[depth], prm.conditional.phGraph_out[0], nullptr,
                                                   nullptr, 0, cudaStreamCaptureModeThreadLocal));
    *parent = ctx->stream;
    ctx->stream = ctx->body_stream[depth];
    return EL_OK;
}

static int end_while(el_ctx* ctx, cudaStream_t parent) {
    cudaGraph_t body = nullptr;
    const cudaError_t e = cudaStreamEndCapture(ctx->stream, &body);
    ctx->stream = parent;
    if (e != cudaSuccess) return set_error(ctx, EL_ERR_CUDA, std::string("loop body: ") + cudaGetErrorString(e));
    return EL_OK;
}

// The mixed solve with both loops on the device: no host polling, so it can sit inside a
// captured step.  The PCG loop runs iterations in pairs (the two direction buffers are back in
// place after each pass); the second of a pair that the budget does not cover returns at once.
template <typename T>
static int enqueue_solve_device_t(el_ctx* ctx, const el_solve_params& prm, int kernels[3]) {
    const long long n = (long long)ctx->ni * ctx->nj * ctx->nk;
    const LGeom g = make_geom(ctx->ni, ctx->nj, ctx->nk);
    Scalars* s0 = ctx->dscal;
    Scalars* s1 = ctx->dscal + 1;
    const SplitOp<T> A64 = split_op<T>(ctx);
    const int max_outer = std::max(1, prm.max_outer);
    auto& mg = ctx->mg32;
    mg[0].rec = ctx->A16;
    mg[0].b = ctx->r32;
    mg[0].x = ctx->z32;
    int nk = 0;
    seg_flags_diag_kernel<<<seg_blocks(ctx, ctx->seg0.total), kSegThreads, 0, ctx->stream>>>(
        g, ctx->diag64, ctx->seg0.total, ctx->seg0.flags);
    nk += 1 + enqueue_compact(ctx, ctx->seg0, g);
    solve_init_kernel<<<seg_blocks(ctx, ctx->seg0.total), kSegThreads, 0, ctx->stream>>>(
        g, seg_arg(ctx->seg0), ctx->rhs64, ctx->x64, iterate_pairs<T>(ctx, EL_SOLVER_MIXED), ctx->r64, s0, prm.tol);
    if (!ctx->records_fresh) {
        pack32_kernel<T><<<grid1d(ctx, n), 256, 0, ctx->stream>>>(n, ctx->diag64, A64.x, A64.y, A64.z, ctx->A32,
                                                                  ctx->A16);
        ++nk;
    }
    nk += 1 + enqueue_coarsen<float, ushort4, float4>(ctx, mg);
    const bool march = ctx->march.on && ctx->solver_tiles;
    if (march) nk += march_enqueue_items(ctx);
    if (ctx->coarse_bar) EL_CUDA_TRY(ctx, cudaMemsetAsync(ctx->coarse_bar, 0, 8, ctx->stream));
    float *p = ctx->p32, *p_alt = ctx->p32b, *r = ctx->r32, *r_alt = ctx->r32b;
    mg[0].b = ctx->r32;
    cudaGraphConditionalHandle h_outer, h_inner;
    cudaStream_t parent_outer, parent_inner;
    int rc = new_handle(ctx, &h_outer);
    if (rc != EL_OK) return rc;
    outer_cond_kernel<<<1, 1, 0, ctx->stream>>>(h_outer, s0, s1, max_outer, prm.max_iter, 0);
    rc = begin_while(ctx, 0, h_outer, &parent_outer);
    if (rc != EL_OK) return rc;
    // one refinement sweep: inner system, its PCG loop, correction and FP64 residual
    inner_init_kernel<<<seg_blocks(ctx, ctx->seg0.total), kSegThreads, 0, ctx->stream>>>(
        g, seg_arg(ctx->seg0), ctx->r64, ctx->r32, ctx->x32, s0, s1, prm.tol, prm.inner_floor, prm.max_iter,
        ctx->partials, ctx->counter);
    auto iteration = [&](int first) {
        if (march) return enqueue_march_iteration(ctx, p, p_alt, r, r_alt, s1, first, mg);
        return enqueue_mg_iteration<float, float4, ushort4, float4>(ctx, ctx->A32, ctx->x32, r, r_alt, ctx->z32, p,
                                                                   p_alt, ctx->ap32, s1, first, mg);
    };
    int body = 1 + (march ? enqueue_march_vcycle(ctx, mg, s1, DOT_INIT)
                          : enqueue_vcycle<float, ushort4, float4>(ctx, mg, ctx->seg0, s1, DOT_INIT));
    body += iteration(1);
    rc = new_handle(ctx, &h_inner);
    if (rc == EL_OK) {
        inner_cond_kernel<<<1, 1, 0, ctx->stream>>>(h_inner, s0, s1, prm.max_iter, 0);
        rc = begin_while(ctx, 1, h_inner, &parent_inner);
    }
    if (rc != EL_OK) {
        end_while(ctx, parent_outer);
        return rc;
    }
    int inner = 0;
    for (int q = 0; q < 2; ++q) inner += iteration(0);
    inner_cond_kernel<<<1, 1, 0, ctx->stream>>>(h_inner, s0, s1, prm.max_iter, 1);
    rc = end_while(ctx, parent_inner);
    accumulate_kernel<<<seg_blocks(ctx, ctx->seg0.total), kSegThreads, 0, ctx->stream>>>(
        g, seg_arg(ctx->seg0), ctx->x64, iterate_pairs<T>(ctx, EL_SOLVER_MIXED), ctx->x32, s1, s0);
    enqueue_refine_residual(ctx, g, A64, s0);
    outer_cond_kernel<<<1, 1, 0, ctx->stream>>>(h_outer, s0, s1, max_outer, prm.max_iter, 1);
    const int rc2 = end_while(ctx, parent_outer);
    mg_restore_pointers(ctx);
    if (rc != EL_OK) return rc;
    if (rc2 != EL_OK) return rc2;
    // kernels outside the loops, per refinement sweep, per pass of the PCG loop
    kernels[0] = nk + 1;
    kernels[1] = body + 1 + 2 + 1;
    kernels[2] = inner + 1;
    return check_launch(ctx, "captured solve");
}

// Streams on which the loop bodies are captured (created outside any capture).
int prepare_device_solve(el_ctx* ctx) {
    for (auto& bs : ctx->body_stream)
        if (!bs) EL_CUDA_TRY(ctx, cudaStreamCreateWithFlags(&bs, cudaStreamNonBlocking));
    return EL_OK;
}

// Enqueues (for stream capture) the mixed solve of the built system; results land in the
// device scalars (s0: converged flag, |r|^2, |b|^2, sweeps, inner iterations).
int enqueue_solve_device(el_ctx* ctx, const el_solve_params& prm, int kernels[3]) {
    if (prm.solver != EL_SOLVER_MIXED) return set_error(ctx, EL_ERR_INVALID_ARGUMENT, "captured steps use the mixed solver");
    return ctx->dtype == EL_F64 ? enqueue_solve_device_t<double>(ctx, prm, kernels)
                                : enqueue_solve_device_t<float>(ctx, prm, kernels);
}

// Whether the mixed solve runs as one graph: the second and later of a row of solves with the same
// parameters.  The host-driven solve stops the device at every poll (two a refinement sweep and one a
// batch of iterations) and starts about twenty kernels a sweep one by one; the graph does neither, but
// making it costs 0.03 to 0.25 ms, which a single solve does not earn back, so a solve whose parameters
// differ from the one before's takes the host-driven path.  75 x 62 x 53 cells:
// 0.98 -> 0.76 ms; a whole step of 48^3 0.94 -> 0.76, of 151 x 97 x 133 2.01 -> 1.88, of 256^3 6.95 -> 6.83
// (parameters that alternate -> the same from call to call).
bool solve_graph_ready(el_ctx* ctx, const el_solve_params& prm) {
    el_ctx::SolveKey key;
    key.tol = prm.tol;
    key.inner_floor = prm.inner_floor;
    key.max_iter = prm.max_iter;
    key.max_outer = prm.max_outer;
    key.records = ctx->records_fresh;
    key.valid = prm.solver == EL_SOLVER_MIXED && !prm.initial_guess && ctx->use_graphs && ctx->prof_mask == 0;
    const bool again = key.valid && key == ctx->solve_last;
    ctx->solve_last = key;
    if (!again) return false;
    if (ctx->solve_graph && ctx->solve_graph_key == key) return true;
    if (ctx->solve_graph) cudaGraphExecDestroy(ctx->solve_graph);
    ctx->solve_graph = nullptr;
    if (prepare_device_solve(ctx) != EL_OK) return false;
    cudaGraph_t graph = nullptr;
    if (cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    const int rc = enqueue_solve_device(ctx, prm, ctx->solve_graph_kernels);
    const cudaError_t e = cudaStreamEndCapture(ctx->stream, &graph);
    const bool ok = rc == EL_OK && e == cudaSuccess && cudaGraphInstantiate(&ctx->solve_graph, graph, 0) == cudaSuccess;
    if (graph) cudaGraphDestroy(graph);
    if (!ok) {
        cudaGetLastError();
        ctx->solve_graph = nullptr;
        ctx->solve_last.valid = false;
        return false;
    }
    ctx->solve_graph_key = key;
    return true;
}

// the mixed solve as the graph of solve_graph_ready(); leaves the scalars in ctx->hscal
int solve_system_graph(el_ctx* ctx, const el_solve_params&, el_solve_stats* st) {
    EL_CUDA_TRY(ctx, cudaGraphLaunch(ctx->solve_graph, ctx->stream));
    Scalars* h = ctx->hscal;
    const int rc = poll(ctx, h, 0);
    if (rc != EL_OK) return rc;
    ctx->launches += ctx->solve_graph_kernels[0] + (long long)h->outer * ctx->solve_graph_kernels[1] +
                     (long long)h->inner_passes * ctx->solve_graph_kernels[2];
    st->fluid_cells = h->count;
    st->iterations = h->inner_total;
    st->outer_iterations = h->outer;
    return finish_solve(ctx, h, st);
}

int solve_system(el_ctx* ctx, const el_solve_params& prm, el_solve_stats* st) {
    return ctx->dtype == EL_F64 ? solve_t<double>(ctx, prm, st) : solve_t<float>(ctx, prm, st);
}

int setup_solver_storage(el_ctx* ctx, int solver) {
    const long long n = (long long)ctx->ni * ctx->nj * ctx->nk;
    if (!ctx->x64) {
        ctx->x64 = (double*)ctx_alloc(ctx, n * 8);
        ctx->r64 = (double*)ctx_alloc(ctx, n * 8);
        ctx->z64 = (double*)ctx_alloc(ctx, n * 8);
        ctx->p64 = (double*)ctx_alloc(ctx, n * 8);
        ctx->p64b = (double*)ctx_alloc(ctx, n * 8);
        ctx->ap64 = (double*)ctx_alloc(ctx, n * 8);
        if (!ctx->x64 || !ctx->r64 || !ctx->z64 || !ctx->p64 || !ctx->p64b || !ctx->ap64)
            return set_error(ctx, EL_ERR_OUT_OF_MEMORY, "solver vectors");
        int rc = alloc_seglist(ctx, ctx->seg0, ctx->ni, ctx->nj, ctx->nk);
        if (rc != EL_OK) return rc;
    }
    if (solver == EL_SOLVER_JACOBI_FP64 && !ctx->inv64) {
        ctx->inv64 = (double*)ctx_alloc(ctx, n * 8);
        if (!ctx->inv64) return set_error(ctx, EL_ERR_OUT_OF_MEMORY, "reciprocal diagonal");
    }
    if (solver == EL_SOLVER_MG_FP64 && ctx->mg64.empty()) {
        ctx->A64rec = (Rec64*)ctx_alloc(ctx, n * sizeof(Rec64));
        if (!ctx->A64rec) return set_error(ctx, EL_ERR_OUT_OF_MEMORY, "multigrid records");
        int rc = build_hierarchy<double>(ctx, ctx->mg64, sizeof(Rec64));
        if (rc != EL_OK) return rc;
    }
    if (solver == EL_SOLVER_MIXED && !ctx->x32) {
        EL_CUDA_TRY(ctx, cudaFuncSetAttribute(mg_bottom_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              (int)sizeof(BottomSmem)));
        // the fused coarse cycle: 1024-thread CTAs, all resident, where cooperative launches
        // exist; otherwise the per-level launches stay in use
        int coop = 0;
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, ctx->device);
        ctx->coarse_per_sm = 0;
        if (coop) {
            EL_CUDA_TRY(ctx, cudaFuncSetAttribute(mg_coarse_cycle_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                  (int)sizeof(BottomSmem)));
            int per_sm = 0;
            EL_CUDA_TRY(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, mg_coarse_cycle_kernel,
                                                                          kCycleThreads, (int)sizeof(BottomSmem)));
            ctx->coarse_bar = (unsigned*)ctx_alloc(ctx, 64);
            if (!ctx->coarse_bar) return set_error(ctx, EL_ERR_OUT_OF_MEMORY, "coarse cycle barrier");
            ctx->coarse_per_sm = per_sm;
        }
        ctx->x32 = (float*)ctx_alloc(ctx, n * 4);
        ctx->r32 = (float*)ctx_alloc(ctx, n * 4);
        ctx->z32 = (float*)ctx_alloc(ctx, n * 4);
        ctx->p32 = (float*)ctx_alloc(ctx, n * 4);
        ctx->p32b = (float*)ctx_alloc(ctx, n * 4);
        ctx->ap32 = (float*)ctx_alloc(ctx, n * 4);
        ctx->r32b = (float*)ctx_alloc(ctx, n * 4);
        ctx->xs = (float2*)ctx_alloc(ctx, n * sizeof(float2));
        ctx->A32 = (float4*)ctx_alloc(ctx, n * sizeof(float4));
        ctx->A16 = (ushort4*)ctx_alloc(ctx, n * sizeof(ushort4));
        if (!ctx->x32 || !ctx->r32 || !ctx->r32b || !ctx->z32 || !ctx->p32 || !ctx->p32b || !ctx->ap32 || !ctx->A32 ||
            !ctx->A16 || !ctx->xs)
            return set_error(ctx, EL_ERR_OUT_OF_MEMORY, "mixed solver vectors");
        int rc = build_hierarchy<float>(ctx, ctx->mg32, sizeof(float4));
        if (rc != EL_OK) return rc;
        ctx->mg32[0].rec = ctx->A16;
        ctx->mg32[0].b = ctx->r32;
        ctx->mg32[0].x = ctx->z32;
        rc = march_setup(ctx);
        if (rc != EL_OK) return rc;
    }
    return EL_OK;
}

EL_CHECK_EXPORT(solve)

}  // namespace el
