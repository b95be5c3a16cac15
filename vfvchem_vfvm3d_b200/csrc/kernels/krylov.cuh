// Krylov-subspace kernels for the restarted GMRES (sm_100a).
//
// The reference solves with faer_gmres::restarted_gmres + JacobiPreconLinOp
// (src/linear/linear_gmres.rs:76-84). Restated here from the published algorithm
// (Saad & Schultz 1986, right preconditioning, Givens least squares) with these device choices:
//   * basis vectors u_i are stored UNNORMALISED, with their norms beta_i in a device array;
//     v_i = u_i / beta_i. The SpMV of step j multiplies by 1/beta_j on the way out, so no separate
//     normalisation pass over the basis is ever made;
//   * orthogonalisation is classical Gram-Schmidt with one re-orthogonalisation (CGS2), which has
//     the stability of modified Gram-Schmidt; each pass is one multi-vector kernel that streams the
//     block's rows of every basis vector once, accumulates per-warp partial dots, and reduces them
//     deterministically (fixed order, no float atomics) in the last block to finish;
//   * the Hessenberg column, the Givens rotation and the residual estimate are finished by that last
//     block, so a whole restart cycle runs without a host synchronisation and is captured in a CUDA
//     graph. Every kernel first reads DevStatus::done and returns at once after convergence.
// Vectors are of type T (double, or float in the mixed-precision inner solve); all dots, norms,
// the Hessenberg matrix and the rotations are double.
#pragma once
#include "../internal.cuh"

namespace vfv {

constexpr int kBlk = 256;        // threads per block of the vector kernels
constexpr int kMaxBasis = 128;   // m + 1 <= kMaxBasis

// Rows of one 16-byte chunk (4 floats, 2 doubles): a thread of the multi-vector kernels owns one
// chunk.
template <typename T>
constexpr int kVecRows = 16 / (int)sizeof(T);

// Shapes of the multi-vector kernels. A block's threads form kVS groups; every group owns the same
// tile of rows and takes each kVS-th basis vector's dot, loading the chunks of kGV of its vectors
// before it uses any of them. In an update the vectors form kChains chains; a thread adds up kCA of them
// at a time (one of float rows: registers), loading the chunks of kGU vectors of each. kMinBlocks bounds the registers.
// All shapes give the same bits, for the shape goes by the rows of a whole batch while a mesh's iterates
// must not: a dot is summed over 64 chunks (two warps, one block of VecSmall), then over four such in
// turn (one block of the others), then over those as in sum_groups; an update adds up the basis vectors
// in the same kChains chains.
struct VecWide {  // many rows: a full SM of threads hides the latency
    static constexpr int kGV = 2, kGU = 2, kCA = 1, kVS = 1, kMinBlocks = 8, kPer = 1;
};
struct VecMid {  // a few blocks per SM: more loads in flight per thread instead
    static constexpr int kGV = 8, kGU = 4, kCA = 2, kVS = 1, kMinBlocks = 4, kPer = 1;
};
struct VecSmall {  // fewer blocks than SMs: smaller tiles, and the basis is split over the block's warps as well
    static constexpr int kGV = 8, kGU = 8, kCA = 1, kVS = 4, kMinBlocks = 3, kPer = 4;  // kPer: blocks whose partials are added first
};
template <typename T, class S>
__host__ __device__ constexpr int64_t vec_block_rows() {
    return (int64_t)(kBlk / S::kVS) * kVecRows<T>;
}

// Per-solve device workspace pointers used by the Krylov kernels.
struct KrylovDev {
    int64_t n;          // rows
    int64_t ldv;        // stride between basis vectors (elements)
    int m;              // restart length
    int nblk;           // blocks of the multi-vector kernels
    double* part;       // [3][kMaxBasis][nblk] per-block partial dots: first pass, second pass, ||w||^2
    unsigned* counter;  // [4] last-block counters
    double* hacc;       // [kMaxBasis] current Hessenberg column (accumulated over the CGS passes)
    double* coef;       // [kMaxBasis] update coefficients d_i / beta_i^2
    double* coefz;      // [kMaxBasis] both CGS passes' coefficients summed (overlapped engine), or null
    double* H;          // [m][m+1] column-major Hessenberg (rotated in place)
    double* cs;         // [m]
    double* sn;         // [m]
    double* g;          // [m+1]
    double* beta;       // [m+1] norms of the stored basis vectors
    double* inv_beta;   // [m+1]
    double* y;          // [m] least-squares solution scaled by 1/beta_i
    DevStatus* st;
    double* wnorm2;     // [1] ||w||^2 of the vector being orthogonalised (the reorthogonalisation test)
    const double* scal; // [0] tol_abs: converged when ||r|| <= tol_abs
                        // [1] inner_floor_rel: a cycle also stops once resid_est <= inner_floor_rel * beta0
};

// ---------------------------------------------------------------- last-block helper
// Threads that wrote partials fence their own writes before calling this (see publish_partial);
// after the block-wide barrier thread 0 takes a ticket, and the block that takes the last ticket
// reads every block's partials.
__device__ __forceinline__ bool last_block_arrive(unsigned* counter) {
    __shared__ bool s_last;
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned t = atomicAdd(counter, 1u);
        s_last = (t == gridDim.x - 1);
    }
    __syncthreads();
    if (s_last) __threadfence();
    return s_last;
}

// store one partial and make it visible device-wide before the block arrives
__device__ __forceinline__ void publish_partial(double* p, double v) {
    *p = v;
    __threadfence();
}

// Sum of the q-th PER of the nb partials, in order
template <int PER>
__device__ __forceinline__ double partial_group(const double* part, int q, int nb) {
    double v[PER];
#pragma unroll
    for (int u = 0; u < PER; ++u) v[u] = PER * q + u < nb ? __ldcg(part + PER * q + u) : 0.0;
    double s = v[0];
#pragma unroll
    for (int u = 1; u < PER; ++u) s += v[u];
    return s;
}

// Sum of part[0..nblk) with all threads of the block, PER partials first, in a fixed order; valid in thread 0.
template <int PER = 1>
__device__ __forceinline__ double reduce_partials(const double* part, int nblk, double* red) {
    double s = 0.0;
    for (int q = threadIdx.x; PER * q < nblk; q += blockDim.x) s += partial_group<PER>(part, q, nblk);
    return block_sum(s, red);
}

// Sum of part[0..nb) with one warp, PER partials first, in a fixed order; valid in every lane.
template <int PER>
__device__ __forceinline__ double sum_groups(const double* part, int nb) {
    const int lane = threadIdx.x & 31, ng = (nb + PER - 1) / PER;
    constexpr int kB = 16;
    double s = 0.0;
    for (int q0 = 0; q0 < ng; q0 += 32 * kB) {
        double v[kB];
#pragma unroll
        for (int k = 0; k < kB; ++k) {
            const int q = q0 + lane + 32 * k;
            v[k] = q < ng ? partial_group<PER>(part, q, nb) : 0.0;
        }
#pragma unroll
        for (int h = kB / 2; h > 0; h >>= 1)
#pragma unroll
            for (int k = 0; k < h; ++k) v[k] += v[k + h];
        s += v[0];
    }
    return warp_sum(s);
}

// ---------------------------------------------------------------- SpMV (CSR, G lanes per row)
constexpr int kSpG = 4;  // lanes per row: rows hold ~16 non-zeros, 4 lanes x 4 loads in flight each

// This lane's share of row `row` of A x. The row's first S*G column indices and values are loaded
// before any x is gathered (S strides per lane, all independent), which keeps several loads in
// flight per lane; rows longer than S*G finish in a tail loop.
template <typename TV, int S>
struct RowFrag {
    int32_t b, e, c[S];
    TV v[S];
};

template <typename TV, int G, int S>
__device__ __forceinline__ void row_load(RowFrag<TV, S>& f, const int32_t* __restrict__ rp, const int32_t* __restrict__ ci,
                                         const TV* __restrict__ val, int64_t row, int lane, bool skip = false) {
    f.b = __ldg(rp + row);
    f.e = __ldg(rp + row + 1);
    if (skip) f.e = f.b;
#pragma unroll
    for (int t = 0; t < S; ++t) {
        const int32_t k = f.b + lane + t * G;
        const bool ok = k < f.e;
        f.c[t] = ok ? __ldcs(ci + k) : -1;
        f.v[t] = ok ? __ldcs(val + k) : TV(0);
    }
}

// x may have been written by the previous kernel of a programmatic-dependent-launch chain: plain loads
// unless RO
template <typename TV, typename TX, typename TA, int G, int S, bool RO = false>
__device__ __forceinline__ TA row_gather(const RowFrag<TV, S>& f, const int32_t* __restrict__ ci, const TV* __restrict__ val, const TX* x,
                                         int lane) {
    TA s = TA(0);
#pragma unroll
    for (int t = 0; t < S; ++t)
        if (f.c[t] >= 0) s += (TA)f.v[t] * (TA)(RO ? __ldg(x + f.c[t]) : x[f.c[t]]);
    // The rest of the row. Shapes of 8 lanes and more serve long rows: S strides are loaded ahead of their
    // gathers again (flow system, 131,072 rows of 79 and 427 entries: double 55.4 -> 52.9 us, float 41.1 ->
    // 39.1). With fewer lanes the rest is an entry or two and the masked loads cost more than they hide
    // (10^6 heat rows, 4 lanes x 4: double 47.2 / 51.7, float 34.9 / 38.8).
    if constexpr (G >= 8) {
        for (int32_t k0 = f.b + lane + S * G; k0 < f.e; k0 += S * G) {
            int32_t c[S];
            TV v[S];
#pragma unroll
            for (int t = 0; t < S; ++t) {
                const bool ok = k0 + t * G < f.e;
                c[t] = ok ? __ldcs(ci + k0 + t * G) : -1;
                v[t] = ok ? __ldcs(val + k0 + t * G) : TV(0);
            }
#pragma unroll
            for (int t = 0; t < S; ++t)
                if (c[t] >= 0) s += (TA)v[t] * (TA)(RO ? __ldg(x + c[t]) : x[c[t]]);
        }
    } else {
        for (int32_t k = f.b + lane + S * G; k < f.e; k += G) {
            const TV v = __ldcs(val + k);
            const int32_t c = __ldcs(ci + k);
            s += (TA)v * (TA)(RO ? __ldg(x + c) : x[c]);
        }
    }
    return s;
}

template <typename TV, typename TX, typename TA, int G, int S = 4>
__device__ __forceinline__ TA row_dot(const int32_t* __restrict__ rp, const int32_t* __restrict__ ci, const TV* __restrict__ val,
                                      const TX* x, int64_t row, int lane) {
    RowFrag<TV, S> f;
    row_load<TV, G, S>(f, rp, ci, val, row, lane);
    return row_gather<TV, TX, TA, G, S>(f, ci, val, x, lane);
}

// y = scale * (A x). Accumulation in TA. `scale` may be null (= 1). Inside a cycle graph (CHAIN) the
// row's indices and values, which no kernel of the cycle writes, are loaded before the wait for the
// kernel that produces x. Alone (st null) there is nothing to wait for and x may come through the
// read-only path (4 lanes x 4: 262,144 rows double 16.3 -> 15.4 us, 10^6 rows float 36.9 -> 34.9).
template <typename TV, typename TX, typename TY, typename TA, int G, int S, bool CHAIN>
__global__ void __launch_bounds__(kBlk) k_spmv(int64_t n, const int32_t* __restrict__ rp, const int32_t* __restrict__ ci,
                                              const TV* __restrict__ val, const TX* x, TY* y, const double* scale, const DevStatus* st) {
    const int lane = threadIdx.x & (G - 1);
    const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / G;
    const bool skip = CHAIN && st->done;  // set once and for all within a cycle: such a launch loads no rows
    RowFrag<TV, S> f;
    if (row < n) row_load<TV, G, S>(f, rp, ci, val, row, lane, skip);
    if constexpr (CHAIN) {
        pdl_wait();
        pdl_launch_dependents();
        if (skip || st->done) return;
    }
    TA s = TA(0);
    if (row < n) s = row_gather<TV, TX, TA, G, S, !CHAIN>(f, ci, val, x, lane);
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, G);
    if (lane == 0 && row < n) {
        const double sc = scale ? *scale : 1.0;
        y[row] = (TY)((double)s * sc);
    }
}

// The solvers' SpMV of matrices with short rows: a thread per row of the sliced layout (SellDev), whose
// indices and values a warp reads in full lines; several lanes per CSR row read runs of 16 to 32 bytes.
// The first K entries are loaded before the wait for the kernel that produces x. The thread keeps one
// sum per lane of the CSR shape (entry q of the row in sum q mod G) and adds them as the lanes' shuffles
// do, so that a row's product has the same bits in either layout: which of them a solver reads can go by
// the size of the whole system. Alone on the 10^6-row heat matrix with one sum per row, CSR with the
// autotuned lanes and sliced: float 33.1 -> 26.9 us, double 47.3 -> 38.8 us (5.5 TB/s of the matrix's
// bytes); 103,823 rows 8.3 -> 6.2 us. The lanes' sums cost nothing that whole solves show (10^6 rows mixed
// 89.0 ms with one sum and with four, 262,144 rows FP64 32.6 / 32.7, a batch of 884,000 rows 33.9 / 34.3).
// scale: the step's 1 / beta_j (SEG: looked up per row from its mesh, scale[mesh * stride + j]).
constexpr int kSellBlocks = 5;  // resident blocks per SM of the double kernel
// the float kernel's: full SMs while the lanes' sums fit 32 registers (with more sums it spills)
template <typename T, int G, bool SEG>
constexpr int kSellMinBlocks = sizeof(T) == 8 ? kSellBlocks : G == 8 ? 6 : G == 4 && SEG ? 7 : 8;
struct SellSeg {
    int stride, j, nm;
    const int64_t* mesh_row;
};
__device__ __forceinline__ int mesh_of_row(const int64_t* __restrict__ mesh_row, int nm, int64_t row) {
    int lo = 0, hi = nm;  // mesh_row[lo] <= row < mesh_row[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(mesh_row + mid) <= row) lo = mid;
        else hi = mid;
    }
    return lo;
}

template <typename T, int G, bool SEG>
__global__ void __launch_bounds__(kSellWindow, (kSellMinBlocks<T, G, SEG>))
    k_spmv_sell(int64_t n, SellDev S, const int32_t* __restrict__ ci, const T* __restrict__ val, const T* x, T* y, const double* scale, SellSeg seg,
                const DevStatus* st) {
    constexpr int K = 8;
    static_assert(K % G == 0, "entry q goes to sum q mod G");
    const int32_t t = (int32_t)(blockIdx.x * blockDim.x + threadIdx.x);
    const bool skip = st && st->done;  // set once and for all within a cycle: such a launch loads no rows
    const int32_t k0 = __ldg(S.so + (t >> 5)), k1 = __ldg(S.so + (t >> 5) + 1);
    const int32_t row = (t & ~(kSellWindow - 1)) + (int32_t)__ldg(S.p8 + t);
    const int32_t kb = k0 + (t & 31), w = skip ? 0 : (k1 - k0) >> 5;
    int32_t c[K];
    T v[K];
#pragma unroll
    for (int q = 0; q < K; ++q) {
        c[q] = q < w ? __ldcs(ci + kb + 32 * q) : -1;
        v[q] = q < w ? __ldcs(val + kb + 32 * q) : T(0);
    }
    int mesh = 0;
    if (SEG && row < n) mesh = mesh_of_row(seg.mesh_row, seg.nm, row);
    pdl_wait();
    pdl_launch_dependents();
    if (skip || (st && st->done)) return;
    T s[G];
#pragma unroll
    for (int g = 0; g < G; ++g) s[g] = T(0);
#pragma unroll
    for (int q = 0; q < K; ++q)
        if (c[q] >= 0) s[q % G] += v[q] * x[c[q]];
    for (int q0 = K; q0 < w; q0 += K) {
#pragma unroll
        for (int q = 0; q < K; ++q) {
            c[q] = q0 + q < w ? __ldcs(ci + kb + 32 * (q0 + q)) : -1;
            v[q] = q0 + q < w ? __ldcs(val + kb + 32 * (q0 + q)) : T(0);
        }
#pragma unroll
        for (int q = 0; q < K; ++q)
            if (c[q] >= 0) s[q % G] += v[q] * x[c[q]];
    }
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1)
#pragma unroll
        for (int g = 0; g < o; ++g) s[g] += s[g + o];
    if (row < n) y[row] = (T)((double)s[0] * scale[SEG ? (int64_t)mesh * seg.stride + seg.j : 0]);
}

// out = (T)(val[k] * dinv[col[k]]) in the sliced layout (right Jacobi scaling folded into the Krylov
// matrix; dinv null: the values), a thread per position; padding is left as it is. For layouts without
// tails (build_pattern_sell keeps no others): every entry of a row lies within its slice's width.
template <typename T>
__global__ void __launch_bounds__(kSellWindow) k_sell_vals(int64_t n, SellDev S, const int32_t* __restrict__ rp, const int32_t* __restrict__ ci,
                                                          const double* __restrict__ val, const double* __restrict__ dinv,
                                                          T* __restrict__ out) {
    const int32_t t = (int32_t)(blockIdx.x * blockDim.x + threadIdx.x);
    const int32_t row = (t & ~(kSellWindow - 1)) + (int32_t)S.p8[t];
    if (row >= n) return;
    const int32_t kb = S.so[t >> 5] + (t & 31), b = rp[row], cnt = rp[row + 1] - b;
    for (int q = 0; q < cnt; ++q) out[kb + 32 * q] = (T)(val[b + q] * (dinv ? dinv[ci[b + q]] : 1.0));
}

// ---------------------------------------------------------------- residual r = b - A x (FP64)
// Writes u0 = r (type T), accumulates ||r||^2, and in the last block starts a new cycle:
// beta[0] = ||r||, g = (beta0, 0, ...), done/converged flags.
template <typename T, int G>
__global__ void __launch_bounds__(kBlk) k_residual(KrylovDev K, const int32_t* __restrict__ rp, const int32_t* __restrict__ ci,
                                                  const double* __restrict__ val, const double* __restrict__ x,
                                                  const double* __restrict__ b, T* __restrict__ u0) {
    __shared__ double red[kBlk / 32];
    const int lane = threadIdx.x & (G - 1);
    const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / G;
    double s = 0.0;
    if (row < K.n) s = row_dot<double, double, double, G>(rp, ci, val, x, row, lane);
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, G);
    double r2 = 0.0;
    if (lane == 0 && row < K.n) {
        const double r = b[row] - s;
        u0[row] = (T)r;
        r2 = r * r;
    }
    const double bs = block_sum(r2, red);
    if (threadIdx.x == 0) publish_partial(K.part + blockIdx.x, bs);
    if (!last_block_arrive(K.counter)) return;
    const double tot = reduce_partials(K.part, gridDim.x, red);
    if (threadIdx.x == 0) {
        *K.counter = 0u;
        const double beta0 = sqrt(tot);
        K.beta[0] = beta0;
        K.inv_beta[0] = 1.0 / beta0;
        K.g[0] = beta0;
        DevStatus* st = K.st;
        st->steps = 0;
        st->beta0 = beta0;
        st->resid_est = beta0;
        const bool fin = isfinite(beta0);
        st->nonfinite = fin ? 0 : 1;
        const bool conv = fin && beta0 <= K.scal[0];
        st->converged = conv ? 1 : 0;
        st->done = (conv || !fin || beta0 == 0.0) ? 1 : 0;
    }
}

// ---------------------------------------------------------------- grouped multi-vector passes
// A thread owns a chunk of kVecRows<T> consecutive rows, counted from its tile's first row, of which
// `cnt` lie in the tile; the others read as zero and are not written. A complete chunk on a 16-byte
// boundary is moved with one load or store, any other row by row: the last one of a tile, and all of a
// tile that starts off such a boundary (the batched kernels' meshes at odd rows). Per vector the
// thread's rows are summed in row order, then across the warp (butterfly), the block's warps and the
// blocks, in fixed orders.
template <typename T>
__device__ __forceinline__ void load_chunk(const T* p, int cnt, bool aligned, T (&x)[kVecRows<T>]) {
    constexpr int R = kVecRows<T>;
    if (cnt == R && aligned) {
        if constexpr (R == 4) {
            const float4 t = *reinterpret_cast<const float4*>(p);
            x[0] = t.x, x[1] = t.y, x[2] = t.z, x[3] = t.w;
        } else {
            const double2 t = *reinterpret_cast<const double2*>(p);
            x[0] = t.x, x[1] = t.y;
        }
    } else {
#pragma unroll
        for (int r = 0; r < R; ++r) x[r] = r < cnt ? p[r] : T(0);
    }
}

template <typename T>
__device__ __forceinline__ void store_chunk(T* p, int cnt, bool aligned, const T (&x)[kVecRows<T>]) {
    constexpr int R = kVecRows<T>;
    if (cnt == R && aligned) {
        if constexpr (R == 4) *reinterpret_cast<float4*>(p) = make_float4(x[0], x[1], x[2], x[3]);
        else *reinterpret_cast<double2*>(p) = make_double2(x[0], x[1]);
    } else {
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (r < cnt) p[r] = x[r];
    }
}

// The tile [first, end) of a multi-vector kernel seen by one thread: its chunk's first row and rows;
// group and place in the group follow from the thread index.
template <typename T, class S>
struct VecTile {
    static constexpr int kThreads = kBlk / S::kVS, kWarps = kThreads / 32;
    int32_t row0;
    int cnt;
    bool aligned;
    __device__ VecTile(int32_t first, int32_t end, bool aligned_) : aligned(aligned_) {
        constexpr int R = kVecRows<T>;
        row0 = first + R * t();
        cnt = max(min(end - row0, R), 0);
    }
    static __device__ __forceinline__ int g() { return S::kVS == 1 ? 0 : (int)threadIdx.x / kThreads; }
    static __device__ __forceinline__ int t() { return S::kVS == 1 ? (int)threadIdx.x : (int)threadIdx.x % kThreads; }
};

// sum of the block's per-warp partials: two warps (64 chunks) at a time
template <int NW>
__device__ __forceinline__ double warps_sum(const double* red) {
    double s = red[0] + red[1];
#pragma unroll
    for (int v = 2; v < NW; v += 2) s += red[v] + red[v + 1];
    return s;
}

// red[i][warp of the group] = that warp's partial of <u_i, wt> for i < nvec (products in double)
template <typename T, class S>
__device__ __forceinline__ void group_dots(const T* V, int64_t ldv, const VecTile<T, S>& q, const T* wt, int nvec, double (*red)[kBlk / 32]) {
    constexpr int R = kVecRows<T>, GV = S::kGV, VS = S::kVS;
    const T* p = V + q.row0 + q.g() * ldv;
    for (int i = q.g(); i < nvec; i += GV * VS, p += GV * VS * ldv) {
        T x[GV][R];
#pragma unroll
        for (int u = 0; u < GV; ++u) load_chunk(p + u * VS * ldv, i + u * VS < nvec ? q.cnt : 0, q.aligned, x[u]);
#pragma unroll
        for (int u = 0; u < GV; ++u) {
            double sq = 0.0;
#pragma unroll
            for (int r = 0; r < R; ++r) sq += (double)x[u][r] * (double)wt[r];
            sq = warp_sum(sq);
            if ((threadIdx.x & 31) == 0 && i + u * VS < nvec) red[i + u * VS][q.t() >> 5] = sq;
        }
    }
}

// this block's partial of ||w||^2, valid in thread 0 (one barrier)
template <typename T, class S>
__device__ __forceinline__ double tile_norm2(const VecTile<T, S>& q, const T* wt, double* red) {
    if (q.g() == 0) {
        double sq = 0.0;
#pragma unroll
        for (int r = 0; r < kVecRows<T>; ++r) sq += (double)wt[r] * (double)wt[r];
        sq = warp_sum(sq);
        if ((threadIdx.x & 31) == 0) red[q.t() >> 5] = sq;
    }
    __syncthreads();
    return threadIdx.x == 0 ? warps_sum<VecTile<T, S>::kWarps>(red) : 0.0;
}

// w = win - sum_i coef[i] u_i (i < nvec) over the tile's rows; wt: the thread's chunk of w. The sum is one
// of kChains chains (vectors c, c + kChains, ... in order), added in order: a block of several groups has
// a chain per group, one of a single group takes them in turn. s_acc: kVecAcc doubles, one of the sums
// per thread and row; out of registers, for the wide shape has none left.
constexpr int kChains = 4;
template <typename T, class S>
constexpr int kVecAcc = kBlk * kVecRows<T>;

template <typename T, class S>
__device__ __forceinline__ void group_update(const T* V, int64_t ldv, const VecTile<T, S>& q, const double* coef, int nvec, const T* win, T* w,
                                             double* s_acc, T (&wt)[kVecRows<T>]) {
    constexpr int R = kVecRows<T>, GV = S::kGU, CA = sizeof(T) == 8 ? S::kCA : 1, VS = S::kVS, TG = VecTile<T, S>::kThreads;
    static_assert(VS == 1 || VS == kChains, "a chain per group, or all of them in one");
    double* mine = s_acc + q.g() * R * TG + q.t();
#pragma unroll 1
    for (int c = q.g(); c < kChains; c += VS * CA) {
        double acc[CA][R];
#pragma unroll
        for (int a = 0; a < CA; ++a)
#pragma unroll
            for (int r = 0; r < R; ++r) acc[a][r] = 0.0;
        const T* p = V + q.row0 + c * ldv;
        for (int i = c; i < nvec; i += GV * kChains, p += GV * kChains * ldv) {
            T x[GV][CA][R];
#pragma unroll
            for (int u = 0; u < GV; ++u)
#pragma unroll
                for (int a = 0; a < CA; ++a)
                    load_chunk(p + (u * kChains + a) * ldv, i + u * kChains + a < nvec ? q.cnt : 0, q.aligned, x[u][a]);
#pragma unroll
            for (int u = 0; u < GV; ++u)
#pragma unroll
                for (int a = 0; a < CA; ++a) {
                    if (i + u * kChains + a < nvec) {
                        const double cf = coef[i + u * kChains + a];
#pragma unroll
                        for (int r = 0; r < R; ++r) acc[a][r] += cf * (double)x[u][a][r];
                    }
                }
        }
#pragma unroll
        for (int a = 0; a < CA; ++a)
#pragma unroll
            for (int r = 0; r < R; ++r) mine[r * TG] = VS > 1 || c + a == 0 ? acc[a][r] : mine[r * TG] + acc[a][r];
    }
    load_chunk(win + q.row0, q.cnt, q.aligned, wt);
    if constexpr (VS > 1) __syncthreads();  // and every group has read win before group 0 overwrites it (win may be w)
#pragma unroll
    for (int r = 0; r < R; ++r) {
        double a = s_acc[r * TG + q.t()];
#pragma unroll
        for (int g = 1; g < VS; ++g) a += s_acc[(g * R + r) * TG + q.t()];
        wt[r] = (T)((double)wt[r] - a);  // rows past the end: 0 - 0
    }
    if (q.g() == 0) store_chunk(w + q.row0, q.cnt, q.aligned, wt);
}

// Up to this many partials per vector the update kernels sum them themselves: two launches per
// Arnoldi step less (8,000 rows: 3.57 against 3.65 ms per solve; 400 partials already cost more than
// the launches they save, 130 against 118 ms at 131,072 rows).
constexpr int kFoldMax = 128;

// sums of the columns c < cnt of part[c][0..nb), nb <= kFoldMax, with the bits of sum_groups: a warp per
// column, several columns' loads in flight; out(c, sum) is called by lane 0. Lanes read consecutive
// partials (every block reads all of them: L2 requests are what this costs); with PER = 4, four lanes'
// values make a group, and the order of the sums is that of sum_groups with group q in lane q.
template <int PER, typename F>
__device__ __forceinline__ void sum_columns(const double* part, int64_t ld, int nb, int cnt, F out) {
    static_assert(PER == 1 || PER == 4, "groups of one or of four lanes");
    constexpr unsigned full = 0xffffffffu;
    constexpr int kCols = PER > 1 ? 4 : 2, kL = kFoldMax / 32;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int c0 = wid; c0 < cnt; c0 += kCols * nw) {
        double v[kCols][kL];
#pragma unroll
        for (int u = 0; u < kCols; ++u)
#pragma unroll
            for (int k = 0; k < kL; ++k)
                v[u][k] = c0 + u * nw < cnt && lane + 32 * k < nb ? __ldcg(part + (int64_t)(c0 + u * nw) * ld + lane + 32 * k) : 0.0;
#pragma unroll
        for (int u = 0; u < kCols; ++u) {
            if constexpr (PER == 4) {
#pragma unroll
                for (int k = 0; k < kL; ++k) {
                    if (32 * k >= nb) continue;
                    const double b = __shfl_down_sync(full, v[u][k], 1), c = __shfl_down_sync(full, v[u][k], 2), d = __shfl_down_sync(full, v[u][k], 3);
                    v[u][k] = v[u][k] + b + c + d;  // in every fourth lane
                }
            }
            double s = (v[u][0] + v[u][2]) + (v[u][1] + v[u][3]);
#pragma unroll
            for (int o = 16; o >= PER; o >>= 1) s += __shfl_xor_sync(full, s, o);
            if (lane == 0 && c0 + u * nw < cnt) out(c0 + u * nw, s);
        }
    }
}
static_assert(kFoldMax == 128, "four partials a lane");

// ---------------------------------------------------------------- multi-dot (first CGS pass)
// Per-block partials of d_i = <u_i, w> for i < nvec (summed by k_dots_finish<true>, or by k_update<FOLD>). with_norm: also the partials of ||w||^2, as vector nvec (the first pass
// of the reorthogonalise-if-needed scheme); only_reorth: a second pass (its partials go to the second
// buffer), skipped unless the first pass asked for it.
template <typename T, class S>
__global__ void __launch_bounds__(kBlk, S::kMinBlocks) k_mdot(KrylovDev K, const T* V, const T* w, int nvec, int with_norm, int only_reorth) {
    pdl_wait();
    pdl_launch_dependents();
    if (K.st->done || (only_reorth && !K.st->reorth)) return;
    __shared__ double red[kMaxBasis][kBlk / 32];
    constexpr int R = kVecRows<T>, NW = VecTile<T, S>::kWarps;
    const VecTile<T, S> q((int32_t)(blockIdx.x * vec_block_rows<T, S>()), (int32_t)K.n, true);
    T wt[R];
    load_chunk(w + q.row0, q.cnt, q.aligned, wt);
    group_dots<T, S>(V, K.ldv, q, wt, nvec, red);
    if (with_norm && q.g() == 0) {
        double sq = 0.0;
#pragma unroll
        for (int r = 0; r < R; ++r) sq += (double)wt[r] * (double)wt[r];
        sq = warp_sum(sq);
        if ((threadIdx.x & 31) == 0) red[nvec][q.t() >> 5] = sq;
    }
    __syncthreads();
    const int nout = nvec + (with_norm ? 1 : 0);
    double* part = K.part + (only_reorth ? (int64_t)kMaxBasis * K.nblk : 0);
    for (int i = threadIdx.x; i < nout; i += blockDim.x) part[(int64_t)i * K.nblk + blockIdx.x] = warps_sum<NW>(red[i]);
}

// Cross-block sums of the multi-dot partials, one warp per basis vector spread over the GPU (a
// last-block reduction here would leave the GPU idle for ~15 us while one block walks
// nvec x nblk partials). FIRST: hacc_i = d_i / beta_i; else hacc_i += d_i / beta_i; both set
// coef_i = d_i / beta_i^2 for the update that follows.
// with_norm: warp nvec sums the partials of ||w||^2 into wnorm2; only_reorth as in k_mdot.
template <class S, bool FIRST>
__global__ void __launch_bounds__(256) k_dots_finish(KrylovDev K, int nvec, int with_norm, int only_reorth) {
    pdl_wait();
    pdl_launch_dependents();
    if (K.st->done || (only_reorth && !K.st->reorth)) return;
    const int lane = threadIdx.x & 31;
    const int c = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (c >= nvec + (with_norm ? 1 : 0)) return;
    const double s = sum_groups<S::kPer>(K.part + (int64_t)((FIRST ? 0 : kMaxBasis) + c) * K.nblk, K.nblk);
    if (lane == 0 && c == nvec) {
        K.wnorm2[0] = s;
        return;
    }
    if (lane == 0) {
        const double ib = K.inv_beta[c];
        if (FIRST) K.hacc[c] = s * ib;
        else K.hacc[c] += s * ib;
        const double cf = s * ib * ib;
        K.coef[c] = cf;
        if (K.coefz) K.coefz[c] = FIRST ? cf : K.coefz[c] + cf;
    }
}

// ---------------------------------------------------------------- Hessenberg column
// Completes Arnoldi step j: the column h[0..j] (in shared memory, with the previous rotations
// cs[0..j), sn[0..j)) is rotated, a new rotation makes its subdiagonal bnext = sqrt(tot) vanish, and
// the rotated column, the norms and g are stored. Whole block; tot and the result are thread 0's.
// Only t -> c h - s t is serial, two operations per row out of shared memory; walking the column in
// global memory took over 10 us at j = 50.
struct ColumnSmem {
    double h[kMaxBasis + 1], cs[kMaxBasis], sn[kMaxBasis];
};
struct ColumnDst {
    double *col, *cs, *sn, *g, *beta, *inv_beta;
};
struct ColumnEnd {
    double est, bnext, rr;
};

__device__ __forceinline__ ColumnEnd arnoldi_column(const ColumnDst& D, ColumnSmem& s, int j, double tot) {
    ColumnEnd e{0.0, 0.0, 0.0};
    __syncthreads();
    if (threadIdx.x == 0) {
        const double gj = D.g[j];
        const double bnext = sqrt(tot);
        double t = s.h[0];
#pragma unroll 4
        for (int i = 0; i < j; ++i) {
            const double hn = s.h[i + 1], c = s.cs[i], sn = s.sn[i];
            s.h[i] = c * t + sn * hn;
            t = c * hn - sn * t;
        }
        const double rr = hypot(t, bnext);
        double c = 1.0, sgn = 0.0;
        if (rr > 0.0) {
            c = t / rr;
            sgn = bnext / rr;
        }
        s.h[j] = rr;
        D.cs[j] = c;
        D.sn[j] = sgn;
        D.beta[j + 1] = bnext;
        D.inv_beta[j + 1] = 1.0 / bnext;
        D.g[j] = c * gj;
        D.g[j + 1] = -sgn * gj;
        e = {fabs(sgn * gj), bnext, rr};
    }
    __syncthreads();
    for (int i = threadIdx.x; i <= j; i += blockDim.x) D.col[i] = s.h[i];
    if (threadIdx.x == 0) D.col[j + 1] = 0.0;
    return e;
}

// ---------------------------------------------------------------- update + second pass
// w <- win - sum_i coef_i u_i (win == w except in the overlapped engine). Then, with FINAL == false, the partials of the second CGS pass
// d'_i = <u_i, w> (k_dots_finish<false> adds d'_i/beta_i into hacc and sets coef); with
// FINAL == true, ||w||^2 and the last block finishes the Hessenberg column j, the Givens rotation
// and the convergence test - unless dgks is set and the test asks for a second pass, whose own
// k_update (launched with only_reorth) then finishes the column. second: the coefficients come from
// the second pass. FOLD: every block sums the (few) partials itself instead of reading the coefficients
// that k_dots_finish left; a template argument, for the sums' registers would spill in the shapes of
// many blocks, which never fold (VecWide, 32 registers, 10^6 rows).
template <typename T, class S, bool FINAL, bool FOLD>
__global__ void __launch_bounds__(kBlk, S::kMinBlocks) k_update(KrylovDev K, const T* V, const T* win, T* w, int nvec, int j, int second,
                                                                int dgks, int only_reorth) {
    pdl_wait();
    pdl_launch_dependents();
    if (K.st->done || (only_reorth && !K.st->reorth)) return;
    constexpr int R = kVecRows<T>, NW = VecTile<T, S>::kWarps;
    __shared__ double red[FINAL ? 1 : kMaxBasis][kBlk / 32];
    __shared__ double s_coef[kMaxBasis];
    __shared__ double s_acc[kVecAcc<T, S>];
    __shared__ ColumnSmem s_col;
    double* h = s_col.h;
    if constexpr (FOLD) {
        sum_columns<S::kPer>(K.part + (second ? (int64_t)kMaxBasis * K.nblk : 0), K.nblk, K.nblk, nvec, [&](int c, double s) {
            const double ib = K.inv_beta[c], hc = s * ib, cf = hc * ib;
            s_coef[c] = cf;
            h[c] = second ? K.hacc[c] + hc : hc;
            if (blockIdx.x == 0) {
                if (!second) K.hacc[c] = hc;
                if (K.coefz) K.coefz[c] = second ? K.coefz[c] + cf : cf;
            }
        });
    } else {
        for (int i = threadIdx.x; i < nvec; i += blockDim.x) {
            s_coef[i] = K.coef[i];
            if (FINAL) h[i] = K.hacc[i];
        }
    }
    if (FINAL)
        for (int i = threadIdx.x; i < j; i += blockDim.x) {
            s_col.cs[i] = K.cs[i];
            s_col.sn[i] = K.sn[i];
        }
    __syncthreads();
    const VecTile<T, S> q((int32_t)(blockIdx.x * vec_block_rows<T, S>()), (int32_t)K.n, true);
    T wt[R];
    group_update<T, S>(V, K.ldv, q, s_coef, nvec, win, w, s_acc, wt);  // win may be w
    if (!FINAL) {
        group_dots<T, S>(V, K.ldv, q, wt, nvec, red);
        __syncthreads();
        double* part = K.part + (int64_t)kMaxBasis * K.nblk;
        // summed by k_dots_finish<false> or the next update
        for (int i = threadIdx.x; i < nvec; i += blockDim.x) part[(int64_t)i * K.nblk + blockIdx.x] = warps_sum<NW>(red[i]);
    } else {
        const double s = tile_norm2<T, S>(q, wt, red[0]);
        double* part = K.part + (int64_t)2 * kMaxBasis * K.nblk;
        if (threadIdx.x == 0) publish_partial(part + blockIdx.x, s);
        if (!last_block_arrive(K.counter + 3)) return;
        const double tot = reduce_partials<S::kPer>(part, gridDim.x, red[0]);
        // first pass of the reorthogonalise-if-needed scheme (Daniel, Gragg, Kaufman & Stewart
        // 1976): a second pass only when the projection removed more than half of ||w||^2
        __shared__ int s_again;
        double wn2 = 0.0;
        if (dgks) {
            __syncthreads();
            wn2 = FOLD ? reduce_partials<S::kPer>(K.part + (int64_t)nvec * K.nblk, K.nblk, red[0]) : K.wnorm2[0];
        }
        if (threadIdx.x == 0) {
            K.counter[3] = 0u;
            s_again = dgks && tot < 0.5 * wn2;
            K.st->reorth = s_again;
        }
        __syncthreads();
        if (s_again) return;
        const ColumnDst D{K.H + (int64_t)j * (K.m + 1), K.cs, K.sn, K.g, K.beta, K.inv_beta};
        const ColumnEnd c = arnoldi_column(D, s_col, j, tot);
        if (threadIdx.x == 0) {
            DevStatus* st = K.st;
            st->steps = j + 1;
            st->total_steps += 1;
            st->resid_est = c.est;
            const bool fin = isfinite(c.est) && isfinite(c.bnext) && isfinite(c.rr);
            if (!fin) st->nonfinite = 1;
            const double floor_abs = K.scal[1] * st->beta0;
            if (!fin || c.rr == 0.0 || c.bnext == 0.0 || c.est <= K.scal[0] || c.est <= floor_abs || j + 1 >= K.m) st->done = 1;
        }
    }
}

// Overlapped engine: the preconditioned image of the new basis vector by linearity,
// z_{j+1} = M^-1 (w - sum_i c_i u_i) = q - sum_i c_i z_i with q = M^-1 w computed concurrently
// with the orthogonalisation and c_i the sum of both CGS passes' coefficients.
template <typename T, class S>
__global__ void __launch_bounds__(kBlk, S::kMinBlocks) k_zupdate(KrylovDev K, T* Z, const T* qv, int nvec, int j) {
    pdl_wait();
    pdl_launch_dependents();
    if (K.st->done) return;
    constexpr int R = kVecRows<T>;
    __shared__ double s_c[kMaxBasis];
    __shared__ double s_acc[kVecAcc<T, S>];
    for (int i = threadIdx.x; i < nvec; i += blockDim.x) s_c[i] = K.coefz[i];
    __syncthreads();
    const VecTile<T, S> q((int32_t)(blockIdx.x * vec_block_rows<T, S>()), (int32_t)K.n, true);
    T zt[R];
    group_update<T, S>(Z, K.ldv, q, s_c, nvec, qv, Z + (int64_t)(j + 1) * K.ldv, s_acc, zt);
}

// ---------------------------------------------------------------- end of cycle
// Back substitution R y = g on the rotated Hessenberg matrix's first k columns, y_i scaled by
// 1/beta_i, the others 0. One warp, lane l holding the unknowns l, l + 32, ...: column by column from
// the last, y_i = g_i / R_ii and g_q -= R_qi y_i for all q < i at once, the next column loaded
// meanwhile (one thread walking the triangle in global memory took 120 us at k = 50, 310 us at 100).
__device__ __forceinline__ void back_substitute(const double* H, int m1, int k, int m, const double* g, const double* inv_beta, double* y) {
    constexpr int kU = kMaxBasis / 32;
    const int lane = threadIdx.x & 31;
    double gv[kU], cur[kU], nxt[kU], yv[kU];
    auto load = [&](int i, double* c) {
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const int q = lane + 32 * u;
            c[u] = i >= 0 && q <= i ? H[(int64_t)i * m1 + q] : 0.0;
        }
    };
#pragma unroll
    for (int u = 0; u < kU; ++u) {
        const int q = lane + 32 * u;
        gv[u] = q < k ? g[q] : 0.0;
        yv[u] = 0.0;
    }
    load(k - 1, cur);
    for (int i = k - 1; i >= 0; --i) {
        load(i - 1, nxt);
        double t = 0.0;
#pragma unroll
        for (int u = 0; u < kU; ++u)
            if (u == i >> 5) t = gv[u] / cur[u];
        const double yi = __shfl_sync(0xffffffffu, t, i & 31);
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const int q = lane + 32 * u;
            if (q < i) gv[u] -= cur[u] * yi;
            else if (q == i) yv[u] = yi;
            cur[u] = nxt[u];
        }
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
        const int q = lane + 32 * u;
        if (q < m) y[q] = q < k ? yv[u] * inv_beta[q] : 0.0;
    }
}

__global__ void k_backsolve(KrylovDev K) { back_substitute(K.H, K.m + 1, K.st->steps, K.m, K.g, K.inv_beta, K.y); }

// z = sum_i y_i u_i (i < steps). MODE 0: x += z; MODE 1: x += dinv .* z; MODE 2: zt = (T)z for a preconditioner.
template <typename T, int MODE>
__global__ void __launch_bounds__(kBlk) k_combine(KrylovDev K, const T* __restrict__ V, double* __restrict__ x,
                                                 const double* __restrict__ dinv, T* __restrict__ zt) {
    __shared__ double s_y[kMaxBasis];
    const int k = K.st->steps;
    for (int i = threadIdx.x; i < k; i += blockDim.x) s_y[i] = K.y[i];
    __syncthreads();
    const int64_t row = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= K.n) return;
    double z = 0.0;
    for (int i = 0; i < k; ++i) z += s_y[i] * (double)V[(int64_t)i * K.ldv + row];
    if (MODE == 0) x[row] += z;
    if (MODE == 1) x[row] += dinv[row] * z;
    if (MODE == 2) zt[row] = (T)z;
}

template <typename T>
__global__ void k_add_to_x(int64_t n, double* __restrict__ x, const T* __restrict__ z) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] += (double)z[i];
}

// ||v||^2 into out (single pass, last-block reduction)
__global__ void __launch_bounds__(kBlk) k_norm2(int64_t n, const double* __restrict__ v, double* part, unsigned* counter, double* out) {
    __shared__ double red[kBlk / 32];
    double s = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) s += v[i] * v[i];
    s = block_sum(s, red);
    if (threadIdx.x == 0) publish_partial(part + blockIdx.x, s);
    if (!last_block_arrive(counter)) return;
    const double tot = reduce_partials(part, gridDim.x, red);
    if (threadIdx.x == 0) {
        *counter = 0u;
        *out = tot;
    }
}

// ---------------------------------------------------------------- matrix preparation
// dinv[i] = 1 / a_ii (diag_pos[i] = slot of the diagonal, -1 if absent -> 1)
__global__ void k_jacobi_inv(int64_t n, const int32_t* __restrict__ diag_pos, const double* __restrict__ val, double* __restrict__ dinv) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int32_t p = diag_pos[i];
    const double d = p >= 0 ? val[p] : 0.0;
    dinv[i] = d != 0.0 ? 1.0 / d : 1.0;
}

// z = M^-1 r for the 4x4 block-Jacobi preconditioner of a field-major 4-field system: block v
// couples rows {v, nb+v, 2nb+v, 3nb+v}; binv is [16][nb] (row-major 4x4 per block). `in` and `out`
// may alias (each thread reads its four entries before writing them).
template <typename T>
__global__ void __launch_bounds__(256) k_bj4_apply(int64_t nb, const T* __restrict__ binv, const T* in, T* out, const DevStatus* st) {
    pdl_wait();
    pdl_launch_dependents();
    if (st && st->done) return;
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nb) return;
    T r[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) r[c] = in[c * nb + v];
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        T acc = binv[(4 * a) * nb + v] * r[0];
#pragma unroll
        for (int c = 1; c < 4; ++c) acc += binv[(4 * a + c) * nb + v] * r[c];
        out[a * nb + v] = acc;
    }
}

// out[k] = (T)(val[k] * dinv[col[k]])  (right Jacobi scaling folded into the Krylov matrix)
template <typename T>
__global__ void k_scale_cols(int64_t nnz, const int32_t* __restrict__ ci, const double* __restrict__ val,
                             const double* __restrict__ dinv, T* __restrict__ out) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < nnz) out[k] = (T)(val[k] * (dinv ? dinv[ci[k]] : 1.0));
}

}  // namespace vfv
