// Per-mesh Krylov recurrences for a batch of independent meshes (sm_100a).
//
// The reference solves every system on its own (one LinearGmres::solve_matrix per system,
// src/transient/transient_base.rs:83-109). A batch here is the concatenation of the meshes' systems
// into one block-diagonal matrix whose SpMV and ILU(0) sweeps run over all meshes at once (both are
// block-diagonal operations), while every mesh keeps its OWN Krylov recurrence: its own dot
// products and norms, Hessenberg matrix, Givens rotations, residual estimate, stopping test and
// `done` flag. A mesh that has converged (or finished its m steps of the cycle) is masked out of the
// orthogonalisation kernels; the cycle ends once every mesh is done.
//
// A mesh's iterates have the bits of the same mesh solved alone: the vector kernels work on tiles that
// start at the mesh's first row (the single-system kernels' tiles), the residual on tiles of kBlk / kSpG
// rows, every per-mesh sum runs over the mesh's own tiles, and the orders of all sums are the same for
// every shape of the vector kernels (which goes by the rows of the whole batch) and for folded sums
// (which go by its largest mesh), as they are for both row layouts of the SpMV. A mesh that starts off a
// 16-byte boundary moves its vectors row by row instead of in 16-byte chunks.
#pragma once
#include "krylov.cuh"

namespace vfv {

// Per-mesh scalar state of the batched recurrence.
struct MeshStat {
    int32_t done;         // the mesh takes no more Arnoldi steps this cycle
    int32_t steps;        // steps of the current cycle
    int32_t converged;    // its true residual met its tolerance (frozen for the rest of the solve)
    int32_t nonfinite;
    int32_t total_steps;  // Arnoldi steps over the whole solve
    int32_t zero_rhs;     // b_mesh = 0: x_mesh = 0
    double beta0;         // ||r|| at the start of the cycle
    double resid_est;     // |g_{j+1}|
    double bnorm;         // ||b_mesh||
};

struct BatchDev {
    int nm, m;
    int64_t ldv;
    const int64_t* mesh_row;   // [nm+1] first row of each mesh
    const int64_t* tile_row;   // [ntile+1] vector tiles (at most vec_block_rows rows, inside one mesh)
    const int32_t* tile_mesh;  // [ntile]
    const int32_t* mesh_tile;  // [nm+1]
    const int64_t* rtile_row;  // [nrtile+1] residual tiles (kBlk / kSpG rows, inside one mesh)
    const int32_t* rtile_mesh; // [nrtile]
    const int32_t* mesh_rtile; // [nm+1]
    int ntile, nrtile;
    double* part;              // [3][kMaxBasis][ntile] per-tile partial dots: first pass, second pass, ||w||^2
    double* rpart;             // [2][nrtile] per-tile partial norms of the residual and of b
    double* hacc;              // [nm][kMaxBasis]
    double* coef;              // [nm][kMaxBasis]
    double* H;                 // [nm][m][m+1] column-major per mesh
    double* cs;                // [nm][m]
    double* sn;                // [nm][m]
    double* g;                 // [nm][m+1]
    double* beta;              // [nm][m+1]
    double* inv_beta;          // [nm][m+1]
    double* y;                 // [nm][m]
    double* tol_abs;           // [nm] tol * ||b_mesh||
    MeshStat* ms;              // [nm]
    unsigned* counter;         // [0] arrivals, [1] done and [2] converged meshes at a cycle's start, [3] active meshes
    unsigned* mesh_counter;    // [nm] tiles of the mesh that have arrived in k_bupdate<FINAL>
    DevStatus* st;             // global: done once every mesh is done
    const double* scal;        // [1]: mixed precision, a mesh's cycle also ends at resid_est <= scal[1] * beta0
};

// y = (A x) * inv_beta[mesh(row)][j]: the single-system SpMV with the step's scale looked up per row.
template <typename TV, typename TX, typename TY, typename TA, int G, int S = 4>
__global__ void __launch_bounds__(kBlk) k_spmv_seg(int64_t n, const int32_t* __restrict__ rp, const int32_t* __restrict__ ci,
                                                  const TV* __restrict__ val, const TX* x, TY* y, const double* inv_beta, int stride, int j,
                                                  const int64_t* __restrict__ mesh_row, int nm, const DevStatus* st) {
    const int lane = threadIdx.x & (G - 1);
    const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / G;
    const bool skip = st->done;  // set once and for all within a cycle: such a launch loads no rows
    RowFrag<TV, S> f;
    int mesh = 0;
    if (row < n) {
        row_load<TV, G, S>(f, rp, ci, val, row, lane, skip);
        mesh = mesh_of_row(mesh_row, nm, row);
    }
    pdl_wait();
    pdl_launch_dependents();
    if (skip || st->done) return;
    TA s = TA(0);
    if (row < n) s = row_gather<TV, TX, TA, G, S>(f, ci, val, x, lane);
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, G);
    if (lane == 0 && row < n) y[row] = (TY)((double)s * inv_beta[(int64_t)mesh * stride + j]);
}

// x = 0 on meshes whose right-hand side is zero (their solution)
__global__ void k_bzero_x(BatchDev B, double* __restrict__ x) {
    const int64_t n = B.mesh_row[B.nm];
    const int64_t row = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (row >= n) return;
    if (B.ms[mesh_of_row(B.mesh_row, B.nm, row)].zero_rhs) x[row] = 0.0;
}

// r = b - A x per residual tile (FP64), u0 = r, per-tile ||r||^2 (k_residual's arithmetic). first: the
// start of a solve, every mesh takes part and the tile's ||b||^2 is summed as well.
template <typename T, int G>
__global__ void __launch_bounds__(kBlk) k_bresidual(BatchDev B, const int32_t* __restrict__ rp, const int32_t* __restrict__ ci,
                                                   const double* __restrict__ val, const double* __restrict__ x,
                                                   const double* __restrict__ b, T* __restrict__ u0, int first) {
    __shared__ double red[kBlk / 32];
    const int t = blockIdx.x;
    const MeshStat& M = B.ms[B.rtile_mesh[t]];
    if (!first && (M.converged || M.zero_rhs)) return;  // frozen mesh: no residual, no partial (its finish skips it)
    const int lane = threadIdx.x & (G - 1);
    const int64_t row = B.rtile_row[t] + threadIdx.x / G;
    const bool in = row < B.rtile_row[t + 1];
    double s = 0.0;
    if (in) s = row_dot<double, double, double, G>(rp, ci, val, x, row, lane);
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o, G);
    double r2 = 0.0, b2 = 0.0;
    if (lane == 0 && in) {
        const double bv = b[row], r = bv - s;
        u0[row] = (T)r;
        r2 = r * r;
        b2 = bv * bv;
    }
    const double rs = block_sum(r2, red);
    if (threadIdx.x == 0) B.rpart[t] = rs;
    if (first) {
        const double bs = block_sum(b2, red);
        if (threadIdx.x == 0) B.rpart[B.nrtile + t] = bs;
    }
}

// Arrival of one mesh's k_bresid_finish CTA: counts the done and converged meshes; the last arrival
// publishes the global flags and resets the counters.
__device__ __forceinline__ void batch_arrive(const BatchDev& B, bool done, bool conv) {
    __threadfence();
    if (done) atomicAdd(B.counter + 1, 1u);
    if (conv) atomicAdd(B.counter + 2, 1u);
    __threadfence();
    const unsigned t = atomicAdd(B.counter, 1u);
    if (t == (unsigned)B.nm - 1) {
        __threadfence();
        const unsigned nd = atomicAdd(B.counter + 1, 0u), nc = atomicAdd(B.counter + 2, 0u);
        DevStatus* st = B.st;
        st->total_steps += st->steps;  // the cycle's steps: its longest mesh's (k_bbacksolve)
        st->steps = 0;
        st->converged = nc == (unsigned)B.nm ? 1 : 0;
        st->done = nd == (unsigned)B.nm ? 1 : 0;
        B.counter[0] = B.counter[1] = B.counter[2] = 0u;
        B.counter[3] = (unsigned)B.nm - nd;
        __threadfence();
    }
}

// Start of a cycle per mesh (k_residual's last block): beta0, g, the convergence test. One CTA per
// mesh. first (a solve's start): also ||b_mesh||, the mesh's tolerance and its fresh state; a mesh
// with b = 0 is done (k_bzero_x sets its x).
__global__ void __launch_bounds__(kBlk) k_bresid_finish(BatchDev B, int first, double tol) {
    __shared__ double red[kBlk / 32];
    const int m = blockIdx.x;
    MeshStat* M = B.ms + m;
    const int t0 = B.mesh_rtile[m], nt = B.mesh_rtile[m + 1] - t0;
    const bool frozen = !first && (M->converged || M->zero_rhs);
    double tot = 0.0, bb = 0.0;
    if (!frozen) tot = reduce_partials(B.rpart + t0, nt, red);
    if (first) {
        __syncthreads();
        bb = reduce_partials(B.rpart + B.nrtile + t0, nt, red);
    }
    if (threadIdx.x != 0) return;
    if (first) {
        const double bn = sqrt(bb);
        *M = MeshStat{};
        M->bnorm = bn;
        M->zero_rhs = bn == 0.0 ? 1 : 0;
        M->nonfinite = isfinite(bn) ? 0 : 1;
        B.tol_abs[m] = tol * bn;
        B.mesh_counter[m] = 0u;
    }
    bool conv = frozen || M->zero_rhs;
    if (!conv) {
        const int m1 = B.m + 1;
        const double beta0 = sqrt(tot);
        B.beta[(int64_t)m * m1] = beta0;
        B.inv_beta[(int64_t)m * m1] = 1.0 / beta0;
        B.g[(int64_t)m * m1] = beta0;
        M->steps = 0;
        M->beta0 = beta0;
        M->resid_est = beta0;
        const bool fin = isfinite(beta0);
        if (!fin) M->nonfinite = 1;
        conv = fin && beta0 <= B.tol_abs[m];
        M->converged = conv ? 1 : 0;
        M->done = (conv || !fin || beta0 == 0.0) ? 1 : 0;
        if (!fin) B.st->nonfinite = 1;
    } else {
        M->done = 1;
        M->steps = 0;
        M->converged = 1;
    }
    batch_arrive(B, M->done != 0, conv);
}

// The tile of block t: a multiple of whole chunks behind its mesh's first row.
template <typename T, class S>
__device__ __forceinline__ VecTile<T, S> batch_tile(const BatchDev& B, int t) {
    const int32_t beg = (int32_t)B.tile_row[t];
    return VecTile<T, S>(beg, (int32_t)B.tile_row[t + 1], (beg & (kVecRows<T> - 1)) == 0);
}

// First CGS pass: per-tile partial dots of the mesh's basis with w (k_mdot per tile).
template <typename T, class S>
__global__ void __launch_bounds__(kBlk, S::kMinBlocks) k_bmdot(BatchDev B, const T* V, const T* w, int nvec) {
    pdl_wait();
    pdl_launch_dependents();
    if (B.st->done) return;
    const int t = blockIdx.x;
    if (B.ms[B.tile_mesh[t]].done) return;
    __shared__ double red[kMaxBasis][kBlk / 32];
    constexpr int R = kVecRows<T>, NW = VecTile<T, S>::kWarps;
    const VecTile<T, S> q = batch_tile<T, S>(B, t);
    T wt[R];
    load_chunk(w + q.row0, q.cnt, q.aligned, wt);
    group_dots<T, S>(V, B.ldv, q, wt, nvec, red);
    __syncthreads();
    for (int i = threadIdx.x; i < nvec; i += blockDim.x) B.part[(int64_t)i * B.ntile + t] = warps_sum<NW>(red[i]);
}

// Per-mesh cross-tile sums (k_dots_finish over the mesh's tiles): one warp per (mesh, vector).
template <class S, bool FIRST>
__global__ void __launch_bounds__(256) k_bdots_finish(BatchDev B, int nvec) {
    pdl_wait();
    pdl_launch_dependents();
    if (B.st->done) return;
    const int lane = threadIdx.x & 31;
    const int64_t wgl = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (wgl >= (int64_t)B.nm * nvec) return;
    const int m = (int)(wgl / nvec), c = (int)(wgl % nvec);
    if (B.ms[m].done) return;
    const int t0 = B.mesh_tile[m], nt = B.mesh_tile[m + 1] - t0;
    const double s = sum_groups<S::kPer>(B.part + (int64_t)((FIRST ? 0 : kMaxBasis) + c) * B.ntile + t0, nt);
    if (lane == 0) {
        const double ib = B.inv_beta[(int64_t)m * (B.m + 1) + c];
        double* hacc = B.hacc + (int64_t)m * kMaxBasis;
        if (FIRST) hacc[c] = s * ib;
        else hacc[c] += s * ib;
        B.coef[(int64_t)m * kMaxBasis + c] = s * ib * ib;
    }
}

// w <- win - sum_i coef_i u_i per tile; FINAL == false: second-pass partial dots; FINAL == true:
// per-tile ||w||^2, and the mesh's last tile to arrive completes its Arnoldi step j: Hessenberg
// column, Givens rotation, stopping test (k_update's arithmetic). The last mesh to stop sets the
// global done flag.
template <typename T, class S, bool FINAL, bool FOLD>
__global__ void __launch_bounds__(kBlk, S::kMinBlocks) k_bupdate(BatchDev B, const T* V, const T* win, T* w, int nvec, int j) {
    pdl_wait();
    pdl_launch_dependents();
    if (B.st->done) return;
    const int t = blockIdx.x;
    const int m = B.tile_mesh[t];
    MeshStat* M = B.ms + m;
    if (M->done) return;
    constexpr int R = kVecRows<T>, NW = VecTile<T, S>::kWarps;
    __shared__ double red[FINAL ? 1 : kMaxBasis][kBlk / 32];
    __shared__ double s_coef[kMaxBasis];
    __shared__ double s_acc[kVecAcc<T, S>];
    __shared__ ColumnSmem s_col;
    const int m1 = B.m + 1;
    const int t0 = B.mesh_tile[m], nt = B.mesh_tile[m + 1] - t0;
    double* hacc = B.hacc + (int64_t)m * kMaxBasis;
    double* cs = B.cs + (int64_t)m * B.m;
    double* sn = B.sn + (int64_t)m * B.m;
    const double* inv_beta = B.inv_beta + (int64_t)m * m1;
    if constexpr (FOLD) {
        sum_columns<S::kPer>(B.part + (FINAL ? (int64_t)kMaxBasis * B.ntile : 0) + t0, B.ntile, nt, nvec, [&](int c, double s) {
            const double ib = inv_beta[c], hc = s * ib;
            s_coef[c] = hc * ib;
            s_col.h[c] = FINAL ? hacc[c] + hc : hc;
            if (!FINAL && t == t0) hacc[c] = hc;
        });
    } else {
        for (int i = threadIdx.x; i < nvec; i += blockDim.x) {
            s_coef[i] = B.coef[(int64_t)m * kMaxBasis + i];
            if (FINAL) s_col.h[i] = hacc[i];
        }
    }
    if (FINAL)
        for (int i = threadIdx.x; i < j; i += blockDim.x) {
            s_col.cs[i] = cs[i];
            s_col.sn[i] = sn[i];
        }
    __syncthreads();
    const VecTile<T, S> q = batch_tile<T, S>(B, t);
    T wt[R];
    group_update<T, S>(V, B.ldv, q, s_coef, nvec, win, w, s_acc, wt);  // win may be w
    if (!FINAL) {
        group_dots<T, S>(V, B.ldv, q, wt, nvec, red);
        __syncthreads();
        double* part = B.part + (int64_t)kMaxBasis * B.ntile;
        for (int i = threadIdx.x; i < nvec; i += blockDim.x) part[(int64_t)i * B.ntile + t] = warps_sum<NW>(red[i]);
    } else {
        const double s = tile_norm2<T, S>(q, wt, red[0]);
        double* part = B.part + (int64_t)2 * kMaxBasis * B.ntile;
        __shared__ bool s_last;
        if (threadIdx.x == 0) {
            publish_partial(part + t, s);
            s_last = atomicAdd(B.mesh_counter + m, 1u) == (unsigned)nt - 1;
        }
        __syncthreads();
        if (!s_last) return;
        __threadfence();
        const double tot = reduce_partials<S::kPer>(part + t0, nt, red[0]);
        double* g = B.g + (int64_t)m * m1;
        const ColumnDst D{B.H + ((int64_t)m * B.m + j) * m1, cs, sn, g, B.beta + (int64_t)m * m1, B.inv_beta + (int64_t)m * m1};
        const ColumnEnd c = arnoldi_column(D, s_col, j, tot);
        if (threadIdx.x != 0) return;
        B.mesh_counter[m] = 0u;
        M->steps = j + 1;
        M->total_steps += 1;
        M->resid_est = c.est;
        const bool fin = isfinite(c.est) && isfinite(c.bnext) && isfinite(c.rr);
        if (!fin) {
            M->nonfinite = 1;
            B.st->nonfinite = 1;
        }
        const double floor_abs = B.scal[1] * M->beta0;
        if (!fin || c.rr == 0.0 || c.bnext == 0.0 || c.est <= B.tol_abs[m] || c.est <= floor_abs || j + 1 >= B.m) {
            M->done = 1;
            __threadfence();
            if (atomicSub(B.counter + 3, 1u) == 1u) B.st->done = 1;
        }
    }
}

// Back substitution per mesh (k_backsolve), one warp per mesh; the cycle's step count is its longest mesh's.
__global__ void __launch_bounds__(128) k_bbacksolve(BatchDev B) {
    const int m = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (m >= B.nm) return;
    const int k = B.ms[m].converged ? 0 : B.ms[m].steps;
    const int m1 = B.m + 1;
    if ((threadIdx.x & 31) == 0 && k > 0) atomicMax(&B.st->steps, k);
    back_substitute(B.H + (int64_t)m * B.m * m1, m1, k, B.m, B.g + (int64_t)m * m1, B.inv_beta + (int64_t)m * m1, B.y + (int64_t)m * B.m);
}

// z = sum_i y_i u_i over the mesh's steps of this cycle (k_combine per row). MODE 0: x += z;
// MODE 1: x += dinv .* z; MODE 2: zt = (T)z (to be preconditioned).
template <typename T, int MODE>
__global__ void __launch_bounds__(kBlk) k_bcombine(BatchDev B, const T* __restrict__ V, double* __restrict__ x,
                                                  const double* __restrict__ dinv, T* __restrict__ zt) {
    __shared__ double s_y[kMaxBasis];
    const int t = blockIdx.x;
    const int m = B.tile_mesh[t];
    const int k = B.ms[m].converged ? 0 : B.ms[m].steps;
    for (int i = threadIdx.x; i < k; i += blockDim.x) s_y[i] = B.y[(int64_t)m * B.m + i];
    __syncthreads();
    const int64_t end = B.tile_row[t + 1];
    for (int64_t row = B.tile_row[t] + threadIdx.x; row < end; row += kBlk) {
        double z = 0.0;
        for (int i = 0; i < k; ++i) z += s_y[i] * (double)V[(int64_t)i * B.ldv + row];
        if (MODE == 0) x[row] += z;
        if (MODE == 1) x[row] += dinv[row] * z;
        if (MODE == 2) zt[row] = (T)z;
    }
}

}  // namespace vfv
