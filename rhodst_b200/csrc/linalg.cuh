// linalg.cuh -- block Krylov kernels of the fully-coupled step: SELL-32
// block SpMV, block-Jacobi and subdomain ILU(0) preconditioners, and the
// vector/reduction pieces of block GMRES (CGS2 orthogonalisation, Givens
// least squares on the device) and BiCGStab.  Matrix storage MT may be
// double, float or bf16; vectors, dot products, Hessenberg and norms are FP64.
#pragma once

#include <climits>
#include <type_traits>

#include "kernels.cuh"
#include "rdst_records.h"

namespace rdst {

// entry e of 5x5 block `flat` in a slice-interleaved store: 32 blocks per
// 800-entry chunk, entries interleaved by lane (SELL slots, ILU factors,
// block-Jacobi / pivot inverses with flat = row)
__device__ __forceinline__ size_t flat_e(int flat, int e) {
    return (size_t)(flat >> 5) * (32 * 25) + (size_t)e * 32 + (flat & 31);
}

// compute type of the block factorisations for storage type MT: FP64
// storage in double, FP32 and BF16 storage in float
template <typename MT> struct IluCT { using T = float; };
template <> struct IluCT<double> { using T = double; };

// inverse of a 5x5 block (Gauss-Jordan, partial pivoting: the first row
// with the largest |a[r][c]| below the diagonal), fully unrolled so that the
// row swaps are selects on registers, not indexed local memory
template <typename T>
__device__ __forceinline__ void inv5(const T A[25], T X[25]) {
    T a[5][10];
#pragma unroll
    for (int i = 0; i < 5; ++i)
#pragma unroll
        for (int j = 0; j < 5; ++j) { a[i][j] = A[5 * i + j]; a[i][j + 5] = (i == j) ? T(1) : T(0); }
#pragma unroll
    for (int c = 0; c < 5; ++c) {
        int p = c;
        T best = fabs(a[c][c]);
#pragma unroll
        for (int r = c + 1; r < 5; ++r) {
            const T v = fabs(a[r][c]);
            if (v > best) { best = v; p = r; }
        }
#pragma unroll
        for (int r = c + 1; r < 5; ++r) {
            const bool sw = r == p;
#pragma unroll
            for (int j = 0; j < 10; ++j) {
                const T t = a[r][j], u = a[c][j];
                a[r][j] = sw ? u : t;
                a[c][j] = sw ? t : u;
            }
        }
        const T piv = T(1) / a[c][c];
#pragma unroll
        for (int j = 0; j < 10; ++j) a[c][j] *= piv;
#pragma unroll
        for (int r = 0; r < 5; ++r) {
            if (r == c) continue;
            const T f = a[r][c];
            if (f != T(0)) {
#pragma unroll
                for (int j = 0; j < 10; ++j) a[r][j] -= f * a[c][j];
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 5; ++i)
#pragma unroll
        for (int j = 0; j < 5; ++j) X[5 * i + j] = a[i][j + 5];
}

// y = A x, or b - A x with b, or with JACOBI the block-Jacobi preconditioner
// applied to that, Dinv (...), in the same pass; x in FP64 or (a Krylov basis
// vector) FP32, products and y in FP64.  One row per thread: bound by the
// bytes of the matrix, on few rows by the chain column -> x of each slot.  So
// all 25 entries and the x of a slot are loaded before the first is used, and
// the next slot's column with them; the register bound that allows it (48,
// FP64 80) leaves warps enough (per launch, before with 32 registers and the
// loads one by one -> now: 442 k-cell wing FP64 117 -> 109 us, 0.95 of the copy
// bandwidth, 1.2 M FP32 174 -> 164, 371 k BF16 67 -> 49, 111 k FP64 45 -> 33).
// Five warps a slice, one per component, were no faster on 4 k to 100 k rows.
template <typename MT, typename XT, bool JACOBI>
__global__ void __launch_bounds__(256, sizeof(MT) == 8 ? 3 : 5) k_spmv(SellMat<MT> A, const XT* __restrict__ x, double* __restrict__ y,
                                              const double* __restrict__ b, const MT* __restrict__ dinv,
                                              const int* __restrict__ active) {
    if (active && !*active) return;
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= A.N) return;
    const int s = r >> 5, lane = r & 31;
    const int base = A.slice_off[s], width = A.slice_w[s];
    double acc[5] = {0, 0, 0, 0, 0};
    int cn = width > 0 ? A.col[(size_t)base * 32 + lane] : -1;      // the next slot's column
    for (int k = 0; k < width; ++k) {
        const size_t slot = (size_t)(base + k);
        const int c = cn;
        if (k + 1 < width) cn = A.col[(slot + 1) * 32 + lane];
        if (c < 0) continue;
        const XT* xc = x + 5 * (size_t)c;
        const MT* v = A.val + slot * (32 * 25) + lane;
        MT m[25];
        XT xv[5];
#pragma unroll
        for (int e = 0; e < 25; ++e) m[e] = v[e * 32];
#pragma unroll
        for (int j = 0; j < 5; ++j) xv[j] = xc[j];
#pragma unroll
        for (int i = 0; i < 5; ++i)
#pragma unroll
            for (int j = 0; j < 5; ++j) acc[i] += tod(m[5 * i + j]) * tod(xv[j]);
    }
    double* yr = y + 5 * r;
    if (JACOBI) {
        if (b) {
#pragma unroll
            for (int i = 0; i < 5; ++i) acc[i] = b[5 * r + i] - acc[i];
        }
#pragma unroll
        for (int i = 0; i < 5; ++i) {
            double a = 0;
#pragma unroll
            for (int j = 0; j < 5; ++j) a += ld(&dinv[flat_e(r, 5 * i + j)]) * acc[j];
            yr[i] = a;
        }
    } else if (b) {
#pragma unroll
        for (int i = 0; i < 5; ++i) yr[i] = b[5 * r + i] - acc[i];
    } else {
#pragma unroll
        for (int i = 0; i < 5; ++i) yr[i] = acc[i];
    }
}

// What the solver starts with, in one pass over the matrix: per row A W and,
// from the same entries, A xbar for the constant 5-vector xbar (the normFactor
// reference field); partial sums per block of |A W - A xbar| + |b - A xbar|, b =
// A W + rhs (x = W dependent; else |rhs| with both products zero), and of the
// five |rhs_c|.  One pass and no vector written, where two products, the two
// sums and their stores took 380 us on 1.2 M cells (FP32): 248 us.
template <typename MT>
__global__ void __launch_bounds__(256) k_solve_init(SellMat<MT> A, int dependentW, const double* __restrict__ W,
                                                    const double* __restrict__ xbar, const double* __restrict__ rhs,
                                                    double* __restrict__ partial) {
    const double xb[5] = {xbar[0], xbar[1], xbar[2], xbar[3], xbar[4]};
    double sum[6] = {0, 0, 0, 0, 0, 0};
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < A.N; r += gridDim.x * blockDim.x) {
        double ax[5] = {0, 0, 0, 0, 0}, pa[5] = {0, 0, 0, 0, 0};
        if (dependentW) {
            const int s = r >> 5, lane = r & 31, base = A.slice_off[s], width = A.slice_w[s];
            for (int k = 0; k < width; ++k) {
                const size_t slot = (size_t)(base + k);
                const int c = A.col[slot * 32 + lane];
                if (c < 0) continue;
                const MT* v = A.val + slot * (32 * 25) + lane;
                MT m[25];
                double xv[5];
#pragma unroll
                for (int e = 0; e < 25; ++e) m[e] = v[e * 32];
#pragma unroll
                for (int j = 0; j < 5; ++j) xv[j] = W[5 * (size_t)c + j];
#pragma unroll
                for (int i = 0; i < 5; ++i)
#pragma unroll
                    for (int j = 0; j < 5; ++j) {
                        const double a = tod(m[5 * i + j]);
                        ax[i] += a * xv[j];
                        pa[i] += a * xb[j];
                    }
            }
        }
        double s1 = 0, s2 = 0;
#pragma unroll
        for (int c = 0; c < 5; ++c) {
            const double q = rhs[5 * (size_t)r + c], b = ax[c] + q;
            s1 += (ax[c] - pa[c]) * (ax[c] - pa[c]);
            s2 += (b - pa[c]) * (b - pa[c]);
            sum[1 + c] += fabs(q);
        }
        sum[0] += sqrt(s1) + sqrt(s2);
    }
#pragma unroll
    for (int c = 0; c < 6; ++c) {
        const double v = block_sum(sum[c]);
        if (threadIdx.x == 0) partial[blockIdx.x * 6 + c] = v;
    }
}

// block-Jacobi: dinv = inv(diagonal block), entry-major [25][N]
template <typename MT>
__global__ void k_dinv(SellMat<MT> A, MT* __restrict__ dinv) {
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= A.N) return;
    const MT* v = A.val + (size_t)A.slice_off[r >> 5] * (32 * 25) + (r & 31);
    double D[25], X[25];
#pragma unroll
    for (int e = 0; e < 25; ++e) D[e] = ld(v + e * 32);
    inv5(D, X);
#pragma unroll
    for (int e = 0; e < 25; ++e) st(&dinv[flat_e(r, e)], X[e]);
}

template <typename MT>
__global__ void k_jacobi(int N, const MT* __restrict__ dinv, const double* __restrict__ x, double* __restrict__ y,
                         const int* __restrict__ active) {
    if (active && !*active) return;
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= N) return;
    double xv[5] = {x[5 * r], x[5 * r + 1], x[5 * r + 2], x[5 * r + 3], x[5 * r + 4]};
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        double a = 0;
#pragma unroll
        for (int j = 0; j < 5; ++j) a += ld(&dinv[flat_e(r, 5 * i + j)]) * xv[j];
        y[5 * r + i] = a;
    }
}

// held cells' rows of the block matrix -> identity (their update is zero;
// the right-hand side of those rows is zero through the residual mask)
template <typename MT>
__global__ void k_hold_rows(SellMat<MT> A, const unsigned char* __restrict__ mask) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= A.N || !mask[r]) return;
    const int sl = r >> 5, w = A.slice_w[sl];
    for (int k = 0; k < w; ++k) {
        const int fid = (A.slice_off[sl] + k) * 32 + (r & 31);
#pragma unroll
        for (int e = 0; e < 25; ++e) st(A.val + flat_e(fid, e), (k == 0 && e % 6 == 0) ? 1.0 : 0.0);
    }
}

// y += x (skipped when *active is 0)
__global__ void k_vadd(long n, const double* __restrict__ x, double* __restrict__ y, const int* __restrict__ active) {
    if (active && !*active) return;
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] += x[i];
}

template <typename MT>
__global__ void k_copy_identity(int n, const double* __restrict__ x, double* __restrict__ y, const int* __restrict__ active) {
    if (active && !*active) return;
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = x[i];
}

// ---------------------------------------------------------------- ILU(0)
// One CTA per subdomain.  Rows of a subdomain are contiguous and sorted by
// wavefront level, so each level is a contiguous row range processed in
// parallel with a CTA barrier between levels (exact ILU(0) within the
// subdomain, block-Jacobi between subdomains).  The factors are stored in
// a fixed-width sliced layout of their own: factor slot s (L_q: s = q < ml,
// U_q: s = ml + q) of row r has id fid = ((r/32)*(ml+mu) + s)*32 + r%32 and
// its entries at flat_e(fid, e); the Jacobian keeps its SELL layout.
struct IluDev {
    int n_parts;
    const int* part_lvl0;   // [n_parts+1] level index range of each part
    const int* lvl_off;     // [n_levels+1] row range of each level
    const int* nlu;         // [N] nl | nu << 8
    const int* low_start;   // [N+1] prefix of nl (first triple range of the row)
    const int* tr_start;    // [n_low+1]
    const int* tr_kj;       // factor id of U_kj
    const int* tr_rj;       // factor id of A_rj (-1: diagonal)
    int ml, mu;             // factor slots per row
    int mu_use;             // U slots the backward sweep applies (0: (D + L)^-1 of Gauss-Seidel)
    const int* lu_col;      // [fid] column of each factor slot (-1: empty)
    const int* lu_src;      // [fid] SELL flat slot of the same block in A
    // factor records of the apply (rdst_records.h; null: not kept): forward
    // and backward, their groups, the first group of each part, and the tasks.
    // Headers and columns are set once, the blocks after each factorisation.
    unsigned char* rec_f;
    unsigned char* rec_b;
    const RecGroup* grp_f;
    const RecGroup* grp_b;
    const int* part_gf;
    const int* part_gb;
    const RecTask* task_f;
    const RecTask* task_b;
    const int* part_tf;     // first forward task of each part
    // the direct factorisation's addressing (null: gather + factor
    // instead).  Per update triple (tr_start ranges):
    // fr_trk: where U_kj is read, the flat SELL slot of A_kj (>= 0), factor
    // id fid of the sliced store as -fid - 1 (row k takes updates of its
    // own), or INT_MIN (a fill block of a row without updates: zero);
    // fr_trt: -1 the diagonal, else the slot of row r that takes it.
    // fr_desc[low_start[r] + q]: (column k of L_q, flat SELL slot of A_rk or
    // -2 for a fill, fr_trk of the slot's first triple, its fr_trt + 2 or 0
    // for none, | 1 << 20 when more triples follow).
    // nlu bit 16: the row updates one of its own off-diagonal slots.
    const int* fr_trk;
    const int* fr_trt;
    const int4* fr_desc;
};

__device__ __forceinline__ int lu_fid(int r, int s, int ms) { return ((r >> 5) * ms + s) * 32 + (r & 31); }

constexpr int ILU_TPB = 128;

// same-subdomain blocks of A -> factor storage (fully parallel, before the
// level-scheduled factorisation); fill slots outside the matrix pattern
// (lu_src -2) restart from zero, empty slots (-1) stay zero
template <typename MT>
__global__ void k_ilu_gather(SellMat<MT> A, MT* __restrict__ lu, const int* __restrict__ lu_src, int n_fid) {
    const int fid = blockIdx.x * blockDim.x + threadIdx.x;
    if (fid >= n_fid) return;
    const int src = lu_src[fid];
    if (src == -1) return;
    if (src < 0) {
#pragma unroll
        for (int e = 0; e < 25; ++e) lu[flat_e(fid, e)] = mt_zero<MT>();
        return;
    }
#pragma unroll
    for (int e = 0; e < 25; ++e) lu[flat_e(fid, e)] = A.val[flat_e(src, e)];
}

// Level-scheduled subdomain factorisation into the factor store: one CTA
// per subdomain, a thread per row of the current level, in the compute
// type of the storage (IluCT).
template <typename MT>
__global__ void __launch_bounds__(ILU_TPB) k_ilu_factor(SellMat<MT> A, MT* __restrict__ lu, MT* __restrict__ dinv,
                                                        IluDev P) {
    using CT = typename IluCT<MT>::T;
    const int part = blockIdx.x;
    const int ms = P.ml + P.mu;
    for (int l = P.part_lvl0[part]; l < P.part_lvl0[part + 1]; ++l) {
        for (int r = P.lvl_off[l] + threadIdx.x; r < P.lvl_off[l + 1]; r += blockDim.x) {
            const int nl = P.nlu[r] & 255;
            const MT* dv = A.val + (size_t)A.slice_off[r >> 5] * (32 * 25) + (r & 31);
            CT D[25];
#pragma unroll
            for (int e = 0; e < 25; ++e) D[e] = ct_ld(dv + e * 32);
            const int q0 = P.low_start[r];
            for (int q = 0; q < nl; ++q) {
                const int fq = lu_fid(r, q, ms);
                const int k = P.lu_col[fq];
                CT Ark[25], Dk[25], Lrk[25];
#pragma unroll
                for (int e = 0; e < 25; ++e) {
                    Ark[e] = ct_ld(lu + flat_e(fq, e));
                    Dk[e] = ct_ld(dinv + flat_e(k, e));
                }
#pragma unroll
                for (int i = 0; i < 5; ++i)
#pragma unroll
                    for (int j = 0; j < 5; ++j) {
                        CT a = 0;
#pragma unroll
                        for (int t = 0; t < 5; ++t) a += Ark[5 * i + t] * Dk[5 * t + j];
                        Lrk[5 * i + j] = a;
                    }
#pragma unroll
                for (int e = 0; e < 25; ++e) ct_st(lu + flat_e(fq, e), Lrk[e]);
                for (int t = P.tr_start[q0 + q]; t < P.tr_start[q0 + q + 1]; ++t) {
                    const int kj = P.tr_kj[t], rj = P.tr_rj[t];
                    CT U[25];
#pragma unroll
                    for (int e = 0; e < 25; ++e) U[e] = ct_ld(lu + flat_e(kj, e));
                    if (rj < 0) {
#pragma unroll
                        for (int i = 0; i < 5; ++i)
#pragma unroll
                            for (int j = 0; j < 5; ++j) {
                                CT a = 0;
#pragma unroll
                                for (int t2 = 0; t2 < 5; ++t2) a += Lrk[5 * i + t2] * U[5 * t2 + j];
                                D[5 * i + j] -= a;
                            }
                    } else {
#pragma unroll
                        for (int i = 0; i < 5; ++i)
#pragma unroll
                            for (int j = 0; j < 5; ++j) {
                                CT a = 0;
#pragma unroll
                                for (int t2 = 0; t2 < 5; ++t2) a += Lrk[5 * i + t2] * U[5 * t2 + j];
                                MT* p = lu + flat_e(rj, 5 * i + j);
                                ct_st(p, ct_ld(p) - a);
                            }
                    }
                }
            }
            CT X[25];
            inv5(D, X);
#pragma unroll
            for (int e = 0; e < 25; ++e) ct_st(dinv + flat_e(r, e), X[e]);
        }
        __syncthreads();
    }
}

constexpr int ILU_APPLY_TPB = 128;
constexpr int ILU_APPLY_MINB = 4;      // resident CTAs per SM the register budget is sized for
constexpr int ILU_MAX_LV = 1023;       // level offsets staged in shared memory up to this many

// One row task of a sweep: the factor row's columns, this lane's entries
// of each slot, its pivot-inverse row (backward sweep) and the starting
// value of y.  Tasks are loaded one ahead of use, so their global loads
// are in flight across the previous task and its barrier; only the loads
// of x (rows finished in earlier levels) stay on the level-to-level chain.
template <typename MT, int NB>
struct IluTask {
    int cq[NB];
    MT v[NB][5];
    MT di[5];
    double y0;
};

template <typename MT, int NB, bool BACK>
__device__ __forceinline__ void ilu_load_task(IluTask<MT, NB>& t, const MT* __restrict__ lu,
                                              const MT* __restrict__ dinv, const int* __restrict__ lu_col,
                                              const double* y_src, int r, bool act, int comp, int s0, int ns,
                                              int ms) {
#pragma unroll
    for (int q = 0; q < NB; ++q) {
        const bool ok = act && q < ns;
        const int fid = ok ? lu_fid(r, s0 + q, ms) : 0;
        t.cq[q] = ok ? lu_col[fid] : -1;
        // empty factor slots hold zeros: the value loads do not wait for the column
#pragma unroll
        for (int j = 0; j < 5; ++j) t.v[q][j] = ok ? lu[flat_e(fid, 5 * comp + j)] : mt_zero<MT>();
    }
    if (BACK) {
#pragma unroll
        for (int j = 0; j < 5; ++j) t.di[j] = act ? dinv[flat_e(r, 5 * comp + j)] : mt_zero<MT>();
    }
    t.y0 = act ? y_src[5 * r + comp] : 0.0;
}

// Tasks of one sweep in order: level by level (forward ascending, backward
// descending), rpp rows per task.  The cursor is uniform over the CTA.
struct IluCursor {
    int l, base;
};

// x = (LU)^-1 b on each subdomain: one CTA per part walks the part's
// wavefront levels forward (x = L^-1 b, unit diagonal) and backward
// (x = U^-1 x with the stored pivot inverses), a barrier between levels.
// Five lanes per row (one per component), six rows per warp.  PF tasks
// are loaded ahead of the one being computed (two with 4- or 2-byte
// factors, one with 8-byte ones: the register budget of four CTAs per SM).
template <typename MT, int NB>
__global__ void __launch_bounds__(ILU_APPLY_TPB, ILU_APPLY_MINB)
    k_ilu_apply(int N, const MT* __restrict__ lu, const MT* __restrict__ dinv, IluDev P,
                const double* __restrict__ b, double* x, const int* __restrict__ active) {
    constexpr int PF = sizeof(MT) < 8 ? 2 : 1;
    if (active && !*active) return;
    __shared__ int s_off[ILU_MAX_LV + 1];
    const int part = blockIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rsub = lane / 5, comp = lane - 5 * (lane / 5);
    const bool lane_ok = lane < 30;
    const int rpp = (blockDim.x >> 5) * 6;
    const int l0 = P.part_lvl0[part], l1 = P.part_lvl0[part + 1];
    const int ml = P.ml, mu = P.mu, ms = ml + mu;
    const bool staged = l1 - l0 <= ILU_MAX_LV;
    if (staged)
        for (int i = threadIdx.x; i <= l1 - l0; i += blockDim.x) s_off[i] = P.lvl_off[l0 + i];
    __syncthreads();
    auto off = [&](int l) { return staged ? s_off[l - l0] : P.lvl_off[l]; };

#pragma unroll 1
    for (int sweep = 0; sweep < 2; ++sweep) {
        const bool back = sweep == 1;
        const int dir = back ? -1 : 1;
        const int s0 = back ? ml : 0, ns = back ? P.mu_use : ml;
        const double* ysrc = back ? x : b;
        IluCursor cur{back ? l1 - 1 : l0, 0};
        auto in_range = [&](int l) { return back ? l >= l0 : l < l1; };
        // task queue: slot 0 is computed, slots 1..PF are in flight
        IluTask<MT, NB> q[PF + 1];
        int rq[PF + 1];
        bool aq[PF + 1], eq[PF + 1], vq[PF + 1];
        auto next = [&](int d) {
            vq[d] = in_range(cur.l);
            rq[d] = 0; aq[d] = false; eq[d] = false;
            if (vq[d]) {
                const int r0 = off(cur.l), n = off(cur.l + 1) - r0;
                rq[d] = r0 + cur.base + warp * 6 + rsub;
                aq[d] = lane_ok && cur.base + warp * 6 + rsub < n;
                cur.base += rpp;
                eq[d] = cur.base >= n;
                if (eq[d]) { cur.l += dir; cur.base = 0; }
            }
            if (back) ilu_load_task<MT, NB, true>(q[d], lu, dinv, P.lu_col, ysrc, rq[d], aq[d], comp, s0, ns, ms);
            else ilu_load_task<MT, NB, false>(q[d], lu, dinv, P.lu_col, ysrc, rq[d], aq[d], comp, s0, ns, ms);
        };
#pragma unroll
        for (int d = 0; d < PF; ++d) next(d);
        while (vq[0]) {
            next(PF);
            double y = q[0].y0;
            if (aq[0]) {
#pragma unroll
                for (int k = 0; k < NB; ++k) {
                    if (q[0].cq[k] >= 0) {
                        const double* xk = x + 5 * q[0].cq[k];
#pragma unroll
                        for (int j = 0; j < 5; ++j) y -= tod(q[0].v[k][j]) * xk[j];
                    }
                }
            }
            if (back) {
                // x_r = inv(U_rr) y: gather the row's five components by
                // shuffle (all lanes take part)
                double a = 0.0;
#pragma unroll
                for (int j = 0; j < 5; ++j) {
                    const double yj = __shfl_sync(0xffffffffu, y, (lane_ok ? 5 * rsub : 0) + j);
                    a += tod(q[0].di[j]) * yj;
                }
                y = a;
            }
            if (aq[0]) x[5 * rq[0] + comp] = y;
            if (eq[0]) __syncthreads();
#pragma unroll
            for (int d = 0; d < PF; ++d) {
                q[d] = q[d + 1]; rq[d] = rq[d + 1]; aq[d] = aq[d + 1]; eq[d] = eq[d + 1]; vq[d] = vq[d + 1];
            }
        }
    }
}

constexpr int ILU_FR_MAXQ = 8;      // lower slots per row the direct factorisation takes

// one IKJ update triple of row r: U_kj read from A (us >= 0), the sliced
// factor store (fid -us - 1) or zero (INT_MIN); L_rk U_kj taken from the
// diagonal (tgt < 0) or from slot tgt of the row in the factor store
template <typename MT, typename CT>
__device__ __forceinline__ void ilu_fr_update(const SellMat<MT>& A, MT* __restrict__ lu, int r, int ms,
                                              const CT (&Lrk)[25], CT (&D)[25], int us, int tgt) {
    CT U[25];
    if (us >= 0) {
#pragma unroll
        for (int e = 0; e < 25; ++e) U[e] = ct_ld(A.val + flat_e(us, e));
    } else if (us != INT_MIN) {
#pragma unroll
        for (int e = 0; e < 25; ++e) U[e] = ct_ld(lu + flat_e(-us - 1, e));
    } else {
#pragma unroll
        for (int e = 0; e < 25; ++e) U[e] = CT(0);
    }
    if (tgt < 0) {
#pragma unroll
        for (int i = 0; i < 5; ++i)
#pragma unroll
            for (int j = 0; j < 5; ++j) {
                CT a = 0;
#pragma unroll
                for (int t2 = 0; t2 < 5; ++t2) a += Lrk[5 * i + t2] * U[5 * t2 + j];
                D[5 * i + j] -= a;
            }
    } else {
        const int ft = lu_fid(r, tgt, ms);
#pragma unroll
        for (int i = 0; i < 5; ++i)
#pragma unroll
            for (int j = 0; j < 5; ++j) {
                CT a = 0;
#pragma unroll
                for (int t2 = 0; t2 < 5; ++t2) a += Lrk[5 * i + t2] * U[5 * t2 + j];
                MT* pe = lu + flat_e(ft, 5 * i + j);
                ct_st(pe, ct_ld(pe) - a);
            }
    }
}

// The subdomain factorisations with the blocks of A read where they lie
// (no gather; the bulk apply's records are written by k_ilu_pack after it):
// one CTA (one warp) per subdomain, a thread per row of the current
// wavefront level, in the compute type of the storage (IluCT: FP32 for FP32
// and BF16 factors).  Row r forms L_rk = A_rk D_k^-1 and the IKJ updates
// from its blocks of A and, of earlier rows, the pivot inverses (dinv) and
// U blocks (A itself, or the factor store for rows whose own blocks take
// updates: those rows first copy their blocks of A there), and stores L and
// its pivot inverse in the sliced factor store, lanes side by side.  The
// addressing of each lower slot is one 16-byte descriptor (fr_desc), all
// read at the row's start.  Same operations, order and roundings as
// k_ilu_gather + k_ilu_factor.
template <typename MT>
__global__ void __launch_bounds__(32) k_ilu_factor_direct(SellMat<MT> A, MT* __restrict__ lu,
                                                          MT* __restrict__ dinv, IluDev P) {
    using CT = typename IluCT<MT>::T;
    __shared__ int s_off[ILU_MAX_LV + 1];
    const int ln = threadIdx.x;
    const int ms = P.ml + P.mu;
    const int part = blockIdx.x;
    const int l0 = P.part_lvl0[part], l1 = P.part_lvl0[part + 1];
    const bool staged = l1 - l0 <= ILU_MAX_LV;
    if (staged)
        for (int i = ln; i <= l1 - l0; i += 32) s_off[i] = P.lvl_off[l0 + i];
    __syncwarp();
    auto off = [&](int l) { return staged ? s_off[l - l0] : P.lvl_off[l]; };
    for (int l = l0; l < l1; ++l) {
        const int end = off(l + 1);
        for (int base = off(l); base < end; base += 32) {
            const int r = base + ln;
            if (r < end) {
                const int nlu = P.nlu[r];
                const int q0 = P.low_start[r];
                const int nl = nlu & 255;
                const int nu = P.mu_use ? (nlu >> 8) & 255 : 0;
                const bool upd = (nlu >> 16) & 1;
                int4 dsc[ILU_FR_MAXQ];
#pragma unroll
                for (int q = 0; q < ILU_FR_MAXQ; ++q)
                    if (q < nl) dsc[q] = P.fr_desc[q0 + q];
                const MT* dv = A.val + (size_t)A.slice_off[r >> 5] * (32 * 25) + (r & 31);
                CT D[25];
#pragma unroll
                for (int e = 0; e < 25; ++e) D[e] = ct_ld(dv + e * 32);
                // a row that updates its own blocks takes them from A into
                // the factor store first (zero where ILU(p) fills)
                if (upd) {
                    for (int sl = 0; sl < nl + nu; ++sl) {
                        const int f = lu_fid(r, sl < nl ? sl : P.ml + sl - nl, ms);
                        const int src = P.lu_src[f];
#pragma unroll
                        for (int e = 0; e < 25; ++e) lu[flat_e(f, e)] = src >= 0 ? A.val[flat_e(src, e)] : mt_zero<MT>();
                    }
                }
#pragma unroll
                for (int q = 0; q < ILU_FR_MAXQ; ++q) {
                    if (q < nl) {
                        const int k = dsc[q].x, sl = dsc[q].y, us0 = dsc[q].z, tw = dsc[q].w;
                        const int fq = lu_fid(r, q, ms);
                        CT Ark[25], Dk[25], Lrk[25];
                        if (upd) {
#pragma unroll
                            for (int e = 0; e < 25; ++e) Ark[e] = ct_ld(lu + flat_e(fq, e));
                        } else {
#pragma unroll
                            for (int e = 0; e < 25; ++e) Ark[e] = sl >= 0 ? ct_ld(A.val + flat_e(sl, e)) : CT(0);
                        }
#pragma unroll
                        for (int e = 0; e < 25; ++e) Dk[e] = ct_ld(dinv + flat_e(k, e));
#pragma unroll
                        for (int i = 0; i < 5; ++i)
#pragma unroll
                            for (int j = 0; j < 5; ++j) {
                                CT a = 0;
#pragma unroll
                                for (int t = 0; t < 5; ++t) a += Ark[5 * i + t] * Dk[5 * t + j];
                                Lrk[5 * i + j] = a;
                            }
#pragma unroll
                        for (int e = 0; e < 25; ++e) ct_st(lu + flat_e(fq, e), Lrk[e]);
                        // update triples: the first rides in the descriptor (w:
                        // its target slot + 2, 0 none; bit 20: more follow)
                        const int tfirst = (tw & 0xfffff) - 2;
                        if (tfirst >= -1) ilu_fr_update(A, lu, r, ms, Lrk, D, us0, tfirst);
                        if (tw >> 20) {
                            for (int t = P.tr_start[q0 + q] + 1; t < P.tr_start[q0 + q + 1]; ++t)
                                ilu_fr_update(A, lu, r, ms, Lrk, D, P.fr_trk[t], P.fr_trt[t]);
                        }
                    }
                }
                CT X[25];
                inv5(D, X);
#pragma unroll
                for (int e = 0; e < 25; ++e) ct_st(dinv + flat_e(r, e), X[e]);
            }
            __syncwarp();
        }
    }
}

// ---- ILU apply with the factor records brought in by bulk copies
//
// x = (L U)^-1 b on each subdomain: one CTA walks the subdomain's wavefront
// levels forward (unit L) and backward (U with the stored pivot inverses).
// What bounds it is the chain of levels: each one reads the x of the level
// before, multiplies and hands its own on, and a warp by itself spends three
// quarters of a task's ~900 cycles on fetching the task.  So everything that
// does not depend on the previous level is taken off that chain:
//  * a producer warp brings the records (rdst_records.h), a group of tasks
//    per cp.async.bulk, into one of two shared-memory stages, and the
//    starting values (b forward, the forward result backward) of the
//    group's rows by coalesced cp.async; both complete on the stage's "full"
//    mbarrier, the compute warps return the stage on its "empty" one;
//  * the tasks, six rows each, go round the W compute warps, and a warp
//    brings its next task's columns, block rows (whole 16-byte words,
//    conflict-free) and starting value into registers while the others walk
//    the levels before it;
//  * a level's end is a named barrier (one id per level in turn) on which a
//    warp only arrives, except for the one level that its next task reads.
// What is left between two levels is the load of the previous level's x
// from the level buffers (two, by level parity), five multiply-adds per
// block, backward the pivot product by shuffles, and the store, without a
// branch: a row short of NB blocks multiplies zeros with the buffers' row of
// zeros.
//
// Five lanes a row (one per component).  The lanes multiply in CT, the
// arithmetic of the factors' storage type (FP64 in double, FP32 and BF16 in
// float); input b and output x stay FP64 vectors.  Each block's product with
// x_k is summed first, then subtracted from y, block by block in column
// order.  Blocks beyond the first NB of a row (rare) are read from the stage
// when they are needed (EXT).
//
// TIGHT: three compute warps (two with FP64) and the registers of six CTAs an
// SM.
//
// Every mbarrier wait is bounded (wait_ms of globaltimer).  A compute warp whose
// wait expires raises bit 2 of the flags (reported as a timeout by the host) and
// computes no more, but takes all that is left of the level barriers of both
// sweeps (rec_give_up): bar.sync has no bound of its own, so no barrier may
// miss a warp.  The others find their own waits expired in turn, and the
// producer waits, bounded by 2 s, for its copies in flight.
__device__ __forceinline__ unsigned long long globaltimer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// global -> shared bulk copy completing on an mbarrier (no multicast)
__device__ __forceinline__ void bulk_g2s(unsigned dst, const void* src, unsigned bytes, unsigned bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try(unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// true once the phase of parity `parity` has completed; false after wait_ms
// (0: at once)
__device__ __noinline__ bool mbar_wait_for(unsigned bar, unsigned parity, unsigned wait_ms) {
    const unsigned long long t0 = globaltimer_ns();
    while (wait_ms) {
        for (int it = 0; it < 64; ++it)
            if (mbar_try(bar, parity)) return true;
        if (globaltimer_ns() - t0 > wait_ms * 1000000ull) break;
    }
    return false;
}
// the CTA's limit: kept here, since an argument more of the call below would
// cost the compute warps a register that the tight instances do not have
__shared__ unsigned s_wait_ms;
__device__ __noinline__ bool mbar_wait_slow(unsigned bar, unsigned parity) {
    return mbar_wait_for(bar, parity, s_wait_ms);
}
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity) {
    return mbar_try(bar, parity) || mbar_wait_slow(bar, parity);
}
// A bounded wait of a solver kernel has expired: bit 2 of the flags, which the
// host reports, and nothing left to do for the rest of the solve (the launches
// that follow would wait out the limit in turn, or go on with half sums).
__device__ __forceinline__ void wait_expired(Scalars* sc) {
    atomicOr(&sc->flags, 4);
    sc->gm_active = sc->gm_used = sc->bi_active = 0;
    sc->converged = 1;
}
__device__ __forceinline__ void cpa8(unsigned dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst), "l"(src) : "memory");
}
// the calling thread's cp.async so far count as one of the arrivals of bar
__device__ __forceinline__ void cpa_arrive(unsigned bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(bar) : "memory");
}

// Shared-memory loads and stores by 32-bit address.  They are issued in
// program order (volatile), so a task's loads go out together ahead of the
// arithmetic; `ok` false: zeros, no load.
__device__ __forceinline__ uint4 lds4(unsigned a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ unsigned lds1(unsigned a) {
    unsigned v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ unsigned lds_byte(unsigned a) {
    unsigned v;
    asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ double lds_double(unsigned a) {
    double v;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ void sts(unsigned a, double v) { asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory"); }
__device__ __forceinline__ void sts(unsigned a, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory"); }
// level-buffer row: five values padded to 16 bytes (6 doubles / 8 floats)
template <typename CT> constexpr int lb_row_bytes() { return sizeof(CT) == 8 ? 48 : 32; }
__device__ __forceinline__ void lb_load(unsigned a, double (&o)[5]) {
    asm volatile("ld.shared.v2.f64 {%0,%1}, [%2];" : "=d"(o[0]), "=d"(o[1]) : "r"(a) : "memory");
    asm volatile("ld.shared.v2.f64 {%0,%1}, [%2];" : "=d"(o[2]), "=d"(o[3]) : "r"(a + 16) : "memory");
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(o[4]) : "r"(a + 32) : "memory");
}
__device__ __forceinline__ void lb_load(unsigned a, float (&o)[5]) {
    asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(o[0]), "=f"(o[1]), "=f"(o[2]), "=f"(o[3]) : "r"(a) : "memory");
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(o[4]) : "r"(a + 16) : "memory");
}
// one row of five entries of a record's values: word `idx` of the task's
// 5 * tot (rdst_records.h)
__device__ __forceinline__ void rec_load(unsigned v, int tot, int idx, bool ok, double (&o)[5], double) {
    asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %5, 0;\n mov.f64 %0, 0d0000000000000000;\n"
                 " mov.f64 %1, %0;\n mov.f64 %2, %0;\n mov.f64 %3, %0;\n mov.f64 %4, %0;\n"
                 " @p ld.shared.v2.f64 {%0,%1}, [%6];\n @p ld.shared.v2.f64 {%2,%3}, [%7];\n @p ld.shared.f64 %4, [%8];\n}"
                 : "=&d"(o[0]), "=&d"(o[1]), "=&d"(o[2]), "=&d"(o[3]), "=&d"(o[4])
                 : "r"((unsigned)ok), "r"(v + 16 * idx), "r"(v + 80 * tot + 16 * idx), "r"(v + 160 * tot + 8 * idx));
}
__device__ __forceinline__ void rec_load(unsigned v, int tot, int idx, bool ok, float (&o)[5], float) {
    asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %5, 0;\n mov.f32 %0, 0f00000000;\n"
                 " mov.f32 %1, %0;\n mov.f32 %2, %0;\n mov.f32 %3, %0;\n mov.f32 %4, %0;\n"
                 " @p ld.shared.v4.f32 {%0,%1,%2,%3}, [%6];\n @p ld.shared.f32 %4, [%7];\n}"
                 : "=&f"(o[0]), "=&f"(o[1]), "=&f"(o[2]), "=&f"(o[3]), "=&f"(o[4])
                 : "r"((unsigned)ok), "r"(v + 16 * idx), "r"(v + 80 * tot + 4 * idx));
}
__device__ __forceinline__ void rec_load(unsigned v, int tot, int idx, bool ok, float (&o)[5], __nv_bfloat16) {
    unsigned a, b, c;
    asm volatile("{\n .reg .pred p;\n .reg .u16 h;\n setp.ne.u32 p, %3, 0;\n mov.u32 %0, 0;\n mov.u32 %1, 0;\n"
                 " mov.u16 h, 0;\n @p ld.shared.v2.u32 {%0,%1}, [%4];\n @p ld.shared.u16 h, [%5];\n cvt.u32.u16 %2, h;\n}"
                 : "=&r"(a), "=&r"(b), "=&r"(c)
                 : "r"((unsigned)ok), "r"(v + 8 * idx), "r"(v + 40 * tot + 2 * idx));
    o[0] = __uint_as_float(a << 16); o[1] = __uint_as_float(a & 0xffff0000u);
    o[2] = __uint_as_float(b << 16); o[3] = __uint_as_float(b & 0xffff0000u);
    o[4] = __uint_as_float(c << 16);
}
// the same words written by the pack
__device__ __forceinline__ void rec_store(unsigned char* v, int tot, int idx, const double (&o)[5]) {
    *reinterpret_cast<double2*>(v + 16 * (size_t)idx) = make_double2(o[0], o[1]);
    *reinterpret_cast<double2*>(v + 80 * (size_t)tot + 16 * (size_t)idx) = make_double2(o[2], o[3]);
    *reinterpret_cast<double*>(v + 160 * (size_t)tot + 8 * (size_t)idx) = o[4];
}
__device__ __forceinline__ void rec_store(unsigned char* v, int tot, int idx, const float (&o)[5]) {
    *reinterpret_cast<float4*>(v + 16 * (size_t)idx) = make_float4(o[0], o[1], o[2], o[3]);
    *reinterpret_cast<float*>(v + 80 * (size_t)tot + 4 * (size_t)idx) = o[4];
}
__device__ __forceinline__ void rec_store(unsigned char* v, int tot, int idx, const __nv_bfloat16 (&o)[5]) {
    uint2 a;
    a.x = (unsigned)__bfloat16_as_ushort(o[0]) | (unsigned)__bfloat16_as_ushort(o[1]) << 16;
    a.y = (unsigned)__bfloat16_as_ushort(o[2]) | (unsigned)__bfloat16_as_ushort(o[3]) << 16;
    *reinterpret_cast<uint2*>(v + 8 * (size_t)idx) = a;
    *reinterpret_cast<unsigned short*>(v + 40 * (size_t)tot + 2 * (size_t)idx) = __bfloat16_as_ushort(o[4]);
}

// the plan's headers and columns -> the start of each group of the records
// (once, when the context is built: a CTA per group)
__global__ void k_rec_meta(const RecGroup* __restrict__ grp, const RecMeta* __restrict__ gm,
                           const uint4* __restrict__ meta, uint4* __restrict__ rec) {
    const RecMeta m = gm[blockIdx.x];
    for (unsigned q = threadIdx.x; q < m.n16; q += blockDim.x)
        rec[(size_t)grp[blockIdx.x].off16 + q] = meta[(size_t)m.off16 + q];
}

// factor blocks -> records (after each factorisation): a warp per task, lane
// (position, component) as the apply reads it, so that every store of a slot
// fills whole sectors of the record; the reads of the sliced stores are 6-row
// pieces of lines that the neighbouring warps share.  L comes from the factor
// store, U from A (from the factor store for rows whose own blocks take
// updates, zero for a fill), backward first the pivot inverse.  There is no
// factor store (lu null) after k_ilu_factor_rec: nf is 0 and no row's own blocks
// take updates.
template <typename MT>
__global__ void __launch_bounds__(256) k_ilu_pack(int nf, int nb, SellMat<MT> A, const MT* __restrict__ lu,
                                                  const MT* __restrict__ dinv, IluDev P) {
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (w >= nf + nb) return;
    const bool back = w >= nf;
    unsigned char* rec = back ? P.rec_b : P.rec_f;
    const RecTask t = back ? P.task_b[w - nf] : P.task_f[w];
    const uint4 h = *reinterpret_cast<const uint4*>(rec + (size_t)t.head16 * 16);
    const uint4 g = *reinterpret_cast<const uint4*>(rec + (size_t)t.head16 * 16 + 16);
    const int n = (int)(h.y & 255u), S = (int)((h.y >> 8) & 255u), tot = (int)(h.w >> 16);
    const int pos = lane / 5, comp = lane - 5 * pos;
    if (lane >= 30 || pos >= n) return;
    unsigned char* v = rec + (size_t)t.group16 * 16 + 16 * (size_t)(h.x >> 16);
    const unsigned char* nks = rec + (size_t)t.group16 * 16 + 16 * ((size_t)(h.x & 0xffffu) + n * ((S + 3) >> 2));
    const int r = (int)h.z + (int)((pos < 4 ? g.y >> (8 * pos) : g.z >> (8 * (pos - 4))) & 255u);
    const int ms = P.ml + P.mu;
    auto copy = [&](const MT* src, int blk) {       // src: entry 0 of the block, entries 32 apart
        MT o[5];
#pragma unroll
        for (int j = 0; j < 5; ++j) o[j] = src ? src[(5 * comp + j) * 32] : mt_zero<MT>();
        rec_store(v, tot, 5 * blk + comp, o);
    };
    if (back) copy(dinv + flat_e(r, 0), pos);
    const bool own_u = back && ((P.nlu[r] >> 16) & 1);
    int blk = (back ? n : 0) + pos;
#pragma unroll 4
    for (int k = 0; k < S; ++k) {
        const int nk = k < 4 ? (int)((g.x >> (8 * k)) & 255u) : (int)nks[k];
        if (pos < nk) {
            const int f = lu_fid(r, back ? P.ml + k : k, ms);
            const int a = back && !own_u ? P.lu_src[f] : 0;
            copy(back && !own_u ? (a >= 0 ? A.val + flat_e(a, 0) : nullptr) : lu + flat_e(f, 0), blk);
        }
        blk += nk;
    }
}

// ---- the factorisation on the apply's tasks
//
// Where no row updates blocks of its own (no three cells of a subdomain are
// pairwise neighbours: quads, hexahedra, the Kuhn tetrahedra and prisms; and
// Gauss-Seidel, which updates nothing) row r of the factorisation is
//   L_rk = A_rk D_k,  D_r = (A_rr - sum_k L_rk A_kr)^-1   over its lower k,
// a chain of levels like the apply's, and it takes the forward sweep's tasks
// in the same way: six rows a warp, five lanes a row (lane i: block row i),
// the W warps taking turns, a named barrier per level.  Before its level a
// warp has the rows of A_rr and A_rk in registers and the blocks A_kr in
// shared memory; what waits for the level before is D_k from the level
// buffers (25 entries a row, by level parity; LBUF false: from global memory
// where the buffers do not fit), the two products and the inverse.  The
// inverse is the Gauss-Jordan elimination of inv5 with the rows on five
// lanes: the pivot row travels by shuffle, row swaps are a change of labels.
// L goes straight into the forward records, so only the backward ones are
// packed afterwards.  Same operations and roundings as k_ilu_factor_direct
// (a row in one thread, ~7,000 cycles a level), which stays for the patterns
// with triangles or fill.  Factorisation and pack, us: 257x65 airfoil FP64 218
// -> 100, RAE2822 334 -> 166, 442 k-cell wing FP64 968 -> 540, 371 k BF16 746 ->
// 301; 1.2 M FP32 (three warps a CTA, six CTAs an SM) 1232 -> 1225.
template <typename MT, int NBP, bool TIGHT, bool LBUF>
__global__ void __launch_bounds__(TIGHT ? 96 : 256, TIGHT ? 6 : 2)
    k_ilu_factor_rec(SellMat<MT> A, MT* dinv, IluDev P) {
    using CT = typename IluCT<MT>::T;
    constexpr int RS = sizeof(CT) == 8 ? 26 : 28;           // 25 entries padded to 16 bytes
    constexpr int NBAR = TIGHT ? 4 : 15;                    // as in k_ilu_apply_rec
    extern __shared__ __align__(16) unsigned char s_fac[];
    CT* s_u = reinterpret_cast<CT*>(s_fac);                 // [W][6][NBP][RS]
    const int part = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, W = blockDim.x >> 5;
    CT* s_d = s_u + (size_t)W * REC_ROWS * NBP * RS;        // [2 lb_rows][RS]
    const int rsub = lane / 5, comp = lane - 5 * rsub, sbase = lane < 30 ? 5 * rsub : 0;
    const int pos0 = lane < 30 ? rsub : 0x7fffffff;
    const int nlev = P.part_lvl0[part + 1] - P.part_lvl0[part];
    const int t1 = P.part_tf[part + 1];
    int arrived = 0, bid = 1;
    auto arrive = [&] {
        if (W > 1) {
            if (!TIGHT) asm volatile("bar.arrive %0, %1;" ::"r"(bid), "r"(W * 32) : "memory");
            else if (bid == 1) asm volatile("bar.arrive 1, %0;" ::"r"(W * 32) : "memory");
            else if (bid == 2) asm volatile("bar.arrive 2, %0;" ::"r"(W * 32) : "memory");
            else if (bid == 3) asm volatile("bar.arrive 3, %0;" ::"r"(W * 32) : "memory");
            else asm volatile("bar.arrive 4, %0;" ::"r"(W * 32) : "memory");
        }
        bid = bid == NBAR ? 1 : bid + 1;
        ++arrived;
    };
    auto await = [&] {
        if (W > 1) {
            if (!TIGHT) asm volatile("bar.sync %0, %1;" ::"r"(bid), "r"(W * 32) : "memory");
            else if (bid == 1) asm volatile("bar.sync 1, %0;" ::"r"(W * 32) : "memory");
            else if (bid == 2) asm volatile("bar.sync 2, %0;" ::"r"(W * 32) : "memory");
            else if (bid == 3) asm volatile("bar.sync 3, %0;" ::"r"(W * 32) : "memory");
            else asm volatile("bar.sync 4, %0;" ::"r"(W * 32) : "memory");
        } else {
            __syncwarp();
        }
        bid = bid == NBAR ? 1 : bid + 1;
        ++arrived;
    };
    // the current task
    CT D[5], Ar[NBP][5];
    int cq[NBP], kq[NBP];
    int n = 0, S = 0, tot = 0, r = 0, dl = 0, own = 0, q0 = 0;
    unsigned nk4 = 0, last = 0;
    bool act = false, kept = false;
    unsigned char* vals = nullptr;
    const unsigned char *cols = nullptr, *nks = nullptr;
    bool upd[NBP];
    auto load = [&](int t) {
        const RecTask tk = P.task_f[t];
        const unsigned char* hp = P.rec_f + (size_t)tk.head16 * 16;
        const uint4 h = *reinterpret_cast<const uint4*>(hp), g = *reinterpret_cast<const uint4*>(hp + 16);
        n = (int)(h.y & 255u);
        S = (int)((h.y >> 8) & 255u);
        last = (h.y >> 16) & REC_WARP_LAST;
        dl = (int)(h.y >> 24);
        tot = (int)(h.w >> 16);
        nk4 = g.x;
        act = pos0 < n;
        const int pos = act ? pos0 : 0;
        cols = P.rec_f + (size_t)tk.group16 * 16 + 16 * (size_t)(h.x & 0xffffu);
        nks = cols + 16 * (size_t)(n * ((S + 3) >> 2));
        vals = P.rec_f + (size_t)tk.group16 * 16 + 16 * (size_t)(h.x >> 16);
        const int rid = (int)((pos < 4 ? g.y >> (8 * pos) : g.z >> (8 * (pos - 4))) & 255u);
        r = (int)h.z + rid;
        kept = (h.w & 0xffffu) != 0xffffu;
        own = (int)(h.w & 0xffffu) + rid;
        q0 = P.low_start[r];
        const int4 c4 = *reinterpret_cast<const int4*>(cols + 16 * pos);
        const int ca[4] = {c4.x, c4.y, c4.z, c4.w};
        const MT* dv = A.val + (size_t)A.slice_off[r >> 5] * (32 * 25) + (r & 31);
#pragma unroll
        for (int j = 0; j < 5; ++j) D[j] = ct_ld(dv + (5 * comp + j) * 32);
        CT* u = s_u + ((size_t)(warp * REC_ROWS + pos) * NBP) * RS + 5 * comp;
#pragma unroll
        for (int q = 0; q < NBP; ++q) {
            cq[q] = ca[q];
            upd[q] = false;
            kq[q] = -1;
            if (act && pos0 < (int)((nk4 >> (8 * q)) & 255u)) {
                const int4 d = P.fr_desc[q0 + q];
                kq[q] = d.x;
                upd[q] = (d.w & 0xfffff) != 0;
                const MT* a = A.val + flat_e(d.y, 5 * comp);
#pragma unroll
                for (int j = 0; j < 5; ++j) Ar[q][j] = ct_ld(a + j * 32);
                if (upd[q]) {
                    const MT* b = A.val + flat_e(d.z, 5 * comp);
#pragma unroll
                    for (int j = 0; j < 5; ++j) u[q * RS + j] = ct_ld(b + j * 32);
                }
            }
        }
        __syncwarp();
        return (int)(g.z >> 16);
    };
    // D_k of one lower neighbour: from the level buffer row of byte offset c
    // of the apply's buffers, or (far, or no buffers) from global memory
    auto pivot_of = [&](int c, int k, CT (&o)[25]) {
        if (LBUF && c >= 0) {
            const CT* p = s_d + (size_t)(c / (sizeof(CT) == 8 ? 48 : 32)) * RS;
            constexpr int V = 16 / (int)sizeof(CT);
            alignas(16) CT tmp[RS];
#pragma unroll
            for (int e = 0; e < RS; e += V)
                *reinterpret_cast<uint4*>(tmp + e) = *reinterpret_cast<const uint4*>(p + e);
#pragma unroll
            for (int e = 0; e < 25; ++e) o[e] = tmp[e];
        } else {
            const MT* p = dinv + flat_e(k, 0);
#pragma unroll
            for (int e = 0; e < 25; ++e) o[e] = ct_ld(p + e * 32);
        }
    };
    // L_rk = A_rk D_k (this lane's row), into the records too; then D -= L_rk U
    auto lower = [&](const CT (&a5)[5], const CT (&Dk)[25], int blk, CT (&L5)[5]) {
        MT o[5];
#pragma unroll
        for (int j = 0; j < 5; ++j) {
            CT a = 0;
#pragma unroll
            for (int t = 0; t < 5; ++t) a += a5[t] * Dk[5 * t + j];
            L5[j] = a;
            ct_st(&o[j], a);
        }
        rec_store(vals, tot, 5 * blk + comp, o);
    };
    auto update = [&](const CT (&L5)[5], auto u) {
#pragma unroll
        for (int j = 0; j < 5; ++j) {
            CT a = 0;
#pragma unroll
            for (int t = 0; t < 5; ++t) a += L5[t] * u(5 * t + j);
            D[j] -= a;
        }
    };
    int t = P.part_tf[part] + warp;
    if (t < t1) {
        const int level = load(t);
        while (arrived < level - 1) arrive();
        if (arrived < level) await();
        for (;;) {
            if (act) {
                int blk = pos0;
#pragma unroll
                for (int q = 0; q < NBP; ++q) {
                    const int nk = (int)((nk4 >> (8 * q)) & 255u);
                    if (pos0 < nk) {
                        CT Dk[25];
                        pivot_of(cq[q], kq[q], Dk);
                        CT L5[5];
                        lower(Ar[q], Dk, blk, L5);
                        const CT* u = s_u + ((size_t)(warp * REC_ROWS + pos0) * NBP + q) * RS;
                        if (upd[q]) update(L5, [&](int e) { return u[e]; });
                    }
                    blk += nk;
                }
                for (int q = NBP; q < S; ++q) {
                    const int nk = q < 4 ? (int)((nk4 >> (8 * q)) & 255u) : (int)nks[q];
                    if (pos0 < nk) {
                        const int4 d = P.fr_desc[q0 + q];
                        const int c = reinterpret_cast<const int*>(cols)[4 * ((q >> 2) * n + pos0) + (q & 3)];
                        CT Dk[25], a5[5], L5[5];
                        pivot_of(c, d.x, Dk);
#pragma unroll
                        for (int j = 0; j < 5; ++j) a5[j] = ct_ld(A.val + flat_e(d.y, 5 * comp + j));
                        lower(a5, Dk, blk, L5);
                        if (d.w & 0xfffff) update(L5, [&](int e) { return ct_ld(A.val + flat_e(d.z, e)); });
                    }
                    blk += nk;
                }
            }
            // X = D^-1: lane `comp` of a row holds row `row` of [D | I]; lane_of
            // packs the lane that holds each row, three bits each
            CT a[10];
#pragma unroll
            for (int j = 0; j < 5; ++j) { a[j] = D[j]; a[5 + j] = comp == j ? CT(1) : CT(0); }
            int row = comp;
            unsigned lane_of = 0u | 1u << 3 | 2u << 6 | 3u << 9 | 4u << 12;
#pragma unroll
            for (int c = 0; c < 5; ++c) {
                int p = c;
                CT best = CT(0);
#pragma unroll
                for (int q = c; q < 5; ++q) {
                    const CT v = fabs(__shfl_sync(0xffffffffu, a[c], sbase + (int)((lane_of >> (3 * q)) & 7u)));
                    if (q == c) best = v;
                    else if (v > best) { best = v; p = q; }
                }
                if (p != c) {
                    const unsigned lc = (lane_of >> (3 * c)) & 7u, lp = (lane_of >> (3 * p)) & 7u;
                    lane_of ^= (lc ^ lp) << (3 * c) | (lc ^ lp) << (3 * p);
                    row = row == c ? p : (row == p ? c : row);
                }
                const CT piv = CT(1) / a[c];
                const bool mine = row == c;
                const CT f = a[c];
                const int src = sbase + (int)((lane_of >> (3 * c)) & 7u);
#pragma unroll
                for (int j = c + 1; j < 10; ++j) {
                    if (mine) a[j] *= piv;
                    const CT pr = __shfl_sync(0xffffffffu, a[j], src);
                    if (!mine && f != CT(0)) a[j] -= f * pr;
                }
            }
            if (act) {
#pragma unroll
                for (int j = 0; j < 5; ++j) {
                    MT o;
                    ct_st(&o, a[5 + j]);
                    dinv[flat_e(r, 5 * row + j)] = o;
                    if (LBUF && kept) s_d[(size_t)own * RS + 5 * row + j] = ct_ld(&o);
                }
            }
            if (last) break;
            for (int q = 1; q < dl; ++q) arrive();
            const bool wait = dl > 0;
            t += W;
            __syncwarp();
            load(t);
            if (wait) await();
        }
    }
    while (arrived < nlev - 1) arrive();
}

// The level barriers of the W compute warps.  An SM has 64 barriers and a kernel
// that names one in a register reserves all 16, which would leave four CTAs an
// SM: the tight instance names its four.
template <bool TIGHT>
__device__ __forceinline__ void level_arrive(int id, int W) {
    if (!TIGHT) asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(W * 32) : "memory");
    else if (id == 1) asm volatile("bar.arrive 1, %0;" ::"r"(W * 32) : "memory");
    else if (id == 2) asm volatile("bar.arrive 2, %0;" ::"r"(W * 32) : "memory");
    else if (id == 3) asm volatile("bar.arrive 3, %0;" ::"r"(W * 32) : "memory");
    else asm volatile("bar.arrive 4, %0;" ::"r"(W * 32) : "memory");
}
template <bool TIGHT>
__device__ __forceinline__ void level_sync(int id, int W) {
    if (!TIGHT) asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(W * 32) : "memory");
    else if (id == 1) asm volatile("bar.sync 1, %0;" ::"r"(W * 32) : "memory");
    else if (id == 2) asm volatile("bar.sync 2, %0;" ::"r"(W * 32) : "memory");
    else if (id == 3) asm volatile("bar.sync 3, %0;" ::"r"(W * 32) : "memory");
    else asm volatile("bar.sync 4, %0;" ::"r"(W * 32) : "memory");
}
template <bool TIGHT>
__device__ __forceinline__ void level_give_up(RecBarriers<TIGHT> bar, int nlev, bool back, int W, Scalars* sc) {
    if ((threadIdx.x & 31) == 0) wait_expired(sc);
    rec_give_up(bar, nlev, back, [&] { level_sync<TIGHT>(bar.id, W); bar.next(); });
}

template <typename MT, int NB, bool EXT, bool TIGHT>
__global__ void __launch_bounds__(TIGHT ? (sizeof(MT) == 8 ? 96 : 128) : 288, TIGHT ? 6 : 2)
    k_ilu_apply_rec(IluDev P, const double* __restrict__ b, double* x, const int* __restrict__ active,
                    int stage_bytes, int y0_rows, int lb_rows, Scalars* sc, unsigned wait_ms) {
    using CT = typename IluCT<MT>::T;
    if (active && !*active) return;
    __shared__ __align__(8) unsigned long long s_bar[2 * REC_STAGES + 1];     // full, empty, forward done
    extern __shared__ __align__(128) unsigned char s_dyn[];
    const int part = blockIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int W = (int)(blockDim.x >> 5) - 1;
    double* s_y0 = reinterpret_cast<double*>(s_dyn + (size_t)REC_STAGES * stage_bytes);       // [REC_STAGES][5 y0_rows]
    unsigned char* s_lb = reinterpret_cast<unsigned char*>(s_y0 + (size_t)REC_STAGES * 5 * y0_rows);   // [2 lb_rows + 1]
    const unsigned full0 = (unsigned)__cvta_generic_to_shared(&s_bar[0]), empty0 = full0 + 8 * REC_STAGES;
    const unsigned fdone = empty0 + 8 * REC_STAGES;
    if (threadIdx.x == 0) {
        for (int k = 0; k < REC_STAGES; ++k) {
            mbar_init(full0 + 8 * k, 33);          // the record's expect_tx, and each producer lane's y0 copies
            mbar_init(empty0 + 8 * k, W);
        }
        mbar_init(fdone, W);
        s_wait_ms = wait_ms;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const int gf0 = P.part_gf[part], ngf = P.part_gf[part + 1] - gf0;
    const int gb0 = P.part_gb[part], ngb = P.part_gb[part + 1] - gb0;

    if (warp == W) {
        // ---------------- producer
        const unsigned stage0 = (unsigned)__cvta_generic_to_shared(s_dyn), y0s = (unsigned)__cvta_generic_to_shared(s_y0);
        int s = 0;
        unsigned ph = 0;                           // parity of the next fill of stage s
        unsigned used = 0, lastp = 0;              // stages that took a copy, parity of the last one
        bool ok = wait_ms != 0;                    // 0: no wait is granted
        auto record = [&](const RecGroup& g, const unsigned char* rec) {
            ok = __all_sync(0xffffffffu, mbar_wait(empty0 + 8 * s, ph ^ 1u));
            if (!ok) return;
            if (lane == 0) {
                mbar_expect_tx(full0 + 8 * s, g.bytes);
                bulk_g2s(stage0 + (unsigned)(s * stage_bytes), rec + (size_t)g.off16 * 16, g.bytes, full0 + 8 * s);
            }
            used |= 1u << s;
            lastp = (lastp & ~(1u << s)) | (ph << s);
        };
        auto start = [&](const RecGroup& g, int st, const double* src) {
            const double* p = src + 5 * (size_t)g.row0;
            const unsigned d = y0s + (unsigned)(st * 5 * y0_rows) * 8;
            for (int i = lane; i < 5 * g.nrows; i += 32) cpa8(d + 8 * i, p + i);
            cpa_arrive(full0 + 8 * st);
        };
        auto step = [&] { if (++s == REC_STAGES) { s = 0; ph ^= 1u; } };
        // the descriptors are read one group ahead: their latency would be
        // paid once per group otherwise
        RecGroup nx = P.grp_f[gf0], nb = P.grp_b[gb0];
        for (int g = 0; g < ngf && ok; ++g) {
            const RecGroup cur = nx;
            if (g + 1 < ngf) nx = P.grp_f[gf0 + g + 1];
            record(cur, P.rec_f);
            if (ok) { start(cur, s, b); step(); }
        }
        // the backward records may run ahead of the forward sweep, their
        // starting values not
        const int nahead = min(REC_STAGES, ngb);
        const int s_first = s;
        for (int g = 0; g < nahead && ok; ++g) {
            const RecGroup cur = nb;
            if (g + 1 < ngb) nb = P.grp_b[gb0 + g + 1];
            record(cur, P.rec_b);
            if (ok) step();
        }
        if (ok) ok = __all_sync(0xffffffffu, mbar_wait(fdone, 0));
        if (ok) {
            int st = s_first;
            for (int g = 0; g < nahead; ++g) {
                start(P.grp_b[gb0 + g], st, x);
                if (++st == REC_STAGES) st = 0;
            }
        }
        for (int g = nahead; g < ngb && ok; ++g) {
            const RecGroup cur = nb;
            if (g + 1 < ngb) nb = P.grp_b[gb0 + g + 1];
            record(cur, P.rec_b);
            if (ok) { start(cur, s, x); step(); }
        }
        // abandoned: copies still in flight land before the CTA's shared memory goes
        if (!ok && lane == 0) {
            wait_expired(sc);
            for (int d = 0; d < REC_STAGES; ++d)
                if ((used >> d) & 1u) mbar_wait_for(full0 + 8 * d, (lastp >> d) & 1u, 2000);
        }
        return;
    }

    // ---------------- compute warps
    constexpr unsigned LRB = lb_row_bytes<CT>();
    const int rsub = lane / 5, comp = lane - 5 * rsub;
    const int pos0 = lane < 30 ? rsub : 0x7fffffff;       // position in the task
    const int sbase = lane < 30 ? 5 * rsub : 0;
    const unsigned dyn = (unsigned)__cvta_generic_to_shared(s_dyn), lb = (unsigned)__cvta_generic_to_shared(s_lb);
    const unsigned y0a = (unsigned)__cvta_generic_to_shared(s_y0);
    const int nlev = P.part_lvl0[part + 1] - P.part_lvl0[part];
    // the row of zeros (every warp its own copy of the same zeros: no warp
    // reads it before it has written it)
    if (lane < (int)LRB / 4) sts(lb + 2 * lb_rows * LRB + 4 * lane, 0.0f);
    __syncwarp();
    int s = 0;                  // stage of the group the warp is in
    unsigned ph = 0;
    auto sweep = [&](auto back_tag, RecBarriers<TIGHT>& bar) -> bool {
        constexpr bool BACK = decltype(back_tag)::value;
        const int ngrp = BACK ? ngb : ngf;
        int grp = 0;                            // group in the sweep
        unsigned gn = 0;                        // the group's address
        bool held = false;                      // the group is not returned yet
        // end of a level on which nobody here waits, of the one before the next task's
        auto arrive = [&] { level_arrive<TIGHT>(bar.id, W); bar.next(); };
        auto await = [&] { level_sync<TIGHT>(bar.id, W); bar.next(); };
        auto enter = [&] {                      // the group in stage s has landed
            gn = dyn + (unsigned)(s * stage_bytes);
            held = true;
            return __all_sync(0xffffffffu, mbar_wait(full0 + 8 * s, ph)) != 0;
        };
        auto release = [&] {
            __syncwarp();
            if (held && lane == 0) mbar_arrive(empty0 + 8 * s);
            held = false;
        };
        auto next_group = [&] {
            release();
            if (++s == REC_STAGES) { s = 0; ph ^= 1u; }
            ++grp;
            return enter();
        };
        // the current task: what its rows need, in registers, and where its
        // blocks lie
        CT v[NB][5], di[5], y = CT(0);
        int cq[NB], r = 0, S = 0, tot = 0, n = 0, pos = 0;
        unsigned own = 0, fl = 0, cc = 0, cv = 0, nk4 = 0, way = 0;
        bool act = false, kept = false;
        auto load = [&](int t) {
            const uint4 h = lds4(gn + 16 + 32 * t), g = lds4(gn + 32 + 32 * t);
            n = (int)(h.y & 255u);
            S = (int)((h.y >> 8) & 255u);
            fl = h.y >> 16;
            tot = (int)(h.w >> 16);
            act = pos0 < n;
            pos = act ? pos0 : 0;
            cc = gn + 16 * (h.x & 0xffffu);
            cv = gn + 16 * (h.x >> 16);
            nk4 = g.x;
            way = g.w;
            const uint4 c4 = lds4(cc + 16 * pos);
            const int rid = (int)((pos < 4 ? g.y >> (8 * pos) : g.z >> (8 * (pos - 4))) & 255u);
            y = (CT)lds_double(y0a + 8u * (unsigned)(5 * (s * y0_rows + (int)(way >> 16) + rid) + comp));
            if (BACK) rec_load(cv, tot, 5 * pos + comp, act, di, MT());
            int blk = (BACK ? n : 0) + pos;
#pragma unroll
            for (int k = 0; k < NB; ++k) {
                const int nk = (int)((nk4 >> (8 * k)) & 255u);
                rec_load(cv, tot, 5 * blk + comp, pos0 < nk, v[k], MT());
                blk += nk;
            }
            const unsigned ca[4] = {c4.x, c4.y, c4.z, c4.w};
#pragma unroll
            for (int k = 0; k < NB; ++k) cq[k] = (int)ca[k];
            r = (int)h.z + rid;
            kept = act && (h.w & 0xffffu) != 0xffffu;
            own = lb + ((h.w & 0xffffu) + rid) * LRB + (unsigned)sizeof(CT) * comp;
            // a group whose last task of this warp is in registers goes back
            if (((way >> 8) & 255u) && (!EXT || S <= NB)) release();
            return (int)(g.z >> 16);
        };
        auto far_row = [&](int c, CT (&o)[5]) {
            const double* xk = x + 5 * (size_t)(-1 - c);
#pragma unroll
            for (int j = 0; j < 5; ++j) o[j] = (CT)xk[j];
        };
        auto product = [&](const CT (&m)[5], const CT (&xk)[5]) {
            CT t = m[0] * xk[0];
#pragma unroll
            for (int j = 1; j < 5; ++j) t += m[j] * xk[j];
            return t;
        };
        // ---- the warp's first task
        if (!enter()) return false;
        int first = warp, ntask = (int)lds1(gn + 8);
        if (first < ntask) {
            for (int T = (int)lds1(gn); first >= T; T = (int)lds1(gn)) {
                first -= T;
                if (!next_group()) return false;
            }
            const int level = load(first);
            while (bar.taken < level - 1) arrive();
            if (bar.taken < level) await();
            for (;;) {
                // ---- the chain: x of the level before, products, hand on
                CT part_k[NB];
                auto blocks = [&](auto far_tag) {
#pragma unroll
                    for (int k = 0; k < NB; ++k) {
                        CT xk[5];
                        lb_load(lb + (decltype(far_tag)::value ? max(cq[k], 0) : cq[k]), xk);
                        if (decltype(far_tag)::value && cq[k] < 0) far_row(cq[k], xk);
                        part_k[k] = product(v[k], xk);
                    }
                };
                if (fl & REC_FAR) blocks(std::true_type{});
                else blocks(std::false_type{});
#pragma unroll
                for (int k = 0; k < NB; ++k) y -= part_k[k];
                if (EXT && S > NB) {
                    int blk = (BACK ? n : 0) + pos;
#pragma unroll
                    for (int k = 0; k < NB; ++k) blk += (int)((nk4 >> (8 * k)) & 255u);
                    for (int k = NB; k < S; ++k) {
                        const int nk = k < 4 ? (int)((nk4 >> (8 * k)) & 255u) : (int)lds_byte(cc + 16 * n * ((S + 3) >> 2) + k);
                        const int c = (int)lds1(cc + 16 * ((k >> 2) * n + pos) + 4 * (k & 3));
                        CT xe[5], m[5];
                        lb_load(lb + max(c, 0), xe);
                        if (c < 0) far_row(c, xe);
                        rec_load(cv, tot, 5 * blk + comp, pos0 < nk, m, MT());
                        y -= product(m, xe);
                        blk += nk;
                    }
                }
                if (BACK) {
                    // x_r = inv(U_rr) y, the row's five components by shuffle
                    CT a = CT(0);
#pragma unroll
                    for (int j = 0; j < 5; ++j) a += di[j] * __shfl_sync(0xffffffffu, y, sbase + j);
                    y = a;
                }
                if (kept) sts(own, y);
                if (act) x[5 * (size_t)r + comp] = (double)y;
                if (fl & REC_WARP_LAST) break;
                // ---- on to the warp's next task
                const int dl = (int)(fl >> 8) & 255;
                for (int q = 1; q < dl; ++q) arrive();
                const int t = (int)(way & 255u);
                for (unsigned q = (way >> 8) & 255u; q > 0; --q)
                    if (!next_group()) return false;
                load(t);
                if (dl > 0) await();
            }
        }
        while (bar.taken < nlev - 1) arrive();
        if (!BACK) {
            __syncwarp();
            if (lane == 0) mbar_arrive(fdone);
        }
        // the groups of the other warps' last tasks pass by
        while (grp + 1 < ngrp)
            if (!next_group()) return false;
        release();
        if (++s == REC_STAGES) { s = 0; ph ^= 1u; }
        return true;
    };
    // a warp that gave up stays in step with the others, who may still run
    RecBarriers<TIGHT> forward(nlev, false);
    if (!sweep(std::false_type{}, forward)) { level_give_up(forward, nlev, false, W, sc); return; }
    RecBarriers<TIGHT> backward(nlev, true);
    if (!sweep(std::true_type{}, backward)) level_give_up(backward, nlev, true, W, sc);
}

// ---------------------------------------------------------------- vectors
// deterministic two-stage reductions: fixed grid -> partials -> one block
constexpr int RED_TPB = 256;
inline int red_blocks(long n) {
    long b = (n + RED_TPB * 4 - 1) / (RED_TPB * 4);
    if (b < 1) b = 1;
    if (b > 592) b = 592;           // 4 x 148 SMs
    return (int)b;
}

// Four consecutive entries of a vector as doubles (16-byte loads, p aligned
// to 16 bytes).
__device__ __forceinline__ void load4(const double* p, double (&o)[4]) {
    const double2 a = reinterpret_cast<const double2*>(p)[0], b = reinterpret_cast<const double2*>(p)[1];
    o[0] = a.x; o[1] = a.y; o[2] = b.x; o[3] = b.y;
}

// per-component sum |r_c| and the foam normFactor pieces
__global__ void __launch_bounds__(RED_TPB) k_abs5(int N, const double* __restrict__ r, double* __restrict__ partial) {
    double a[5] = {0, 0, 0, 0, 0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x)
#pragma unroll
        for (int c = 0; c < 5; ++c) a[c] += fabs(r[5 * i + c]);
#pragma unroll
    for (int c = 0; c < 5; ++c) {
        double v = block_sum(a[c]);
        if (threadIdx.x == 0) partial[blockIdx.x * 5 + c] = v;
    }
}

// sum over cells of the 5 components (for the average x)
__global__ void __launch_bounds__(RED_TPB) k_sum5(int N, const double* __restrict__ x, double* __restrict__ partial) {
    double a[5] = {0, 0, 0, 0, 0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x)
#pragma unroll
        for (int c = 0; c < 5; ++c) a[c] += x[5 * i + c];
#pragma unroll
    for (int c = 0; c < 5; ++c) {
        double v = block_sum(a[c]);
        if (threadIdx.x == 0) partial[blockIdx.x * 5 + c] = v;
    }
}

__global__ void k_mean5_finalize(const double* __restrict__ partial, int nb, int N, double* __restrict__ xbar) {
    for (int c = 0; c < 5; ++c) {
        double s = 0;
        for (int b = threadIdx.x; b < nb; b += blockDim.x) s += partial[b * 5 + c];
        s = block_sum(s);
        if (threadIdx.x == 0) xbar[c] = s / N;
    }
}

// linear residual per component / normFactor
__global__ void k_linres_finalize(const double* __restrict__ partial, int nb, Scalars* sc) {
    for (int c = 0; c < 5; ++c) {
        double s = 0;
        for (int b = threadIdx.x; b < nb; b += blockDim.x) s += partial[b * 5 + c];
        s = block_sum(s);
        if (threadIdx.x == 0) {
            sc->lin_final[c] = s / sc->nf;
        }
    }
}

// BlockSolverPerformance check: converged if every component below the
// tolerance, or below relTol x initial, or maxIter reached (after minIter).
// A solve that stops on maxIter alone raises bit 3 of the step flags (the
// solver performance's converged() is false); one that stops on the
// tolerances clears it.
struct Criteria { double tol, relTol; int minIter, maxIter; };
__device__ __forceinline__ void solver_check(Scalars* sc, const Criteria& k, int count) {
    const double tol = k.tol, relTol = k.relTol;
    const int minIter = k.minIter, maxIter = k.maxIter;
    if (count) sc->lin_iterations += 1;
    int it = sc->lin_iterations;
    bool t = true, r = relTol > 0;
    for (int c = 0; c < 5; ++c) {
        if (!(sc->lin_final[c] < tol)) t = false;
        if (!(sc->lin_final[c] < relTol * sc->lin_initial[c])) r = false;
    }
    // (or a wait has expired: no iteration will change anything)
    sc->converged = ((it >= minIter) && (t || r || it >= maxIter)) || (sc->flags & 4);
    if (sc->converged) sc->flags = (t || r) ? (sc->flags & ~8) : (sc->flags | 8);
}
__global__ void k_check(Scalars* sc, Criteria k, int count) {
    if (threadIdx.x == 0) solver_check(sc, k, count);
}
// sums of k_solve_init -> normFactor, initial residual, no iterations, check
__global__ void k_solve_start(const double* __restrict__ partial, int nb, Scalars* sc, Criteria k) {
    double t[6];
#pragma unroll
    for (int c = 0; c < 6; ++c) {
        double s = 0;
        for (int b = threadIdx.x; b < nb; b += blockDim.x) s += partial[b * 6 + c];
        t[c] = block_sum(s);
    }
    if (threadIdx.x != 0) return;
    sc->nf = t[0] + 1.0e-20;
    for (int c = 0; c < 5; ++c) sc->lin_initial[c] = sc->lin_final[c] = t[1 + c] / sc->nf;
    sc->lin_iterations = 0;
    solver_check(sc, k, 0);
}

// ---------------------------------------------------------------- GMRES
// One Arnoldi vector's orthogonalisation in one cooperative launch: two
// classical Gram-Schmidt passes, each with dots of its own (the coefficients of
// the second formed from the Gram matrix of the basis instead would save a read
// of it, but leave the basis less orthogonal, by |w| / |w - V h|: 4e-14 where two
// passes leave 5e-16 at a ratio of 86).
//
// A launch per pass and one per sum costs more than the passes themselves up
// to about 1e5 unknowns; the passes are therefore separated by a grid-wide
// barrier (all blocks resident: cooperative launch), each block adding up
// the blocks' partial sums by itself in the same order.
//
// With a basis in FP32 (FP32 and BF16 Jacobians) the Arnoldi vector is rounded
// to FP32 after every direction and in every preconditioner application, so a
// last-bit difference in a coefficient is a difference of 1e-7 in the solve.
// The kernel therefore keeps the sums of the separate launches it replaces to the
// order of every addition, for both storages: red_blocks(n) "blocks" of 256
// threads (a CTA takes two at a time, all of one SM's in turn), four entries a
// thread per piece, the pieces in ascending order, the warps' tree, the eight
// warps one after the other, then the blocks' sums as one block of 256 threads
// adds them up.  Vectors are padded to 64 entries of zeros, so no load needs a
// test for the end.  The loads of eight vectors at a time are issued together,
// whatever their number (FP32, 1.2 M cells, mean of 20 directions: 230 -> 203 us;
// keeping sixteen vectors in registers between the two uses spilled and was
// slower).  It is bound by the three reads of the basis, on small meshes by the
// barriers and the chain of loads between them.  Per direction, mean of 20,
// FP64, against the ten launches of before (dots, update and dots, update and
// norm, each with its own sum, then the rotation and the scaling): 4 k cells
// 45 -> 20 us, 442 k 170 -> 124.
constexpr int ORTH_TPB = 512;
constexpr int ORTH_NV = 16;                     // basis vectors whose dots a thread holds at once
constexpr int ORTH_MAXV = 64;                   // GMRES directions at most

// f(integral_constant<cnt>) for 1 <= cnt <= MAXC: the loads of a round are all
// issued before the first is used only if their number is known
template <int MAXC, typename F>
__device__ __forceinline__ void with_count(int cnt, F&& f) {
    if constexpr (MAXC > 1) {
        if (cnt < MAXC) { with_count<MAXC - 1>(cnt, f); return; }
    }
    f(std::integral_constant<int, MAXC>());
}
// four consecutive entries as they are stored
template <typename VT> struct Raw4;
template <> struct Raw4<float> { using T = float4; };
struct __align__(16) Doubles4 { double2 a, b; };
template <> struct Raw4<double> { using T = Doubles4; };
__device__ __forceinline__ void raw4(const float4& a, double (&o)[4]) { o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w; }
__device__ __forceinline__ void raw4(const Doubles4& v, double (&o)[4]) { o[0] = v.a.x; o[1] = v.a.y; o[2] = v.b.x; o[3] = v.b.y; }

__device__ __forceinline__ void copy4(const double (&a)[4], double (&o)[4]) { o[0] = a[0]; o[1] = a[1]; o[2] = a[2]; o[3] = a[3]; }

// the warp's sums of 16 values: lane l gets that of a[l / 2]
__device__ __forceinline__ double warp_sum16(double (&a)[16]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 16; o > 1; o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < o / 2; ++i) {
            const double send = up ? a[i] : a[i + o / 2], keep = up ? a[i + o / 2] : a[i];
            a[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    return a[0] + __shfl_xor_sync(0xffffffffu, a[0], 1);
}

// All blocks of a cooperative launch, the round-th time in it (from 1); false
// after wait_ms (0: at once).  A launch that gave up leaves the counter as it is,
// so the solver kernels do nothing more (wait_expired) until the host has cleared
// it (k_clear_expired, k_init_scalars).
__device__ __forceinline__ bool grid_barrier(Scalars* sc, unsigned round, unsigned wait_ms) {
    unsigned* bar = &sc->orth_bar;
    const unsigned target = round * gridDim.x;
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
        unsigned v;
        unsigned long long t0 = 0;
        int ok = 0;
        for (unsigned it = 0; wait_ms; ++it) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
            if (v >= target) { ok = 1; break; }
            if ((it & 255u) == 255u) {
                const unsigned long long now = globaltimer_ns();
                if (t0 == 0) t0 = now;
                else if (now - t0 > wait_ms * 1000000ull) break;
            }
        }
        if (!ok) wait_expired(sc);
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// out[c] = sum over the blocks of part[c * nb + block], c < ncol, by all
// threads of the block (a warp per column, eight columns in flight)
template <int TPB_>
__device__ __forceinline__ void sum_columns(const double* part, int ncol, int nb, double* out) {
    constexpr int NW = TPB_ / 32;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int c0 = 0; c0 < ncol; c0 += 8 * NW) {
        double s[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) s[q] = 0.0;
        for (int b = lane; b < nb; b += 32)
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if (c0 + wid + NW * q < ncol) s[q] += __ldcg(part + (size_t)(c0 + wid + NW * q) * nb + b);
#pragma unroll
        for (int q = 0; q < 8; ++q)
            if (c0 + wid + NW * q < ncol) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) s[q] += __shfl_xor_sync(0xffffffffu, s[q], o);
                if (lane == 0) out[c0 + wid + NW * q] = s[q];
            }
    }
    __syncthreads();
}

// two consecutive entries as doubles
__device__ __forceinline__ void load2(const double* p, double (&o)[2]) {
    const double2 a = *reinterpret_cast<const double2*>(p);
    o[0] = a.x; o[1] = a.y;
}
__device__ __forceinline__ void load2(const float* p, double (&o)[2]) {
    const float2 a = *reinterpret_cast<const float2*>(p);
    o[0] = a.x; o[1] = a.y;
}
// two entries stored, the padding past n left as it is
__device__ __forceinline__ void store2(double* p, long i0, long n, const double (&a)[2]) {
    if (i0 + 2 <= n) *reinterpret_cast<double2*>(p + i0) = make_double2(a[0], a[1]);
    else if (i0 < n) p[i0] = a[0];
}
__device__ __forceinline__ void store2(float* p, long i0, long n, const double (&a)[2]) {
    if (i0 + 2 <= n) *reinterpret_cast<float2*>(p + i0) = make_float2((float)a[0], (float)a[1]);
    else if (i0 < n) p[i0] = (float)a[0];
}
// a -= sum_j c_j V_j at entries i0, i0 + 1
template <typename VT>
__device__ __forceinline__ void orth_subtract(const VT* V, long ldv, int nv, const double* c, long i0, double (&a)[2]) {
    int j = 0;
    for (; j + 8 <= nv; j += 8) {
        double v[8][2];
#pragma unroll
        for (int q = 0; q < 8; ++q) load2(V + (j + q) * ldv + i0, v[q]);
#pragma unroll
        for (int q = 0; q < 8; ++q) { a[0] -= c[j + q] * v[q][0]; a[1] -= c[j + q] * v[q][1]; }
    }
    if (j < nv) {
        double v[7][2];
#pragma unroll
        for (int q = 0; q < 7; ++q)
            if (j + q < nv) load2(V + (j + q) * ldv + i0, v[q]);
#pragma unroll
        for (int q = 0; q < 7; ++q)
            if (j + q < nv) { a[0] -= c[j + q] * v[q][0]; a[1] -= c[j + q] * v[q][1]; }
    }
}

// the cycle's start (one block): bh = beta e_0
__device__ __forceinline__ void gm_start(Scalars* sc, double beta) {
    for (int q = threadIdx.x; q < 65; q += blockDim.x) sc->bh[q] = q == 0 ? beta : 0.0;
    if (threadIdx.x == 0) {
        sc->beta = beta;
        sc->gm_active = beta != 0.0;
        sc->gm_used = 0;
    }
}
// H(:, i) = h with the earlier rotations, its own (foam givensRotation) and
// bh (one block; the rotations come through shared memory)
__device__ __forceinline__ void gm_rotate(Scalars* sc, const double* h, double* s_cs, double* s_sn, int i, int m,
                                          double beta) {
    __syncthreads();
    if ((int)threadIdx.x < i) { s_cs[threadIdx.x] = sc->cs[threadIdx.x]; s_sn[threadIdx.x] = sc->sn[threadIdx.x]; }
    __syncthreads();
    if (threadIdx.x != 0) return;
    double hh = h[0];
    for (int j = 0; j < i; ++j) {
        const double Hji = hh, Hn = h[j + 1];
        sc->H[j * m + i] = s_cs[j] * Hji - s_sn[j] * Hn;
        hh = s_sn[j] * Hji + s_cs[j] * Hn;
    }
    double c, s;
    if (beta == 0.0) { c = 1; s = 0; }
    else if (fabs(beta) > fabs(hh)) { double tau = -hh / beta; s = 1.0 / sqrt(1.0 + tau * tau); c = s * tau; }
    else { double tau = -beta / hh; c = 1.0 / sqrt(1.0 + tau * tau); s = c * tau; }
    sc->cs[i] = c;
    sc->sn[i] = s;
    const double bhi = sc->bh[i], bhn = sc->bh[i + 1];
    sc->bh[i] = c * bhi - s * bhn;
    sc->bh[i + 1] = s * bhi + c * bhn;
    sc->H[i * m + i] = c * hh - s * beta;
    sc->beta = beta;
    sc->gm_used = i + 1;
    if (beta == 0.0) sc->gm_active = 0;
}
// the last block out leaves the barrier as the next launch needs it
__device__ __forceinline__ void grid_leave(Scalars* sc) {
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(&sc->orth_out, 1u) == gridDim.x - 1) { sc->orth_bar = 0; sc->orth_out = 0; }
}

// sum of part[0..nb) as one block of RED_TPB threads takes it: thread t the
// entries t, t + RED_TPB, .., a tree over each warp, a tree over the warps;
// by one warp, all lanes the result
__device__ __forceinline__ double sum_as_block(const double* part, int nb) {
    constexpr int NW = RED_TPB / 32;            // 8
    const int lane = threadIdx.x & 31;
    double s[NW];
#pragma unroll
    for (int q = 0; q < NW; ++q) s[q] = 0.0;
    for (int b0 = 0; b0 < nb; b0 += RED_TPB)
#pragma unroll
        for (int q = 0; q < NW; ++q) {
            const int b = b0 + 32 * q + lane;
            if (b < nb) s[q] += __ldcg(part + b);
        }
    // the eight trees at once: after three halvings lane l holds warp l / 4's
    // partial sum over its four lanes' residues, two more steps complete it
#pragma unroll
    for (int o = 16, h = NW / 2; h > 0; o >>= 1, h >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int q = 0; q < h; ++q) {
            const double send = up ? s[q] : s[q + h], keep = up ? s[q + h] : s[q];
            s[q] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    double v = s[0];
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    // tree over the warps (lane 4 w): partners 4, 2, 1 warps apart
    v += __shfl_xor_sync(0xffffffffu, v, 16);
    v += __shfl_xor_sync(0xffffffffu, v, 8);
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    return v;
}

// Orthogonalise w against V_0 .. V_{nv-1}, beta = |w|, and (vout) V_nv =
// w / beta; H(:, nv-1), its Givens rotation and bh by the first block.  nv 0
// starts a cycle: beta = |w|, V_0 = w / beta, bh = beta e_0.  w may be vout
// (FP64 basis).  nbv: red_blocks(n); partial: 2 nv + 1 columns of nbv doubles.
//
// SPLIT, where every "block" can have a CTA of its own (then a thread has at most
// one piece): both halves of the CTA hold the same pieces of w, in registers from
// the first pass to the last, and share the basis vectors of the dots between
// them; w is not written (FP64, 4 k cells: 23.3 -> 20.4 us, 17 k: 29.3 -> 25.5).
template <typename VT, bool SPLIT>
__global__ void __launch_bounds__(ORTH_TPB, 1)
    k_orth_cgs2(long n, int nv, const VT* V, long ldv, double* w, VT* vout, double* partial, Scalars* sc, int m, int nbv,
                unsigned wait_ms) {
    if (nv > 0 ? !sc->gm_active : (sc->flags & 4) != 0) return;
    constexpr int NWB = RED_TPB / 32;               // warps of a virtual block
    __shared__ double s_red[ORTH_TPB / 32][ORTH_NV];
    __shared__ double s_h[2][ORTH_MAXV], s_rot[2][ORTH_MAXV], s_b;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, g = tid / RED_TPB, t = tid % RED_TPB;
    const int i = nv - 1;
    const long nc = (n + 3) / 4, stride = (long)nbv * RED_TPB;
    unsigned round = 0;
    auto barrier = [&] { return grid_barrier(sc, ++round, wait_ms); };
    // every virtual block of this CTA, two at a time (f is called by all
    // threads, with a block past the end for a CTA's odd last one)
    auto blocks = [&](auto f) {
        if (SPLIT) f((int)blockIdx.x);
        else for (int b0 = 2 * blockIdx.x; b0 < nbv; b0 += 2 * gridDim.x) f(b0 + g);
    };
    // the block's sums of cnt values into columns col.. : a tree over each
    // warp, the warps one after the other
    auto block_sums = [&](double (&acc)[ORTH_NV], int cnt, int col, int vb) {
        const double s = warp_sum16(acc);
        if ((lane & 1) == 0) s_red[wid][lane >> 1] = s;
        __syncthreads();
        if (t < cnt && vb < nbv) {
            double v = 0;
            for (int q = 0; q < NWB; ++q) v += s_red[g * NWB + q][t];
            partial[(size_t)(col + t) * nbv + vb] = v;
        }
        __syncthreads();
    };
    auto dot4 = [&](double& acc, const double (&v)[4], const double (&a)[4]) {
        acc += v[0] * a[0] + v[1] * a[1] + v[2] * a[2] + v[3] * a[3];
    };
    auto store4 = [&](long i0, const double (&a)[4]) {
        if (i0 + 4 <= n) {
            reinterpret_cast<double2*>(w + i0)[0] = make_double2(a[0], a[1]);
            reinterpret_cast<double2*>(w + i0)[1] = make_double2(a[2], a[3]);
        } else {
            for (int e = 0; e < 4 && i0 + e < n; ++e) w[i0 + e] = a[e];
        }
    };
    double keep[4] = {0, 0, 0, 0};                  // SPLIT: the thread's piece of w
    if (SPLIT && nv > 0) {
        const long c = (long)blockIdx.x * RED_TPB + t;
        if (c < nc) load4(w + 4 * c, keep);
    }
    // entries k.. of C vectors from V_j on, as they are stored
    auto fetch = [&](int j, long k, auto& x, auto cnt) {
#pragma unroll
        for (int q = 0; q < decltype(cnt)::value; ++q)
            x[q] = *reinterpret_cast<const typename Raw4<VT>::T*>(V + (j + q) * ldv + k);
    };
    // a -= sum_j coef_j V_j at entries k.. (ascending j)
    auto reduce = [&](const double* coef, long k, double (&a)[4]) {
        auto some = [&](int j, auto cnt) {
            constexpr int C = decltype(cnt)::value;
            typename Raw4<VT>::T x[C];
            fetch(j, k, x, cnt);
#pragma unroll
            for (int q = 0; q < C; ++q) {
                double v[4];
                raw4(x[q], v);
#pragma unroll
                for (int e = 0; e < 4; ++e) a[e] -= coef[j + q] * v[e];
            }
        };
        int j = 0;
        for (; j + 8 <= nv; j += 8) some(j, std::integral_constant<int, 8>());
        if (j < nv) with_count<7>(nv - j, [&](auto cnt) { some(j, cnt); });
    };
    // dots with vectors jb.. < nv into columns col + jb..; with `coef` the
    // vector is first reduced by coef_j V_j over all j (once, jb 0)
    auto dots = [&](int col, const double* coef) {
        const int per = SPLIT && nv <= ORTH_NV ? ORTH_NV / 2 : ORTH_NV;      // vectors of a group at once
        for (int j0 = 0; j0 < nv; j0 += SPLIT ? 2 * per : per) {
            const int jb = SPLIT ? j0 + per * g : j0;
            const int cnt = min(per, nv - jb);
            blocks([&](int vb) {
                double acc[ORTH_NV];
#pragma unroll
                for (int q = 0; q < ORTH_NV; ++q) acc[q] = 0.0;
                if (vb < nbv)
                    for (long c = (long)vb * RED_TPB + t; c < nc; c += stride) {
                        double a[4];
                        if (SPLIT) {
                            if (coef && j0 == 0) reduce(coef, 4 * c, keep);
                            copy4(keep, a);
                        } else {
                            load4(w + 4 * c, a);
                            if (coef && j0 == 0) {
                                reduce(coef, 4 * c, a);
                                store4(4 * c, a);
                            }
                        }
                        auto some = [&](auto from, auto tag) {
                            constexpr int F = decltype(from)::value, C = decltype(tag)::value;
                            typename Raw4<VT>::T x[C];
                            fetch(jb + F, 4 * c, x, tag);
#pragma unroll
                            for (int q = 0; q < C; ++q) {
                                double v[4];
                                raw4(x[q], v);
                                dot4(acc[F + q], v, a);
                            }
                        };
                        using Zero = std::integral_constant<int, 0>;
                        using Half = std::integral_constant<int, ORTH_NV / 2>;
                        if (cnt >= ORTH_NV / 2) {
                            some(Zero(), Half());
                            if (cnt > ORTH_NV / 2)
                                with_count<ORTH_NV / 2>(cnt - ORTH_NV / 2, [&](auto tag) { some(Half(), tag); });
                        } else if (cnt > 0) {
                            with_count<ORTH_NV / 2>(cnt, [&](auto tag) { some(Zero(), tag); });
                        }
                    }
                block_sums(acc, cnt, col + jb, vb);
            });
        }
    };
    double beta;
    if (nv == 0) {
        // |w|^2 entry by entry, the warps' sums by a tree
        blocks([&](int block) {
            const int vb = SPLIT && g ? nbv : block;
            double acc = 0.0;
            if (vb < nbv)
                for (long k = (long)vb * RED_TPB + t; k < n; k += stride) {
                    const double a = w[k];
                    acc += a * a;
                }
            acc = warp_sum(acc);
            if (lane == 0) s_red[wid][0] = acc;
            __syncthreads();
            if (t < 32) {
                double v = t < NWB ? s_red[g * NWB + t][0] : 0.0;
                v = warp_sum(v);
                if (t == 0 && vb < nbv) partial[vb] = v;
            }
            __syncthreads();
        });
        if (!barrier()) return;
        if (wid == 0) {
            const double s = sum_as_block(partial, nbv);
            if (lane == 0) s_b = sqrt(s);
        }
    } else {
        double* part1 = partial + (size_t)nv * nbv;
        double* part2 = partial + 2 * (size_t)nv * nbv;
        auto sums = [&](const double* part, double* out) {
            for (int j = wid; j < nv; j += ORTH_TPB / 32) {
                const double s = sum_as_block(part + (size_t)j * nbv, nbv);
                if (lane == 0) out[j] = s;
            }
            __syncthreads();
        };
        dots(0, nullptr);
        if (!barrier()) return;
        sums(partial, s_h[0]);
        dots(nv, s_h[0]);
        if (!barrier()) return;
        sums(part1, s_h[1]);
        blocks([&](int vb) {
            double acc[ORTH_NV];
#pragma unroll
            for (int q = 0; q < ORTH_NV; ++q) acc[q] = 0.0;
            if (vb < nbv)
                for (long c = (long)vb * RED_TPB + t; c < nc; c += stride) {
                    double a[4];
                    if (SPLIT) {
                        reduce(s_h[1], 4 * c, keep);
                        copy4(keep, a);
                    } else {
                        load4(w + 4 * c, a);
                        reduce(s_h[1], 4 * c, a);
                        store4(4 * c, a);
                    }
                    acc[0] += a[0] * a[0] + a[1] * a[1] + a[2] * a[2] + a[3] * a[3];
                }
            block_sums(acc, SPLIT && g ? 0 : 1, 2 * nv, vb);
        });
        if (!barrier()) return;
        if (wid == 0) {
            const double s = sum_as_block(part2, nbv);
            if (lane == 0) s_b = sqrt(s);
        }
    }
    __syncthreads();
    beta = s_b;
    if (vout && beta != 0.0)
        blocks([&](int vb) {
            if (vb < nbv)
                for (long c = (long)vb * RED_TPB + t; c < nc; c += stride)
                    for (int hf = SPLIT ? g : 0; hf < (SPLIT ? g + 1 : 2); ++hf) {
                        const long i0 = 4 * c + 2 * hf;
                        double a[2];
                        if (SPLIT && nv > 0) { a[0] = hf ? keep[2] : keep[0]; a[1] = hf ? keep[3] : keep[1]; }
                        else load2(w + i0, a);
                        a[0] /= beta;
                        a[1] /= beta;
                        store2(vout, i0, n, a);
                    }
        });
    if (blockIdx.x == 0) {
        if (nv == 0) gm_start(sc, beta);
        else {
            __syncthreads();
            if (tid < nv) s_h[0][tid] += s_h[1][tid];
            gm_rotate(sc, s_h[0], s_rot[0], s_rot[1], i, m, beta);
        }
    }
    grid_leave(sc);
}

// dx += V y with H y = bh (each block solves for y itself, H through shared
// memory: 20 rows in ~3 us, where a launch of one thread reading H from
// global memory took 25)
template <typename VT>
__global__ void __launch_bounds__(ORTH_TPB, 2) k_gm_update(long n, int m, const VT* __restrict__ V, long ldv,
                                                           double* __restrict__ dx, const Scalars* __restrict__ sc) {
    __shared__ double s_y[ORTH_MAXV];
    extern __shared__ double s_H[];                 // [used][used]
    const int tid = threadIdx.x, used = sc->gm_used;
    for (int q = tid; q < used * used; q += ORTH_TPB) s_H[q] = sc->H[(q / used) * m + q % used];
    if (tid < used) s_y[tid] = sc->bh[tid];
    __syncthreads();
    if (tid == 0) {
        for (int i = used - 1; i >= 0; --i) {
            double sum = s_y[i];
#pragma unroll 4
            for (int j = i + 1; j < used; ++j) sum -= s_H[i * used + j] * s_y[j];
            s_y[i] = sum / s_H[i * used + i];
        }
    }
    __syncthreads();
    if (tid < used) s_y[tid] = -s_y[tid];
    __syncthreads();
    const long nh = (n + 1) / 2;
    for (long c = (long)blockIdx.x * ORTH_TPB + tid; c < nh; c += (long)gridDim.x * ORTH_TPB) {
        double a[2];
        load2(dx + 2 * c, a);
        orth_subtract(V, ldv, used, s_y, 2 * c, a);
        store2(dx, 2 * c, n, a);
    }
}

// ---------------------------------------------------------------- BiCGStab
// The vector work between the preconditioner and matrix applications of an
// iteration, in cooperative launches (a thread per cell, the sums over a
// bounded grid barrier as in k_orth_cgs2): two launches an iteration where dots,
// their sums, the scalars, the updates, the residual sum and the check took
// seventeen, each a few us on the meshes this solver is used on.  An iteration
// after the converged one (bi_active 0) does nothing, so the host need not
// wait for each check before it launches the next (run_steps).  RAE2822, 23,552
// cells, steps of 7 to 12 iterations, a run of six: 12.2 -> 11.5 ms.  One CTA an
// SM (the count shared with k_orth_cgs2) leaves bandwidth unused on large meshes,
// but is still less than the launches it replaces took: 442 k cells 200 -> 134 us
// an iteration, 1.2 M 436 -> 361.
constexpr int BI_TPB = 256;
constexpr int BI_COLS = 8;          // columns of partial sums

template <int K>
__device__ __forceinline__ void bi_columns(double (&x)[K], double* partial, int col) {
    __shared__ double s_red[BI_TPB / 32][K];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < K; ++q) {
        const double v = warp_sum(x[q]);
        if (lane == 0) s_red[wid][q] = v;
    }
    __syncthreads();
    if (threadIdx.x < K) {
        double v = 0;
        for (int q = 0; q < BI_TPB / 32; ++q) v += s_red[q][threadIdx.x];
        partial[(size_t)(col + threadIdx.x) * gridDim.x + blockIdx.x] = v;
    }
}

// r = rw = p = rhs, v = 0, rho = rw . r
__global__ void __launch_bounds__(BI_TPB) k_bi_start(int N, const double* __restrict__ rhs, double* __restrict__ r,
                                                     double* __restrict__ rw, double* __restrict__ p,
                                                     double* __restrict__ v, double* partial, Scalars* sc,
                                                     unsigned wait_ms) {
    if (sc->flags & 4) return;
    __shared__ double s_sum[1];
    double d[1] = {0.0};
    for (long i = (long)blockIdx.x * BI_TPB + threadIdx.x; i < N; i += (long)gridDim.x * BI_TPB)
#pragma unroll
        for (int c = 0; c < 5; ++c) {
            const double a = rhs[5 * i + c];
            r[5 * i + c] = a;
            rw[5 * i + c] = a;
            p[5 * i + c] = a;
            v[5 * i + c] = 0.0;
            d[0] += a * a;
        }
    bi_columns(d, partial, 0);
    if (!grid_barrier(sc, 1, wait_ms)) return;
    if (blockIdx.x == 0) {
        sum_columns<BI_TPB>(partial, 1, gridDim.x, s_sum);
        if (threadIdx.x == 0) {
            sc->bi_rho = s_sum[0];
            sc->bi_active = 1;
        }
    }
    grid_leave(sc);
}

// alpha = rho / (rw . v); s = r - alpha v
__global__ void __launch_bounds__(BI_TPB) k_bi_alpha(int N, const double* __restrict__ rw, const double* __restrict__ r,
                                                     const double* __restrict__ v, double* __restrict__ s,
                                                     double* partial, Scalars* sc, unsigned wait_ms) {
    if (!sc->bi_active) return;
    __shared__ double s_sum[1];
    const double rho = sc->bi_rho;
    double d[1] = {0.0};
    for (long i = (long)blockIdx.x * BI_TPB + threadIdx.x; i < N; i += (long)gridDim.x * BI_TPB)
#pragma unroll
        for (int c = 0; c < 5; ++c) d[0] += rw[5 * i + c] * v[5 * i + c];
    bi_columns(d, partial, 0);
    if (!grid_barrier(sc, 1, wait_ms)) return;
    sum_columns<BI_TPB>(partial, 1, gridDim.x, s_sum);
    const double alpha = rho / s_sum[0];
    for (long i = (long)blockIdx.x * BI_TPB + threadIdx.x; i < N; i += (long)gridDim.x * BI_TPB)
#pragma unroll
        for (int c = 0; c < 5; ++c) s[5 * i + c] = r[5 * i + c] - alpha * v[5 * i + c];
    if (blockIdx.x == 0 && threadIdx.x == 0) sc->bi_alpha = alpha;
    grid_leave(sc);
}

// omega = (t . s) / (t . t); x += alpha ph + omega sh; r = s - omega t; the
// residual sums and the check; rho, beta and the next p = r + beta (p - omega v)
__global__ void __launch_bounds__(BI_TPB) k_bi_omega(int N, double* __restrict__ x, double* __restrict__ r,
                                                     const double* __restrict__ ph, const double* __restrict__ sh,
                                                     const double* __restrict__ s, const double* __restrict__ t,
                                                     const double* __restrict__ rw, const double* __restrict__ v,
                                                     double* __restrict__ p, double* partial, Scalars* sc, Criteria k,
                                                     unsigned wait_ms) {
    if (!sc->bi_active) return;
    __shared__ double s_sum[6];
    const double alpha = sc->bi_alpha, rho0 = sc->bi_rho;
    const long i0 = (long)blockIdx.x * BI_TPB + threadIdx.x, stride = (long)gridDim.x * BI_TPB;
    double d[2] = {0.0, 0.0};
    for (long i = i0; i < N; i += stride)
#pragma unroll
        for (int c = 0; c < 5; ++c) {
            const double tc = t[5 * i + c];
            d[0] += tc * tc;
            d[1] += tc * s[5 * i + c];
        }
    bi_columns(d, partial, 0);
    if (!grid_barrier(sc, 1, wait_ms)) return;
    sum_columns<BI_TPB>(partial, 2, gridDim.x, s_sum);
    const double omega = s_sum[0] > 0 ? s_sum[1] / s_sum[0] : 0.0;
    double a[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    for (long i = i0; i < N; i += stride)
#pragma unroll
        for (int c = 0; c < 5; ++c) {
            const long e = 5 * i + c;
            x[e] += alpha * ph[e] + omega * sh[e];
            const double rn = s[e] - omega * t[e];
            r[e] = rn;
            a[c] += fabs(rn);
            a[5] += rw[e] * rn;
        }
    double* part2 = partial + 2 * (size_t)gridDim.x;
    bi_columns(a, part2, 0);
    if (!grid_barrier(sc, 2, wait_ms)) return;
    sum_columns<BI_TPB>(part2, 6, gridDim.x, s_sum);
    const double rho = s_sum[5], beta = rho / rho0 * (alpha / omega);
    for (long i = i0; i < N; i += stride)
#pragma unroll
        for (int c = 0; c < 5; ++c) {
            const long e = 5 * i + c;
            p[e] = r[e] + beta * (p[e] - omega * v[e]);
        }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        for (int c = 0; c < 5; ++c) sc->lin_final[c] = s_sum[c] / sc->nf;
        sc->bi_rho = rho;
        solver_check(sc, k, 1);
        if (sc->converged) sc->bi_active = 0;
    }
    grid_leave(sc);
}

}  // namespace rdst
