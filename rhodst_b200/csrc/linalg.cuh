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

// y = A x  (or y = b - A x when b != nullptr); one row per thread; x in
// FP64 or (a Krylov basis vector) FP32, products and y in FP64
template <typename MT, typename XT = double>
__global__ void __launch_bounds__(256) k_spmv(SellMat<MT> A, const XT* __restrict__ x, double* __restrict__ y,
                                              const double* __restrict__ b, const int* __restrict__ active) {
    if (active && !*active) return;
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= A.N) return;
    const int s = r >> 5, lane = r & 31;
    const int base = A.slice_off[s], width = A.slice_w[s];
    double acc[5] = {0, 0, 0, 0, 0};
    for (int k = 0; k < width; ++k) {
        size_t slot = (size_t)(base + k);
        int c = A.col[slot * 32 + lane];
        if (c < 0) continue;
        const XT* xc = x + 5 * c;
        double xv[5] = {tod(xc[0]), tod(xc[1]), tod(xc[2]), tod(xc[3]), tod(xc[4])};
        const MT* v = A.val + slot * (32 * 25) + lane;
#pragma unroll
        for (int i = 0; i < 5; ++i)
#pragma unroll
            for (int j = 0; j < 5; ++j) acc[i] += ld(v + (5 * i + j) * 32) * xv[j];
    }
    double* yr = y + 5 * r;
    if (b) {
#pragma unroll
        for (int i = 0; i < 5; ++i) yr[i] = b[5 * r + i] - acc[i];
    } else {
#pragma unroll
        for (int i = 0; i < 5; ++i) yr[i] = acc[i];
    }
}

// y = A xbar for a constant 5-vector xbar (normFactor reference field)
template <typename MT>
__global__ void k_spmv_const(SellMat<MT> A, const double* __restrict__ xbar, double* __restrict__ y) {
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= A.N) return;
    const int s = r >> 5, lane = r & 31;
    const int base = A.slice_off[s], width = A.slice_w[s];
    double acc[5] = {0, 0, 0, 0, 0};
    double xv[5] = {xbar[0], xbar[1], xbar[2], xbar[3], xbar[4]};
    for (int k = 0; k < width; ++k) {
        size_t slot = (size_t)(base + k);
        if (A.col[slot * 32 + lane] < 0) continue;
        const MT* v = A.val + slot * (32 * 25) + lane;
        for (int i = 0; i < 5; ++i)
            for (int j = 0; j < 5; ++j) acc[i] += ld(v + (5 * i + j) * 32) * xv[j];
    }
    for (int i = 0; i < 5; ++i) y[5 * r + i] = acc[i];
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
// SM.  Every
// mbarrier wait is bounded (2 s of globaltimer): on expiry the warp raises
// bit 2 of *flags (reported as a timeout by the host), takes part in the
// sweep's remaining level barriers, so that no other warp stays in one, and
// ends; they find their own waits expired in turn, and the producer waits,
// again bounded, for its copies in flight.
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
// true once the phase of parity `parity` has completed; false after 2 s
__device__ __noinline__ bool mbar_wait_slow(unsigned bar, unsigned parity) {
    const unsigned long long t0 = globaltimer_ns();
    for (;;) {
        for (int it = 0; it < 64; ++it)
            if (mbar_try(bar, parity)) return true;
        if (globaltimer_ns() - t0 > 2000000000ull) return false;
    }
}
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity) {
    return mbar_try(bar, parity) || mbar_wait_slow(bar, parity);
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

// factor blocks -> records (after each factorisation): a warp per task, lane
// (position, component) as the apply reads it, so that every store of a slot
// fills whole sectors of the record; the reads of the sliced stores are 6-row
// pieces of lines that the neighbouring warps share.  L comes from the factor
// store, U from A (from the factor store for rows whose own blocks take
// updates, zero for a fill), backward first the pivot inverse.
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
        const int nk = k < 4 ? (int)((g.x >> (8 * k)) & 255u) : (int)v[k - 16];
        if (pos < nk) {
            const int f = lu_fid(r, back ? P.ml + k : k, ms);
            const MT* src = lu + flat_e(f, 0);
            if (back && !own_u) {
                const int a = P.lu_src[f];
                src = a >= 0 ? A.val + flat_e(a, 0) : nullptr;
            }
            copy(src, blk);
        }
        blk += nk;
    }
}

template <typename MT, int NB, bool EXT, bool TIGHT>
__global__ void __launch_bounds__(TIGHT ? (sizeof(MT) == 8 ? 96 : 128) : 288, TIGHT ? 6 : 2)
    k_ilu_apply_rec(IluDev P, const double* __restrict__ b, double* x, const int* __restrict__ active,
                    int stage_bytes, int y0_rows, int lb_rows, int* flags) {
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
        bool ok = true;
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
            atomicOr(flags, 4);
            for (int d = 0; d < REC_STAGES; ++d)
                if ((used >> d) & 1u) mbar_wait(full0 + 8 * d, (lastp >> d) & 1u);
        }
        return;
    }

    // ---------------- compute warps
    constexpr unsigned LRB = lb_row_bytes<CT>();
    // ids of the level barriers: more than the W levels a warp can be ahead of
    // the slowest.  An SM has 64 barriers and a kernel that names one in a
    // register reserves all 16, which would leave four CTAs an SM.
    constexpr int NBAR = TIGHT ? 4 : 15;
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
    auto sweep = [&](auto back_tag) -> bool {
        constexpr bool BACK = decltype(back_tag)::value;
        const int ngrp = BACK ? ngb : ngf;
        int grp = 0, arrived = 0, bid = 1;      // group in the sweep; level barriers arrived on, the next one's id
        unsigned gn = 0;                        // the group's address
        bool held = false;                      // the group is not returned yet
        auto arrive = [&] {                     // end of a level on which nobody here waits
            if (TIGHT) {
                if (bid == 1) asm volatile("bar.arrive 1, %0;" ::"r"(W * 32) : "memory");
                else if (bid == 2) asm volatile("bar.arrive 2, %0;" ::"r"(W * 32) : "memory");
                else if (bid == 3) asm volatile("bar.arrive 3, %0;" ::"r"(W * 32) : "memory");
                else asm volatile("bar.arrive 4, %0;" ::"r"(W * 32) : "memory");
            } else {
                asm volatile("bar.arrive %0, %1;" ::"r"(bid), "r"(W * 32) : "memory");
            }
            bid = bid == NBAR ? 1 : bid + 1;
            ++arrived;
        };
        auto await = [&] {                      // end of the level before the next task's
            if (TIGHT) {
                if (bid == 1) asm volatile("bar.sync 1, %0;" ::"r"(W * 32) : "memory");
                else if (bid == 2) asm volatile("bar.sync 2, %0;" ::"r"(W * 32) : "memory");
                else if (bid == 3) asm volatile("bar.sync 3, %0;" ::"r"(W * 32) : "memory");
                else asm volatile("bar.sync 4, %0;" ::"r"(W * 32) : "memory");
            } else {
                asm volatile("bar.sync %0, %1;" ::"r"(bid), "r"(W * 32) : "memory");
            }
            bid = bid == NBAR ? 1 : bid + 1;
            ++arrived;
        };
        auto enter = [&] {                      // the group in stage s has landed
            gn = dyn + (unsigned)(s * stage_bytes);
            held = true;
            if (__all_sync(0xffffffffu, mbar_wait(full0 + 8 * s, ph))) return true;
            if (lane == 0) atomicOr(flags, 4);
            while (arrived < nlev - 1) await();      // in step with the others, who may still run
            return false;
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
            while (arrived < level - 1) arrive();
            if (arrived < level) await();
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
                        const int nk = k < 4 ? (int)((nk4 >> (8 * k)) & 255u) : (int)lds_byte(cv - 16 + k);
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
        while (arrived < nlev - 1) arrive();
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
    if (!sweep(std::false_type{})) return;
    sweep(std::true_type{});
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

// partial[blk * nv + j] = sum_i V_j[i] * w[i], j < nv (nv <= 8 per launch)
__global__ void __launch_bounds__(RED_TPB) k_multidot(long n, int nv, const double* __restrict__ V, long ldv,
                                                      const double* __restrict__ w, double* __restrict__ partial,
                                                      int pstride, const int* __restrict__ active) {
    if (active && !*active) return;
    double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        double wi = w[i];
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (j < nv) acc[j] += V[j * ldv + i] * wi;
    }
    for (int j = 0; j < nv; ++j) {
        double v = block_sum(acc[j]);
        if (threadIdx.x == 0) partial[(long)blockIdx.x * pstride + j] = v;
    }
}

// Deterministic block reduction of NV per-thread values: warp shuffles,
// then one fixed-order sum over the warps; result -> partial[blk*pstride+j].
template <int NV>
__device__ __forceinline__ void block_multi_sum(double (&acc)[NV], int nv, double* __restrict__ partial, int pstride) {
    __shared__ double sh[RED_TPB / 32][NV];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        if (j < nv) {
            double v = warp_sum(acc[j]);
            if (lane == 0) sh[wid][j] = v;
        }
    }
    __syncthreads();
    if (threadIdx.x < nv) {
        double v = 0;
        for (int w2 = 0; w2 < (int)(blockDim.x >> 5); ++w2) v += sh[w2][threadIdx.x];
        partial[(long)blockIdx.x * pstride + threadIdx.x] = v;
    }
}

// partial[blk][j] = sum_i V_j[i] w[i] for j < nv <= NV (one pass over w)
// Four consecutive entries of a vector as doubles (16-byte loads; the
// caller guarantees 4-entry alignment of p), or fewer at the vector's end.
__device__ __forceinline__ void load4(const double* __restrict__ p, double (&o)[4]) {
    const double2 a = reinterpret_cast<const double2*>(p)[0], b = reinterpret_cast<const double2*>(p)[1];
    o[0] = a.x; o[1] = a.y; o[2] = b.x; o[3] = b.y;
}
__device__ __forceinline__ void load4(const float* __restrict__ p, double (&o)[4]) {
    const float4 a = *reinterpret_cast<const float4*>(p);
    o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w;
}
template <typename T>
__device__ __forceinline__ void load4_tail(const T* __restrict__ p, long rem, double (&o)[4]) {
#pragma unroll
    for (int e = 0; e < 4; ++e) o[e] = e < rem ? tod(p[e]) : 0.0;
}
template <typename T>
__device__ __forceinline__ void load4_any(const T* __restrict__ p, long i0, long n, double (&o)[4]) {
    if (i0 + 4 <= n) load4(p + i0, o);
    else load4_tail(p + i0, n - i0, o);
}

// partial[blk * pstride + j] = sum_i V_j[i] w[i], j < nv: four entries per
// thread and 16-byte loads; V (fp64 or fp32) has a row stride ldv that is
// a multiple of 4 entries.  Full chunks take a branch-free path so that
// the loads of all nv vectors are in flight together.
template <int NV, typename VT = double>
__global__ void __launch_bounds__(RED_TPB, 2) k_vmultidot(long n, int nv, const VT* __restrict__ V, long ldv,
                                                       const double* __restrict__ w, double* __restrict__ partial,
                                                       int pstride, const int* __restrict__ active) {
    if (active && !*active) return;
    double acc[NV];
#pragma unroll
    for (int j = 0; j < NV; ++j) acc[j] = 0.0;
    const long nc = (n + 3) / 4, nfull = n / 4;
    for (long c = (long)blockIdx.x * blockDim.x + threadIdx.x; c < nc; c += (long)gridDim.x * blockDim.x) {
        const long i0 = 4 * c;
        double wv[4];
        if (c < nfull) {
            load4(w + i0, wv);
#pragma unroll
            for (int j = 0; j < NV; ++j)
                if (j < nv) {
                    double v[4];
                    load4(V + j * ldv + i0, v);
                    acc[j] += v[0] * wv[0] + v[1] * wv[1] + v[2] * wv[2] + v[3] * wv[3];
                }
        } else {
            load4_tail(w + i0, n - i0, wv);
            for (int j = 0; j < nv && j < NV; ++j) {
                double v[4];
                load4_tail(V + j * ldv + i0, n - i0, v);
                acc[j] += v[0] * wv[0] + v[1] * wv[1] + v[2] * wv[2] + v[3] * wv[3];
            }
        }
    }
    block_multi_sum<NV>(acc, nv, partial, pstride);
}

// w -= sum_j coef[j] V_j (j < nv), then in the same pass either the dots
// V_j . w_new (mode 0: the second CGS2 pass) or w_new . w_new (mode 1);
// four entries per thread as in k_vmultidot
template <int NV, typename VT = double>
__global__ void __launch_bounds__(RED_TPB, 2) k_maxpy_dot(long n, int nv, const VT* __restrict__ V, long ldv,
                                                       const double* __restrict__ coef, double* __restrict__ w,
                                                       double* __restrict__ partial, int pstride, int mode,
                                                       const int* __restrict__ active) {
    if (active && !*active) return;
    __shared__ double cs[NV];
    if (threadIdx.x < NV) cs[threadIdx.x] = threadIdx.x < nv ? coef[threadIdx.x] : 0.0;
    __syncthreads();
    double acc[NV];
#pragma unroll
    for (int j = 0; j < NV; ++j) acc[j] = 0.0;
    const long nc = (n + 3) / 4, nfull = n / 4;
    for (long c = (long)blockIdx.x * blockDim.x + threadIdx.x; c < nc; c += (long)gridDim.x * blockDim.x) {
        const long i0 = 4 * c;
        double a[4];
        if (c < nfull) {
            load4(w + i0, a);
#pragma unroll
            for (int j = 0; j < NV; ++j)
                if (j < nv) {
                    double v[4];
                    load4(V + j * ldv + i0, v);
#pragma unroll
                    for (int e = 0; e < 4; ++e) a[e] -= cs[j] * v[e];
                }
            reinterpret_cast<double2*>(w + i0)[0] = make_double2(a[0], a[1]);
            reinterpret_cast<double2*>(w + i0)[1] = make_double2(a[2], a[3]);
            if (mode == 0) {
                // second read of V_j: the lines were just fetched (L1 hit)
#pragma unroll
                for (int j = 0; j < NV; ++j)
                    if (j < nv) {
                        double v[4];
                        load4(V + j * ldv + i0, v);
                        acc[j] += v[0] * a[0] + v[1] * a[1] + v[2] * a[2] + v[3] * a[3];
                    }
            }
        } else {
            load4_tail(w + i0, n - i0, a);
            for (int j = 0; j < nv && j < NV; ++j) {
                double v[4];
                load4_tail(V + j * ldv + i0, n - i0, v);
                for (int e = 0; e < 4; ++e) a[e] -= cs[j] * v[e];
            }
            for (int e = 0; e < 4; ++e)
                if (i0 + e < n) w[i0 + e] = a[e];
            if (mode == 0) {
                for (int j = 0; j < nv && j < NV; ++j) {
                    double v[4];
                    load4_tail(V + j * ldv + i0, n - i0, v);
                    acc[j] += v[0] * a[0] + v[1] * a[1] + v[2] * a[2] + v[3] * a[3];
                }
            }
        }
        if (mode != 0) acc[0] += a[0] * a[0] + a[1] * a[1] + a[2] * a[2] + a[3] * a[3];
    }
    block_multi_sum<NV>(acc, mode == 0 ? nv : 1, partial, pstride);
}

// out[j] = sum_b partial[b * pstride + j] (fixed order); optional sqrt
__global__ void k_finalize(const double* __restrict__ partial, int nb, int nv, int pstride, double* __restrict__ out,
                           int take_sqrt, const int* __restrict__ active) {
    if (active && !*active) return;
    int j = blockIdx.x;
    if (j >= nv) return;
    double s = 0;
    for (int b = threadIdx.x; b < nb; b += blockDim.x) s += partial[(long)b * pstride + j];
    s = block_sum(s);
    if (threadIdx.x == 0) out[j] = take_sqrt ? sqrt(s) : s;
}

// w -= sum_j coef[j] V_j (j < nv); coef on the device
template <typename VT = double>
__global__ void k_maxpy(long n, int nv, const VT* __restrict__ V, long ldv, const double* __restrict__ coef,
                        double* __restrict__ w, double sign, const int* __restrict__ active) {
    if (active && !*active) return;
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double a = w[i];
    for (int j = 0; j < nv; ++j) a -= sign * coef[j] * tod(V[j * ldv + i]);
    w[i] = a;
}

// x /= *s
__global__ void k_scale_inv(long n, double* __restrict__ x, const double* __restrict__ s, const int* __restrict__ active) {
    if (active && !*active) return;
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] = x[i] / *s;
}

// v = w / *s stored as a (FP32) basis vector
template <typename VT>
__global__ void k_scale_store(long n, const double* __restrict__ w, VT* __restrict__ v, const double* __restrict__ s,
                              const int* __restrict__ active) {
    if (active && !*active) return;
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) v[i] = (VT)(w[i] / *s);
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

// sum_i |Ax_i - pA_i| + |Ax_i + s_i - pA_i| (normFactor, x = W, b = A W + s)
__global__ void __launch_bounds__(RED_TPB) k_normfactor(int N, const double* __restrict__ Ax, const double* __restrict__ s,
                                                        const double* __restrict__ pA, int dependentW,
                                                        double* __restrict__ partial) {
    double a = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
        double s1 = 0, s2 = 0;
#pragma unroll
        for (int c = 0; c < 5; ++c) {
            double ax = dependentW ? Ax[5 * i + c] : 0.0;
            double pa = dependentW ? pA[5 * i + c] : 0.0;
            double b = ax + s[5 * i + c];
            s1 += (ax - pa) * (ax - pa);
            s2 += (b - pa) * (b - pa);
        }
        a += sqrt(s1) + sqrt(s2);
    }
    a = block_sum(a);
    if (threadIdx.x == 0) partial[blockIdx.x] = a;
}

__global__ void k_nf_finalize(const double* __restrict__ partial, int nb, Scalars* sc) {
    double s = 0;
    for (int b = threadIdx.x; b < nb; b += blockDim.x) s += partial[b];
    s = block_sum(s);
    if (threadIdx.x == 0) sc->nf = s + 1.0e-20;
}

__global__ void k_mean5_finalize(const double* __restrict__ partial, int nb, int N, double* __restrict__ xbar) {
    for (int c = 0; c < 5; ++c) {
        double s = 0;
        for (int b = threadIdx.x; b < nb; b += blockDim.x) s += partial[b * 5 + c];
        s = block_sum(s);
        if (threadIdx.x == 0) xbar[c] = s / N;
    }
}

// linear residual per component / normFactor -> initial or final
__global__ void k_linres_finalize(const double* __restrict__ partial, int nb, Scalars* sc, int initial) {
    for (int c = 0; c < 5; ++c) {
        double s = 0;
        for (int b = threadIdx.x; b < nb; b += blockDim.x) s += partial[b * 5 + c];
        s = block_sum(s);
        if (threadIdx.x == 0) {
            const double v = s / sc->nf;
            if (initial) { sc->lin_initial[c] = v; sc->lin_final[c] = v; }
            else sc->lin_final[c] = v;
        }
    }
}

// BlockSolverPerformance check: converged if every component below the
// tolerance, or below relTol x initial, or maxIter reached (after minIter).
// A solve that stops on maxIter alone raises bit 3 of the step flags (the
// solver performance's converged() is false); one that stops on the
// tolerances clears it.
__global__ void k_check(Scalars* sc, double tol, double relTol, int minIter, int maxIter, int count) {
    if (threadIdx.x != 0) return;
    if (count) sc->lin_iterations += 1;
    int it = sc->lin_iterations;
    bool t = true, r = relTol > 0;
    for (int c = 0; c < 5; ++c) {
        if (!(sc->lin_final[c] < tol)) t = false;
        if (!(sc->lin_final[c] < relTol * sc->lin_initial[c])) r = false;
    }
    sc->converged = (it >= minIter) && (t || r || it >= maxIter);
    if (sc->converged) sc->flags = (t || r) ? (sc->flags & ~8) : (sc->flags | 8);
}

// ---------------------------------------------------------------- GMRES
__global__ void k_gm_start(Scalars* sc) {
    if (threadIdx.x != 0) return;
    for (int i = 0; i < 65; ++i) sc->bh[i] = 0.0;
    for (int i = 0; i < 64 * 65; ++i) sc->H[i] = 0.0;
    sc->bh[0] = sc->beta;
    sc->gm_active = (sc->beta != 0.0);
    sc->gm_used = 0;
}

// H[:,i] = h1 + h2 (CGS2), Givens rotations (foam givensRotation), bh
__global__ void k_gm_givens(Scalars* sc, int i, int m) {
    if (threadIdx.x != 0 || !sc->gm_active) return;
    double* H = sc->H;
    for (int j = 0; j <= i; ++j) H[j * m + i] = sc->hcol[0][j] + sc->hcol[1][j];
    double beta = sc->beta;
    for (int j = 0; j < i; ++j) {
        double Hji = H[j * m + i];
        H[j * m + i] = sc->cs[j] * Hji - sc->sn[j] * H[(j + 1) * m + i];
        H[(j + 1) * m + i] = sc->sn[j] * Hji + sc->cs[j] * H[(j + 1) * m + i];
    }
    double hh = H[i * m + i], c, s;
    if (beta == 0.0) { c = 1; s = 0; }
    else if (fabs(beta) > fabs(hh)) { double tau = -hh / beta; s = 1.0 / sqrt(1.0 + tau * tau); c = s * tau; }
    else { double tau = -beta / hh; c = 1.0 / sqrt(1.0 + tau * tau); s = c * tau; }
    sc->cs[i] = c;
    sc->sn[i] = s;
    double bhi = sc->bh[i];
    sc->bh[i] = c * bhi - s * sc->bh[i + 1];
    sc->bh[i + 1] = s * bhi + c * sc->bh[i + 1];
    H[i * m + i] = c * H[i * m + i] - s * beta;
    sc->gm_used = i + 1;
    if (beta == 0.0) sc->gm_active = 0;
}

__global__ void k_gm_backsub(Scalars* sc, int m) {
    if (threadIdx.x != 0) return;
    int used = sc->gm_used;
    for (int i = used - 1; i >= 0; --i) {
        double sum = sc->bh[i];
        for (int j = i + 1; j < used; ++j) sum -= sc->H[i * m + j] * sc->yh[j];
        sc->yh[i] = sum / sc->H[i * m + i];
    }
    for (int i = used; i < m; ++i) sc->yh[i] = 0.0;
}

// ---------------------------------------------------------------- BiCGStab
// p = r + beta (p - omega v)
__global__ void k_bi_p(long n, const double* __restrict__ r, const double* __restrict__ v, double* __restrict__ p,
                       const Scalars* sc) {
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = r[i] + sc->bi_beta * (p[i] - sc->bi_omega * v[i]);
}
__global__ void k_bi_scal_rho(Scalars* sc) {       // rho, beta from rw.r
    if (threadIdx.x != 0) return;
    sc->bi_rhoOld = sc->bi_rho;
    sc->bi_rho = sc->hcol[0][0];
    sc->bi_beta = sc->bi_rho / sc->bi_rhoOld * (sc->bi_alpha / sc->bi_omega);
}
__global__ void k_bi_scal_alpha(Scalars* sc) {
    if (threadIdx.x != 0) return;
    sc->bi_alpha = sc->bi_rho / sc->hcol[0][0];
}
__global__ void k_bi_s(long n, const double* __restrict__ r, const double* __restrict__ v, double* __restrict__ s,
                       const Scalars* sc) {
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) s[i] = r[i] - sc->bi_alpha * v[i];
}
__global__ void k_bi_scal_omega(Scalars* sc) {     // omega = (t.s)/(t.t)
    if (threadIdx.x != 0) return;
    double tt = sc->hcol[0][0], ts = sc->hcol[0][1];
    sc->bi_omega = tt > 0 ? ts / tt : 0.0;
}
__global__ void k_bi_update(long n, double* __restrict__ x, double* __restrict__ r, const double* __restrict__ ph,
                            const double* __restrict__ sh, const double* __restrict__ s, const double* __restrict__ t,
                            const Scalars* sc) {
    long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    x[i] += sc->bi_alpha * ph[i] + sc->bi_omega * sh[i];
    r[i] = s[i] - sc->bi_omega * t[i];
}
__global__ void k_bi_init(Scalars* sc) {
    if (threadIdx.x != 0) return;
    sc->bi_rho = 1e300;
    sc->bi_alpha = 0.0;
    sc->bi_omega = 1e300;
}

}  // namespace rdst
