// Batched ACA+ compression of admissible H-matrix blocks, FP64.
//
// One CTA (a cluster of them for large blocks) runs the whole ACA+ loop of one (block, slip pass) task, following
// BlockTree.ACA_plus_full_traceS/D (src/Hmatrix.py:581-1011):
//  * reference row set / column set of 3 consecutive rows (cols), restarted by
//    reset_reference_row/col (:620-648) when a pivot falls inside them;
//  * pivots are chosen on the A1 operator only and reused for A2 and B, each
//    with its own pivot value alpha (:718-726);
//  * stops on |alpha| < 1e-4 (:697), on the step-size test (:727-736: absolute
//    ||u_k|| ||v_k/alpha|| < eps, or a relative test against a running
//    Frobenius-norm estimate), when max_iter = min(m, n) is reached, or when a
//    reference set cannot be placed (scan_all).
// Rows/columns are indexed in the block's local order (element ids ascending,
// the order of the reference's row_cluster/col_cluster), so the same starting
// indices give the same pivot sequence.  argmax ties resolve to the highest
// index and NaN ranks above every number, as a stable ascending argsort does.
// The GF entries come from the full-space TD kernel (td_gf.cuh).  Residual
// updates use explicitly rounded products (no FMA contraction) in the order
// of the reference's numpy expressions.
#include <stdio.h>
#include "pq3d_common.cuh"
#include "td_gf.cuh"
#include "td_hs.cuh"
#include "hm_layout.cuh"
#include <cuda_bf16.h>
#include <cooperative_groups.h>

using namespace pq3d;

struct AcaTask {
    int64_t rows_off, cols_off;  // offsets into the element-id lists
    int64_t ws_off;              // offset (doubles) of this task's workspace
    int32_t m, n, kmax, pass;    // pass 0 = strike slip (Ss=1), 1 = dip slip (Ds=1)
    int32_t iref0, jref0;        // randint(m) - 3 and randint(n) - 3
};

// Workspace of a task (doubles): U[kmax][3][m], V[kmax][3][n], RIref[3][n] (A1),
// RJref[3][m] (A1), RIstar[3][n], RJstar[3][m].
__host__ __device__ inline int64_t aca_ws_doubles(int m, int n, int kmax)
{
    return (int64_t)kmax * 3 * (m + n) + 6 * (int64_t)(m + n);
}

PQ3D_EXPORT int64_t pq3d_aca_ws_doubles(int m, int n, int kmax) { return aca_ws_doubles(m, n, kmax); }
PQ3D_EXPORT size_t pq3d_aca_task_bytes(void) { return sizeof(AcaTask); }

// Where the time goes: a task is a chain of max rank iterations, each with a residual row and
// a residual column (n + m GF evaluations of some 700 FP64 instructions and a k-term update),
// two pivot searches and the stopping test.  Blocks run from 33 to 20,000 rows, half the work in
// those of at most 256, so what counts is how many tasks an SM has in flight, how short the
// chain between evaluations is, and that the few large ones do not end last:
//  * three kernels by size: tasks of at most 256 rows and columns on 128 threads, several per
//    SM; up to 1,024 on a cluster of two CTAs of 256; larger ones on a cluster of eight, with
//    reductions over distributed shared memory.  Largest first, each kernel's CTAs filling up
//    behind the one before (programmatic launch) and returning at once for tasks of another
//    size;
//  * one residual routine for rows, columns and reference sets, its GF code once: inlined per
//    use the kernel was 225 KB, more than the instruction cache holds;
//  * the candidate searches of row and column in one reduction of ordered bits (redux.sync),
//    the cross terms of the relative test one term per warp, the new row and column written
//    straight to V and U: seven barriers an iteration instead of 50 + 10 per term;
//  * a small task's reference sets in shared memory.
// B200, the kernels of one batch, against one 256-thread CTA a task and one per SM (236
// registers): 2,500 elements at the absolute stop 4.2 -> 1.55 ms, 20,480 at 1e-4 17.9 -> about
// 5 ms, half space 4,000 12.5 -> 8.9 ms; factors bitwise unchanged.  With one CTA of 512 a large
// task the 20k batch ended with its 5,120-row blocks alone (7.6 ms).
constexpr int ACA_SMALL = 256, ACA_MEDIUM = 1024;
constexpr int ACA_TERMS = 128;        // cross terms reduced at a time

// Barrier of a task's CTAs.
template <int CL>
__device__ __forceinline__ void task_sync()
{
    if (CL == 1) {
        __syncthreads();
    } else {
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
}

// p of the task's CTA `rank`.
template <int CL, typename T>
__device__ __forceinline__ const T *task_peer(const T *p, int rank)
{
    if (CL == 1) return p;
    return cooperative_groups::this_cluster().map_shared_rank(const_cast<T *>(p), rank);
}

// A pivot candidate: |value| as ordered bits (NaN, canonical, above every number) and index + 1
// (0: none).  Larger value first, then larger index.
struct Best {
    unsigned long long k;
    unsigned i;
};

__device__ inline unsigned long long magnitude(double v)
{
    return v != v ? 0x7ff8000000000000ull : (unsigned long long)__double_as_longlong(fabs(v));
}

__device__ inline void take(Best &a, unsigned long long k, unsigned i)
{
    if (k > a.k || (k == a.k && i > a.i)) { a.k = k; a.i = i; }
}

__device__ inline Best warp_best(Best a)
{
    const unsigned hi = (unsigned)(a.k >> 32), mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned lo = hi == mh ? (unsigned)a.k : 0u, ml = __reduce_max_sync(0xffffffffu, lo);
    const unsigned i = hi == mh && (unsigned)a.k == ml ? a.i : 0u;
    return Best{((unsigned long long)mh << 32) | ml, __reduce_max_sync(0xffffffffu, i)};
}

__device__ inline bool bit_get(const uint32_t *bm, int i) { return (bm[i >> 5] >> (i & 31)) & 1u; }

struct AcaCtx {
    const double *xg, *ev;
    const SrcRec *rec;
    const HsRec *hs;      // half-space records (HS instantiation only)
    int hs_mode;
    const int32_t *rows, *cols;
    double mu, lam, nu;
    int m, n, pass, k;
    int t;                // thread of the task: its CTA in the cluster * NT + threadIdx.x
    double *U, *V;  // U[q][c][m], V[q][c][n]
};

// Best of NB candidates over the task's CTAs, known to every thread.  The buffer of the call's
// parity, so the next call needs no barrier before it writes.
template <int NT, int CL, int NB>
__device__ __forceinline__ void task_best(Best (&b)[NB], Best (*red)[2][NT / 32], int &parity)
{
    static_assert(NT / 32 * CL <= 64, "two entries per lane");
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    Best (*r)[NT / 32] = red[parity];
    parity ^= 1;
#pragma unroll
    for (int q = 0; q < NB; ++q) {
        b[q] = warp_best(b[q]);
        if (lane == 0) r[q][wid] = b[q];
    }
    task_sync<CL>();
#pragma unroll
    for (int q = 0; q < NB; ++q) {
        b[q] = Best{0ull, 0u};
#pragma unroll
        for (int e = lane; e < NT / 32 * CL; e += 32) {
            const Best o = task_peer<CL>(r[q], e / (NT / 32))[e % (NT / 32)];
            take(b[q], o.k, o.i);
        }
        b[q] = warp_best(b[q]);
    }
}

// Residual entries of `cnt` rows (row: I = F0 + r, all columns) or columns (J = F0 + r, all
// rows): out[c][r][e] for components c < ncomp (1 or 3).  Returns the thread's best A1 entry
// among those not in bm (the last row or column's, when bm is given).
template <bool HS, int NT, int CL>
__device__ __noinline__ Best residual(const AcaCtx &C, bool row, int F0, int cnt, int ncomp, double *out, int64_t ostride,
                                      const uint32_t *bm)
{
    const int len = row ? C.n : C.m;
    Best best{0ull, 0u};
#pragma unroll 1
    for (int e = C.t; e < cnt * len; e += NT * CL) {
        const int r = e / len, x = e - r * len;
        const int I = row ? F0 + r : x, J = row ? x : F0 + r;
        const int re = C.rows[I], ce = C.cols[J];
        double obs[3] = {C.xg[3 * re], C.xg[3 * re + 1], C.xg[3 * re + 2]};
        double f[9];
#pragma unroll
        for (int q = 0; q < 9; ++q) f[q] = C.ev[9 * re + q];
        double t[3];
        if (HS) gf_traction_one_hs(obs, f, C.rec[ce], C.hs[ce], C.hs_mode, C.mu, C.lam, C.nu, C.pass, t);
        else gf_traction_one(obs, f, C.rec[ce], C.mu, C.lam, C.nu, C.pass, t);
        const double *u = C.U + I, *v = C.V + J;
        const int64_t us = C.m, vs = C.n;
        if (ncomp == 1) {
#pragma unroll 4
            for (int q = 0; q < C.k; ++q) t[0] = __dsub_rn(t[0], __dmul_rn(u[3 * q * us], v[3 * q * vs]));
            out[e] = t[0];
        } else {
#pragma unroll 4
            for (int q = 0; q < C.k; ++q) {
#pragma unroll
                for (int c = 0; c < 3; ++c)
                    t[c] = __dsub_rn(t[c], __dmul_rn(u[(3 * q + c) * us], v[(3 * q + c) * vs]));
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) out[c * ostride + e] = t[c];
            if (bm && !bit_get(bm, x)) take(best, magnitude(t[0]), x + 1);
        }
    }
    return best;
}

// Next reference set of 3 after `ref` whose first index is not excluded
// (reset_reference_row/col, src/Hmatrix.py:620-648); scan: none was found.
__device__ inline int next_reference(int ref, int len, const uint32_t *bm, bool &scan)
{
    const int max_attempts = len / 3 + 1;
    int attempt = 0;
    scan = false;
    while (true) {
        ref = ((ref + 3) % len + len) % len;
        ref -= ref % 3;
        attempt++;
        if (!bit_get(bm, ref)) return ref;
        if (attempt > max_attempts) { scan = true; return ref; }
    }
}

template <bool HS, int NT, int CL>
__global__ void __launch_bounds__(NT, HS ? 256 / NT : 512 / NT)
k_aca(const double *__restrict__ xg, const double *__restrict__ ev, const SrcRec *__restrict__ rec,
      const int32_t *__restrict__ rowlist, const int32_t *__restrict__ collist, const AcaTask *__restrict__ tasks,
      double *__restrict__ ws, double mu, double lam, double eps, int rel_mode, int32_t *__restrict__ rank_out,
      int32_t *__restrict__ flag_out, const HsRec *__restrict__ hs, int hs_mode, int max_mn)
{
    constexpr bool SMALL = CL == 1;
    constexpr int GT = NT * CL, NW = NT / 32;
    extern __shared__ uint32_t bits[];
    __shared__ Best red_am[2][2][NW];
    __shared__ double s_red[2][NW], s_uv[2][ACA_TERMS];
    __shared__ double s_ref[SMALL ? 7 * ACA_SMALL : 1];   // small tasks: reference sets and v / alpha

    // The next smaller size's kernel may start with this one.  Every kernel's last CTA ends
    // after the kernel before it, so the smallest one's completion is that of all.
    if (!SMALL) asm volatile("griddepcontrol.launch_dependents;");
    const int task = blockIdx.x / CL, crank = blockIdx.x % CL;
    const AcaTask T = tasks[task];
    const int mx = T.m > T.n ? T.m : T.n;
    const bool bad = T.m < 0 || T.n < 0 || mx > max_mn;   // the pivot bitmaps are sized for max_mn
    const int size = mx <= ACA_SMALL ? 1 : (mx <= ACA_MEDIUM ? 2 : 8);
    if (bad || size != CL) {
        if (bad && SMALL && threadIdx.x == 0) {
            rank_out[task] = 0;
            flag_out[task] = 8;
        }
        if (blockIdx.x == gridDim.x - 1) asm volatile("griddepcontrol.wait;" ::: "memory");
        return;
    }
    const int m = T.m, n = T.n, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t *prevI = bits;
    uint32_t *prevJ = bits + ((m + 31) >> 5);
    for (int e = threadIdx.x; e < ((m + 31) >> 5) + ((n + 31) >> 5); e += NT) bits[e] = 0u;

    AcaCtx C;
    C.xg = xg; C.ev = ev; C.rec = rec; C.hs = hs; C.hs_mode = hs_mode;
    C.rows = rowlist + T.rows_off;
    C.cols = collist + T.cols_off;
    C.mu = mu; C.lam = lam; C.nu = 1.0 / (1.0 + lam / mu) / 2.0;
    C.m = m; C.n = n; C.pass = T.pass; C.k = 0; C.t = crank * NT + threadIdx.x;
    double *base = ws + T.ws_off;
    C.U = base;
    C.V = base + (int64_t)T.kmax * 3 * m;
    double *RIref = C.V + (int64_t)T.kmax * 3 * n;  // [3][n] (A1 only)
    double *RJref = RIref + 3 * (int64_t)n;         // [3][m]
    double *RIs = RJref + 3 * (int64_t)m;           // [3][n]: a row without room in V
    double *RJs = RIs + 3 * (int64_t)n;             // [3][m]: a column without room in U
    double *w = RIs;                                // [n]: v / alpha of the last term
    if (SMALL) {
        RIref = s_ref;
        RJref = s_ref + 3 * ACA_SMALL;
        w = s_ref + 6 * ACA_SMALL;
    }
    task_sync<CL>();

    const int max_iter = m < n ? m : n;
    int flags = 0, parity = 0, nz = 0;
    double frob2 = 0.0;
    bool scan, reset_row = false, reset_col = false;

    int Iref = next_reference(T.iref0, m, prevI, scan), Jref = next_reference(T.jref0, n, prevJ, scan);
    int ni = Iref + 3 <= m ? 3 : m - Iref, nj = Jref + 3 <= n ? 3 : n - Jref;
    residual<HS, NT, CL>(C, true, Iref, ni, 1, RIref, 0, nullptr);
    residual<HS, NT, CL>(C, false, Jref, nj, 1, RJref, 0, nullptr);
    reset_row = reset_col = true;

    for (int it = 0; it < max_iter; ++it) {
        // reference sets brought up to date with the last term (a reset one already is), and the
        // pivot candidates from them (A1 only), in one pass: threads keep their entries
        if (reset_row || reset_col) task_sync<CL>();
        Best cand[2] = {{0ull, 0u}, {0ull, 0u}};      // row (of the column sets), column (of the row sets)
        {
            const double *uq = C.U + (int64_t)3 * (C.k - 1) * m;     // last term's column (A1), when there is one
#pragma unroll 1
            for (int e = C.t; e < n + m; e += GT) {
                const bool col = e < n;
                const int x = col ? e : e - n, len = col ? n : m, cnt = col ? ni : nj, first = col ? Iref : Jref;
                const bool fresh = col ? reset_row : reset_col;
                double *ref = (col ? RIref : RJref) + x;
                const double *other = col ? uq : w;                  // factor of the set's row (column)
                const double mine = fresh ? 0.0 : (col ? w : uq)[x];
                unsigned long long v = 0ull;
#pragma unroll
                for (int r = 0; r < 3; ++r) {
                    if (r < cnt) {
                        double y = ref[(int64_t)r * len];
                        if (!fresh) {
                            y = __dsub_rn(y, __dmul_rn(other[first + r], mine));
                            ref[(int64_t)r * len] = y;
                        }
                        const unsigned long long k = magnitude(y);
                        v = k > v ? k : v;
                    }
                }
                if (!bit_get(col ? prevJ : prevI, x)) take(cand[col ? 1 : 0], v, x + 1);
            }
        }
        task_best<NT, CL>(cand, red_am, parity);
        int Istar = (int)cand[0].i - 1, Jstar = (int)cand[1].i - 1;
        if (Istar < 0 || Jstar < 0) { flags |= 4; break; }  // everything excluded
        // the term's row and column go straight to V and U (unscaled), while there is room
        const int q = C.k;
        const bool room = q < T.kmax;
        double *Uq = room ? C.U + (int64_t)3 * q * m : RJs, *Vq = room ? C.V + (int64_t)3 * q * n : RIs;
        const bool row_first = __longlong_as_double((long long)cand[0].k) > __longlong_as_double((long long)cand[1].k);
#pragma unroll 1
        for (int half = 0; half < 2; ++half) {
            // the first pivot's row (column), whose largest A1 entry gives the other pivot
            const bool row = (half == 0) == row_first;
            Best b[1] = {residual<HS, NT, CL>(C, row, row ? Istar : Jstar, 1, 3, row ? Vq : Uq, row ? n : m,
                                      half == 0 ? (row ? prevJ : prevI) : nullptr)};
            if (half == 0) {
                task_best<NT, CL>(b, red_am, parity);
                (row ? Jstar : Istar) = (int)b[0].i - 1;
            } else {
                task_sync<CL>();
            }
        }
        const double alpha = Vq[Jstar], alpha1 = Vq[(int64_t)n + Jstar], alpha2 = Vq[2 * (int64_t)n + Jstar];
        if (fabs(alpha) < 1e-4) break;
        if (!room) { flags |= 1; break; }
        task_sync<CL>();                 // every thread has read the pivots: V is scaled in place
        if (threadIdx.x == 0) {
            prevI[Istar >> 5] |= 1u << (Istar & 31);
            prevJ[Jstar >> 5] |= 1u << (Jstar & 31);
        }
        const double d0 = alpha + 1e-16, d1 = alpha1 + 1e-16, d2 = alpha2 + 1e-16;
        const bool zeroB = fabs(alpha2) < 1e-10;
        // V rows, v / alpha, and the step size ||u_k|| * ||v_k / alpha|| (A1)
        double su = 0.0, sv = 0.0, cross = 0.0;
#pragma unroll 1
        for (int j = C.t; j < n; j += GT) {
            const double v = Vq[j], wj = v / alpha;
            w[j] = wj;
            Vq[j] = v / d0;
            Vq[(int64_t)n + j] = Vq[(int64_t)n + j] / d1;
            Vq[2 * (int64_t)n + j] = zeroB ? 0.0 : Vq[2 * (int64_t)n + j] / d2;
            sv += wj * wj;
        }
#pragma unroll 1
        for (int i = C.t; i < m; i += GT) {
            su += Uq[i] * Uq[i];
            nz |= Uq[2 * (int64_t)m + i] != 0.0;
        }
        task_sync<CL>();
#pragma unroll 1
        for (int o = 16; o > 0; o >>= 1) {
            su += __shfl_down_sync(0xffffffffu, su, o);
            sv += __shfl_down_sync(0xffffffffu, sv, o);
        }
        if (lane == 0) {
            s_red[0][wid] = su;
            s_red[1][wid] = sv;
        }
        // ||S_k||_F^2 = ||S_{k-1}||^2 + 2 sum_{p<k} (u_p.u_k)(v_p.v_k) + ||u_k||^2 ||v_k||^2.  Each CTA
        // forms the products over its share of the rows and columns, four terms a warp at once;
        // every warp then sums the shares in the same order.
        const int i0 = (int)((int64_t)m * crank / CL), i1 = (int)((int64_t)m * (crank + 1) / CL);
        const int j0 = (int)((int64_t)n * crank / CL), j1 = (int)((int64_t)n * (crank + 1) / CL);
        int pb = 0;
        do {
            const int pe = rel_mode ? (q < pb + ACA_TERMS ? q : pb + ACA_TERMS) : 0;
#pragma unroll 1
            for (int p0 = pb + wid; p0 < pe; p0 += 4 * NW) {
                double uu[4] = {0.0, 0.0, 0.0, 0.0}, vv[4] = {0.0, 0.0, 0.0, 0.0};
                const int np = (pe - p0 + NW - 1) / NW;
                const int64_t us = (int64_t)3 * m * NW, vs = (int64_t)3 * n * NW;
                const double *up = C.U + (int64_t)3 * p0 * m, *vp = C.V + (int64_t)3 * p0 * n;
#pragma unroll 1
                for (int i = i0 + lane; i < i1; i += 32) {
                    const double x = Uq[i];
#pragma unroll
                    for (int t = 0; t < 4; ++t)
                        if (t < np) uu[t] += up[t * us + i] * x;
                }
#pragma unroll 1
                for (int j = j0 + lane; j < j1; j += 32) {
                    const double x = w[j];
#pragma unroll
                    for (int t = 0; t < 4; ++t)
                        if (t < np) vv[t] += vp[t * vs + j] * x;
                }
#pragma unroll 1
                for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        uu[t] += __shfl_down_sync(0xffffffffu, uu[t], o);
                        vv[t] += __shfl_down_sync(0xffffffffu, vv[t], o);
                    }
                if (lane == 0)
#pragma unroll
                    for (int t = 0; t < 4; ++t)
                        if (t < np) {
                            s_uv[0][p0 + t * NW - pb] = uu[t];
                            s_uv[1][p0 + t * NW - pb] = vv[t];
                        }
            }
            task_sync<CL>();
            for (int p = pb + lane; p < pe; p += 32) {
                double uu = 0.0, vv = 0.0;
#pragma unroll 1
                for (int c = 0; c < CL; ++c) {
                    uu += task_peer<CL>(s_uv[0], c)[p - pb];
                    vv += task_peer<CL>(s_uv[1], c)[p - pb];
                }
                cross += uu * vv;
            }
            pb += ACA_TERMS;
            if (rel_mode && pb < q) task_sync<CL>();          // s_uv is written again
        } while (rel_mode && pb < q);
        su = sv = 0.0;
#pragma unroll 1
        for (int e = lane; e < NW * CL; e += 32) {
            su += task_peer<CL>(s_red[0], e / NW)[e % NW];
            sv += task_peer<CL>(s_red[1], e / NW)[e % NW];
        }
#pragma unroll 1
        for (int o = 16; o > 0; o >>= 1) {
            su += __shfl_xor_sync(0xffffffffu, su, o);
            sv += __shfl_xor_sync(0xffffffffu, sv, o);
            cross += __shfl_xor_sync(0xffffffffu, cross, o);
        }
        const double step = sqrt(su * sv);
        bool stop;
        if (rel_mode) {
            frob2 += 2.0 * cross + su * sv;
            stop = step <= eps * sqrt(fabs(frob2));
        } else {
            stop = step < eps;
        }
        C.k = q + 1;
        if (stop) break;
        if (it == max_iter - 1) break;
        reset_row = Iref <= Istar && Istar < Iref + 3;
        reset_col = Jref <= Jstar && Jstar < Jref + 3;
        if (reset_row) {
            Iref = next_reference(Iref, m, prevI, scan);
            if (scan) break;
            ni = Iref + 3 <= m ? 3 : m - Iref;
            residual<HS, NT, CL>(C, true, Iref, ni, 1, RIref, 0, nullptr);
        }
        if (reset_col) {
            Jref = next_reference(Jref, n, prevJ, scan);
            if (scan) break;
            nj = Jref + 3 <= n ? 3 : n - Jref;
            residual<HS, NT, CL>(C, false, Jref, nj, 1, RJref, 0, nullptr);
        }
    }
    // An all-zero B factor is dropped (src/Hmatrix.py:769-775): any thread of the task that saw
    // a non-zero entry.
    if (!SMALL) task_sync<CL>();            // s_red is no longer read
    nz = __syncthreads_or(nz);
    if (!SMALL) {
        if (threadIdx.x == 0) s_red[0][0] = nz;
        task_sync<CL>();
        for (int c = 0; c < CL; ++c) nz |= task_peer<CL>(s_red[0], c)[0] != 0.0;
        task_sync<CL>();                    // a CTA's shared memory outlives the others' reads
    }
    if (!nz) flags |= 2;
    if (C.t == 0) {
        rank_out[task] = C.k;
        flag_out[task] = flags;
    }
    if (blockIdx.x == gridDim.x - 1) asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <bool HS, int NT, int CL, class... A>
static cudaError_t launch_size(bool behind, unsigned nt, int mn, cudaStream_t stream, A... args)
{
    const size_t smem = (size_t)(2 * ((mn + 31) / 32) + 2) * sizeof(uint32_t);       // the pivot bitmaps
    if (smem > 32 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(k_aca<HS, NT, CL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nt * CL);
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (behind) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (CL > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = CL;
        attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, k_aca<HS, NT, CL>, args...);
}

// The sizes of the batch's largest task and below, largest first.
template <bool HS, class... A>
static int launch_aca(unsigned nt, int max_mn, cudaStream_t stream, A... args)
{
    if ((size_t)(2 * ((max_mn + 31) / 32) + 2) * sizeof(uint32_t) > 200 * 1024) return PQ3D_ERR_ARG;
    if (max_mn > ACA_MEDIUM) PQ3D_CHECK((launch_size<HS, 256, 8>(false, nt, max_mn, stream, args...)));
    if (max_mn > ACA_SMALL)
        PQ3D_CHECK((launch_size<HS, 256, 2>(max_mn > ACA_MEDIUM, nt, max_mn < ACA_MEDIUM ? max_mn : ACA_MEDIUM, stream,
                                            args...)));
    PQ3D_CHECK((launch_size<HS, 128, 1>(max_mn > ACA_SMALL, nt, max_mn < ACA_SMALL ? max_mn : ACA_SMALL, stream, args...)));
    return pq3d_launch_status();
}

PQ3D_EXPORT int pq3d_aca_batched(const double *d_xg, const double *d_ev, const void *d_rec,
                                 const int32_t *d_rowlist, const int32_t *d_collist, const void *d_tasks,
                                 int64_t n_tasks, double *d_ws, double mu, double lam, double eps,
                                 int rel_mode, int max_mn, int32_t *d_rank, int32_t *d_flags,
                                 const void *d_hs, int hs_mode, cudaStream_t stream)
{
    if (n_tasks < 0 || max_mn < 0) return PQ3D_ERR_ARG;
    if (hs_mode < 0 || hs_mode > 2 || (hs_mode && !d_hs)) return PQ3D_ERR_ARG;
    if (n_tasks == 0) return PQ3D_OK;
    if (!d_xg || !d_ev || !d_rec || !d_rowlist || !d_collist || !d_tasks || !d_ws || !d_rank || !d_flags)
        return PQ3D_ERR_ARG;
    for (int64_t t0 = 0; t0 < n_tasks; t0 += 65535) {
        const unsigned nt = (unsigned)(n_tasks - t0 < 65535 ? n_tasks - t0 : 65535);
        const AcaTask *tasks = (const AcaTask *)d_tasks + t0;
        const SrcRec *rec = (const SrcRec *)d_rec;
        const HsRec *hs = hs_mode ? (const HsRec *)d_hs : nullptr;
        const int rc = hs_mode ? launch_aca<true>(nt, max_mn, stream, d_xg, d_ev, rec, d_rowlist, d_collist, tasks, d_ws, mu,
                                                  lam, eps, rel_mode, d_rank + t0, d_flags + t0, hs, hs_mode, max_mn)
                               : launch_aca<false>(nt, max_mn, stream, d_xg, d_ev, rec, d_rowlist, d_collist, tasks, d_ws,
                                                   mu, lam, eps, rel_mode, d_rank + t0, d_flags + t0, hs, 0, max_mn);
        if (rc != PQ3D_OK) return rc;
    }
    return PQ3D_OK;
}

// ---------------------------------------------------------------- packing
// Pack one ACA task's factors into the matvec layout (tree order).
struct PackTask {
    int64_t ws_off;      // ACA workspace of this task
    int64_t u_off, v_off; // block offsets in the packed U / V arrays
    int64_t rows_off, cols_off;
    int32_t m, n, kmax, k, pass, kS, kD, K, Q, r0, c0, zeroB;
};

template <typename T>
__device__ inline T cvt(double v);
template <>
__device__ inline double cvt<double>(double v) { return v; }
template <>
__device__ inline float cvt<float>(double v) { return (float)v; }
template <>
__device__ inline __nv_bfloat16 cvt<__nv_bfloat16>(double v) { return __float2bfloat16_rn((float)v); }

// A warp per (term, component) vector pair, 32 warps a task in PACK_SLICES CTAs.  (One CTA over all
// entries of a task, with a 64-bit division each, took 2.4 ms for 20,480 elements in FP64, now 1.14.)
constexpr int PACK_SLICES = 4, PACK_THREADS = 256;

template <typename T, int CW>
__global__ void __launch_bounds__(PACK_THREADS)
k_aca_pack(const PackTask *__restrict__ tasks, const double *__restrict__ ws, const int32_t *__restrict__ rowlist,
           const int32_t *__restrict__ collist, const int32_t *__restrict__ iperm, T *__restrict__ Uout,
           T *__restrict__ Vout)
{
    const PackTask &P = tasks[blockIdx.x];
    const int m = P.m, n = P.n, lane = threadIdx.x & 31;
    const double *U = ws + P.ws_off;
    const double *V = U + (int64_t)P.kmax * 3 * m;
    const int32_t *rows = rowlist + P.rows_off, *cols = collist + P.cols_off;
    constexpr int NW = PACK_SLICES * PACK_THREADS / 32;
    for (int e = blockIdx.y * (PACK_THREADS / 32) + (threadIdx.x >> 5); e < 3 * P.k; e += NW) {
        const int q = e / 3, c = e - 3 * q;
        const bool zero = c == 2 && P.zeroB;
        // U columns of this pass; V rows: S pass c*kS + q, D pass 3kS + c*kD + q
        const int col = P.pass == 0 ? q : P.kS + q, row = P.pass == 0 ? c * P.kS + q : 3 * P.kS + c * P.kD + q;
        const double *u = U + (int64_t)e * m, *v = V + (int64_t)e * n;
#pragma unroll 4
        for (int i = lane; i < m; i += 32)
            Uout[P.u_off + u_index(m, iperm[rows[i]] - P.r0, c, col, CW)] = cvt<T>(zero ? 0.0 : u[i]);
#pragma unroll 4
        for (int j = lane; j < n; j += 32)
            Vout[P.v_off + v_index(P.Q, row, P.c0 % CW + iperm[cols[j]] - P.c0, CW)] = cvt<T>(zero ? 0.0 : v[j]);
    }
}

PQ3D_EXPORT size_t pq3d_pack_task_bytes(void) { return sizeof(PackTask); }

// dtype: 0 = FP64 (CW 2), 1 = FP32 (CW 4), 2 = BF16 (CW 8).  Output arrays must be zeroed.
PQ3D_EXPORT int pq3d_aca_pack(const void *d_tasks, int64_t n_tasks, const double *d_ws, const int32_t *d_rowlist,
                              const int32_t *d_collist, const int32_t *d_iperm, int dtype, void *d_U, void *d_V,
                              cudaStream_t stream)
{
    if (n_tasks < 0) return PQ3D_ERR_ARG;
    if (n_tasks == 0) return PQ3D_OK;
    if (!d_tasks || !d_ws || !d_rowlist || !d_collist || !d_iperm || !d_U || !d_V) return PQ3D_ERR_ARG;
    for (int64_t t0 = 0; t0 < n_tasks; t0 += 65535) {
        const dim3 nt((unsigned)(n_tasks - t0 < 65535 ? n_tasks - t0 : 65535), PACK_SLICES);
        const PackTask *tk = (const PackTask *)d_tasks + t0;
        if (dtype == 0)
            k_aca_pack<double, 2><<<nt, PACK_THREADS, 0, stream>>>(tk, d_ws, d_rowlist, d_collist, d_iperm, (double *)d_U, (double *)d_V);
        else if (dtype == 1)
            k_aca_pack<float, 4><<<nt, PACK_THREADS, 0, stream>>>(tk, d_ws, d_rowlist, d_collist, d_iperm, (float *)d_U, (float *)d_V);
        else if (dtype == 2)
            k_aca_pack<__nv_bfloat16, 8><<<nt, PACK_THREADS, 0, stream>>>(tk, d_ws, d_rowlist, d_collist, d_iperm,
                                                                (__nv_bfloat16 *)d_U, (__nv_bfloat16 *)d_V);
        else
            return PQ3D_ERR_ARG;
    }
    return pq3d_launch_status();
}
