// Green's-function kernels: per-source records, pair evaluations, dense
// near-field block assembly, and the two host-pointer drop-ins with the
// reference's C signatures (src/TDstressFS_C.cpp:2048-2143).
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include <mutex>

#include "pq3d_common.cuh"
#include "td_gf.cuh"
#include "td_hs.cuh"
#include "hm_layout.cuh"

using namespace pq3d;

// ---------------------------------------------------------------- records
__global__ void k_src_records(const double *__restrict__ nodes, const int64_t *__restrict__ tri,
                              int64_t n_elem, SrcRec *__restrict__ rec)
{
    int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= n_elem) return;
    const double *P1 = nodes + 3 * (tri[3 * e + 0] - 1);
    const double *P2 = nodes + 3 * (tri[3 * e + 1] - 1);
    const double *P3 = nodes + 3 * (tri[3 * e + 2] - 1);
    SrcRec s;
    make_src_rec(P1, P2, P3, s);
    rec[e] = s;
}

PQ3D_EXPORT size_t pq3d_src_record_bytes(void) { return sizeof(SrcRec); }

PQ3D_EXPORT int pq3d_src_records(const double *d_nodes, const int64_t *d_tri, int64_t n_elem,
                                 void *d_rec, cudaStream_t stream)
{
    if (n_elem < 0 || (n_elem > 0 && (!d_nodes || !d_tri || !d_rec))) return PQ3D_ERR_ARG;
    if (n_elem == 0) return PQ3D_OK;
    int th = 128;
    k_src_records<<<(unsigned)((n_elem + th - 1) / th), th, 0, stream>>>(d_nodes, d_tri, n_elem, (SrcRec *)d_rec);
    return pq3d_launch_status();
}

__global__ void k_hs_records(const double *__restrict__ nodes, const int64_t *__restrict__ tri, int64_t n_elem,
                             HsRec *__restrict__ hs)
{
    int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= n_elem) return;
    HsRec h;
    make_hs_rec(nodes + 3 * (tri[3 * e + 0] - 1), nodes + 3 * (tri[3 * e + 1] - 1), nodes + 3 * (tri[3 * e + 2] - 1), h);
    hs[e] = h;
}

PQ3D_EXPORT size_t pq3d_hs_record_bytes(void) { return sizeof(HsRec); }

PQ3D_EXPORT int pq3d_hs_records(const double *d_nodes, const int64_t *d_tri, int64_t n_elem, void *d_hs,
                                cudaStream_t stream)
{
    if (n_elem < 0 || (n_elem > 0 && (!d_nodes || !d_tri || !d_hs))) return PQ3D_ERR_ARG;
    if (n_elem == 0) return PQ3D_OK;
    k_hs_records<<<(unsigned)((n_elem + 127) / 128), 128, 0, stream>>>(d_nodes, d_tri, n_elem, (HsRec *)d_hs);
    return pq3d_launch_status();
}

static bool hs_args_ok(const void *hs, int mode) { return mode == 0 || ((mode == 1 || mode == 2) && hs); }

// ---------------------------------------------------------------- traction pairs
// out[p*6 + 0..5] = (A1s, A2s, Bs, A1d, A2d, Bd) for receiver rows[p], source cols[p].
template <bool HS>
__global__ void k_traction_pairs(const double *__restrict__ xg, const double *__restrict__ ev,
                                 const SrcRec *__restrict__ rec, const int64_t *__restrict__ rows,
                                 const int64_t *__restrict__ cols, int64_t npairs, double mu, double lam,
                                 double *__restrict__ out, const HsRec *__restrict__ hs, int hs_mode)
{
    int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (p >= npairs) return;
    int64_t r = rows[p], c = cols[p];
    double nu = 1.0 / (1.0 + lam / mu) / 2.0;
    double obs[3] = {xg[3 * r], xg[3 * r + 1], xg[3 * r + 2]};
    double f[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) f[k] = ev[9 * r + k];
    double t[6];
    if (HS) gf_traction_sd_hs(obs, f, rec[c], hs[c], hs_mode, mu, lam, nu, t);
    else gf_traction_sd(obs, f, rec[c], mu, lam, nu, t);
#pragma unroll
    for (int k = 0; k < 6; ++k) out[6 * p + k] = t[k];
}

PQ3D_EXPORT int pq3d_traction_pairs(const double *d_xg, const double *d_ev, const void *d_rec,
                                    const int64_t *d_rows, const int64_t *d_cols, int64_t npairs,
                                    double mu, double lam, double *d_out, const void *d_hs, int hs_mode,
                                    cudaStream_t stream)
{
    if (npairs < 0 || !hs_args_ok(d_hs, hs_mode)) return PQ3D_ERR_ARG;
    if (npairs == 0) return PQ3D_OK;
    if (!d_xg || !d_ev || !d_rec || !d_rows || !d_cols || !d_out) return PQ3D_ERR_ARG;
    int th = 128;
    const unsigned g = (unsigned)((npairs + th - 1) / th);
    if (hs_mode)
        k_traction_pairs<true><<<g, th, 0, stream>>>(d_xg, d_ev, (const SrcRec *)d_rec, d_rows, d_cols, npairs, mu,
                                                     lam, d_out, (const HsRec *)d_hs, hs_mode);
    else
        k_traction_pairs<false><<<g, th, 0, stream>>>(d_xg, d_ev, (const SrcRec *)d_rec, d_rows, d_cols, npairs, mu,
                                                      lam, d_out, nullptr, 0);
    return pq3d_launch_status();
}

// ---------------------------------------------------------------- stress at points
// Full stress/strain tensors for receivers (X,Y,Z) and sources P (P1, P2, P3 each), general
// Burgers vector (Ts, Ss, Ds); half-space adds the image and free-surface terms.
//
// One source (the reference's row of a block, its grids): the CTA makes the source's records
// once in shared memory, the angles, image and sides each in a lane of their own, instead of
// every thread its own through nine inverse and direct trigonometric functions in a row
// (40,001 receivers in the half space 73 -> 54 us).
// Several sources: one thread per (source, receiver) pair, its records in local memory.
struct PointRecs {
    SrcRec src;
    HsRec hs;
};

template <bool HS>
__device__ void make_point_recs(const double *__restrict__ P, PointRecs &R)
{
    const int t = threadIdx.x;
    if (t < 3 || (HS && t >= 32 && t < 35)) {          // angle t of the source, angle t - 32 of its image
        const double m = t < 3 ? 1.0 : -1.0;
        const int k = t & 31;
        const double P1[3] = {P[0], P[1], m * P[2]}, P2[3] = {P[3], P[4], m * P[5]}, P3[3] = {P[6], P[7], m * P[8]};
        SrcRec s;
        double c[3];
        make_src_frame(P1, P2, P3, s, c);
        SrcRec &o = t < 3 ? R.src : R.hs.img;
        make_src_angle(c[k], o.cA[k], o.sA[k]);
        if (k == 0) {
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                o.vn[j] = s.vn[j]; o.vs[j] = s.vs[j]; o.vd[j] = s.vd[j]; o.P2[j] = s.P2[j];
                o.p1[j] = s.p1[j]; o.p3[j] = s.p3[j]; o.e12[j] = s.e12[j]; o.e13[j] = s.e13[j]; o.e23[j] = s.e23[j];
            }
        }
    } else if (HS && t >= 64 && t < 67) {              // side t - 64
        const int k = t - 64;
        const double A[3] = {P[3 * k], P[3 * k + 1], P[3 * k + 2]};
        const int l = (k + 1) % 3;
        const double B[3] = {P[3 * l], P[3 * l + 1], P[3 * l + 2]};
        HsSide S;
        make_hs_side(A, B, S);
        R.hs.side[k] = S;
    } else if (HS && t == 96) {
        R.hs.surface = (P[2] == 0 && P[5] == 0 && P[8] == 0) ? 1 : 0;
    }
}

template <bool HS, bool ONE>
__global__ void __launch_bounds__(128)
k_stress_points(const double *__restrict__ X, const double *__restrict__ Y, const double *__restrict__ Z,
                int64_t xstride, const double *__restrict__ P, int64_t pstride, int64_t npairs, double Ss, double Ds,
                double Ts, double mu, double lam, int halfspace, double *__restrict__ stress,
                double *__restrict__ strain)
{
    __shared__ PointRecs shared;
    __shared__ double out[2][128 * 6];
    const int64_t p0 = blockIdx.x * (int64_t)128, p = p0 + threadIdx.x;
    const int64_t xi = p * xstride, si = p * pstride;
    const bool on = p < npairs;
    double obs[3];
    if (on) { obs[0] = X[xi]; obs[1] = Y[xi]; obs[2] = Z[xi]; }
    if (ONE) {
        make_point_recs<HS>(P, shared);
        __syncthreads();
    }
    if (on) {
        double e[6], sig[6];
        const double *P1 = P + 9 * si, *P2 = P + 9 * si + 3, *P3 = P + 9 * si + 6;
        SrcRec own;
        if (!ONE) make_src_rec(P1, P2, P3, own);
        const SrcRec &s = ONE ? shared.src : own;
        double X1[3];
        to_td_frame(obs, s, X1);
        double nu = 1.0 / (1.0 + lam / mu) / 2.0;
        const double b[1][3] = {{Ts, Ss, Ds}};
        double ee[1][6];
        td_strain_multi<1, true>(X1, s, nu, b, ee);
        if (HS) {
            HsRec h;
            if (!ONE) make_hs_rec(P1, P2, P3, h);
            hs_add_strain<1, true, true>(obs, s, ONE ? shared.hs : h, nu, b, halfspace, ee);
        }
        for (int c = 0; c < 6; ++c) e[c] = ee[0][c];
        hooke(e, mu, lam, sig);
#pragma unroll
        for (int c = 0; c < 6; ++c) {
            out[0][6 * threadIdx.x + c] = sig[c];
            out[1][6 * threadIdx.x + c] = e[c];
        }
    }
    // consecutive stores: the drop-ins' small calls write host memory here
    __syncthreads();
    const int n6 = 6 * (int)(npairs - p0 < 128 ? npairs - p0 : 128);
    for (int k = threadIdx.x; k < n6; k += 128) stress[6 * p0 + k] = out[0][k];
    if (strain)
        for (int k = threadIdx.x; k < n6; k += 128) strain[6 * p0 + k] = out[1][k];
}

// Device-pointer form of both reference entry points.  n_pts receivers and
// n_src sources, one of which is 1 (xstride/pstride 0 broadcast the single one).
PQ3D_EXPORT int pq3d_stress_points(const double *d_X, const double *d_Y, const double *d_Z, int64_t n_pts,
                                   const double *d_P /* n_src x 9: P1,P2,P3 */, int64_t n_src,
                                   double Ss, double Ds, double Ts, double mu, double lam, int halfspace,
                                   double *d_stress, double *d_strain, cudaStream_t stream)
{
    if (n_pts < 0 || n_src < 0) return PQ3D_ERR_ARG;
    if (n_pts != 1 && n_src != 1 && n_pts != n_src) return PQ3D_ERR_ARG;
    int64_t np = n_pts > n_src ? n_pts : n_src;
    if (n_pts == 0 || n_src == 0) return PQ3D_OK;
    if (!d_X || !d_Y || !d_Z || !d_P || !d_stress) return PQ3D_ERR_ARG;
    if (halfspace < 0 || halfspace > 2) return PQ3D_ERR_ARG;
    const unsigned g = (unsigned)((np + 127) / 128);
    const auto k = n_src == 1 ? (halfspace ? k_stress_points<true, true> : k_stress_points<false, true>)
                              : (halfspace ? k_stress_points<true, false> : k_stress_points<false, false>);
    k<<<g, 128, 0, stream>>>(d_X, d_Y, d_Z, n_pts == 1 ? 0 : 1, d_P, n_src == 1 ? 0 : 1, np, Ss, Ds, Ts, mu, lam,
                             halfspace, d_stress, d_strain);
    return pq3d_launch_status();
}

// Host-pointer drop-ins.  Same signature, argument meaning and output layout as
// the reference (no return value); inputs are staged to the device, the pair
// kernel runs, outputs come back before return.  A CUDA failure is reported on
// stderr and the outputs are filled with NaN (the reference has no error channel).
static void fill_nan(double *a, size_t n)
{
    if (!a) return;
    for (size_t i = 0; i < n; ++i) a[i] = __builtin_nan("");
}

// Staging of the drop-ins: per device, one device buffer and one mapped pinned
// host buffer, grown to the largest call that needs them and kept until exit, and
// one stream.  The reference calls its entry points for every row and column of
// small blocks, so per-call allocations and copies would cost more than the work:
// calls of up to 1 MB pack their inputs into the pinned buffer, which the kernel
// reads and writes in place.  us per call, B200, one copy each way -> in place, on two
// hosts: one source in the full space, 64 receivers 46 -> 36 and 45 -> 34, 1,000 52 -> 45 and
// 50 -> 41, 6,000 89 -> 92 and 86 -> 76, 8,700 114 -> 117 and 107 -> 98; in the half space 56 -> 51 and
// 141 -> 135 for 64 and 8,700 (first host); 64 sources 40 -> 31, 6,000 131 -> 131.  Larger calls are
// bound by the host's copies into the caller's arrays either way.  Calls on a device are
// serialised by a mutex (the buffers are shared).
namespace {
constexpr int kDropinDevices = 64;
struct DropinStage {
    double *buf = nullptr, *hbuf = nullptr;
    size_t cap = 0, hcap = 0;
    cudaStream_t st = nullptr;
};
std::mutex g_dropin_mu[kDropinDevices];
DropinStage g_dropin[kDropinDevices];

int grow(double *&p, size_t &cap, size_t need, bool host)
{
    if (cap >= need) return PQ3D_OK;
    const size_t c = need > 2 * cap ? need : 2 * cap;
    if (p) {
        if (host) cudaFreeHost(p);
        else cudaFree(p);
    }
    p = nullptr;
    cap = 0;
    const cudaError_t e = host ? cudaHostAlloc((void **)&p, c * sizeof(double), cudaHostAllocMapped)
                               : cudaMalloc((void **)&p, c * sizeof(double));
    if (e != cudaSuccess) {
        p = nullptr;
        return PQ3D_ERR_CUDA;
    }
    cap = c;
    return PQ3D_OK;
}
}  // namespace

static int stress_host(const double *X, const double *Y, const double *Z, size_t npt,
                       const double *P9, size_t nsrc, double Ss, double Ds, double Ts, double mu,
                       double lam, bool hs, double *stress, double *strain)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDropinDevices) return PQ3D_ERR_CUDA;
    std::lock_guard<std::mutex> lk(g_dropin_mu[dev]);
    DropinStage &S = g_dropin[dev];
    const size_t np = npt > nsrc ? npt : nsrc;
    const size_t nin = 3 * npt + 9 * nsrc, need = nin + 12 * np;   // inputs, then stress + strain
    if (!S.st && cudaStreamCreateWithFlags(&S.st, cudaStreamNonBlocking) != cudaSuccess) {
        S.st = nullptr;
        return PQ3D_ERR_CUDA;
    }
    // small calls: pack into the mapped buffer; large calls (over 1 MB) copy the
    // caller's arrays directly, where packing would cost more
    const bool packed = need * sizeof(double) <= (size_t(1) << 20);
    if (packed ? grow(S.hbuf, S.hcap, need, true) != PQ3D_OK : grow(S.buf, S.cap, need, false) != PQ3D_OK)
        return PQ3D_ERR_CUDA;
    double *h = S.hbuf, *d = S.buf;
    if (packed && cudaHostGetDevicePointer((void **)&d, h, 0) != cudaSuccess) return PQ3D_ERR_CUDA;
    double *dS = d + nin;
    const cudaStream_t st = S.st;
    const size_t b = npt * sizeof(double), bp = 9 * nsrc * sizeof(double);
    if (packed) {
        memcpy(h, X, b);
        memcpy(h + npt, Y, b);
        memcpy(h + 2 * npt, Z, b);
        memcpy(h + 3 * npt, P9, bp);
    } else if (cudaMemcpyAsync(d, X, b, cudaMemcpyHostToDevice, st) != cudaSuccess ||
               cudaMemcpyAsync(d + npt, Y, b, cudaMemcpyHostToDevice, st) != cudaSuccess ||
               cudaMemcpyAsync(d + 2 * npt, Z, b, cudaMemcpyHostToDevice, st) != cudaSuccess ||
               cudaMemcpyAsync(d + 3 * npt, P9, bp, cudaMemcpyHostToDevice, st) != cudaSuccess) {
        return PQ3D_ERR_CUDA;
    }
    int rc = pq3d_stress_points(d, d + npt, d + 2 * npt, (int64_t)npt, d + 3 * npt, (int64_t)nsrc, Ss, Ds, Ts, mu,
                                lam, hs ? 2 : 0, dS, strain ? dS + 6 * np : nullptr, st);
    if (rc != PQ3D_OK) return rc;
    const size_t bs = 6 * np * sizeof(double);
    if (packed) {
        if (cudaStreamSynchronize(st) != cudaSuccess) return PQ3D_ERR_CUDA;
        memcpy(stress, h + nin, bs);
        if (strain) memcpy(strain, h + nin + 6 * np, bs);
        return PQ3D_OK;
    }
    if (cudaMemcpyAsync(stress, dS, bs, cudaMemcpyDeviceToHost, st) != cudaSuccess) return PQ3D_ERR_CUDA;
    if (strain && cudaMemcpyAsync(strain, dS + 6 * np, bs, cudaMemcpyDeviceToHost, st) != cudaSuccess)
        return PQ3D_ERR_CUDA;
    return cudaStreamSynchronize(st) == cudaSuccess ? PQ3D_OK : PQ3D_ERR_CUDA;
}

// Replaces TDstressFS_C (src/TDstressFS_C.cpp:2048-2095): one source triangle, n receivers.
PQ3D_EXPORT void TDstressFS_C(const double *X, const double *Y, const double *Z, size_t n,
                              const double *P1, const double *P2, const double *P3, double Ss,
                              double Ds, double Ts, double mu, double lambda_, bool jud_halfspace,
                              double *stress, double *strain)
{
    if (n == 0) return;
    if (jud_halfspace) {
        double zmax = Z[0];
        for (size_t i = 1; i < n; ++i) zmax = Z[i] > zmax ? Z[i] : zmax;
        if (zmax > 0 || P1[2] > 0 || P2[2] > 0 || P3[2] > 0)
            printf("Half-space solution: Z coordinates must be negative!\n");
    }
    double P9[9] = {P1[0], P1[1], P1[2], P2[0], P2[1], P2[2], P3[0], P3[1], P3[2]};
    int rc = stress_host(X, Y, Z, n, P9, 1, Ss, Ds, Ts, mu, lambda_, jud_halfspace, stress, strain);
    if (rc != PQ3D_OK) {
        fprintf(stderr, "pq3d TDstressFS_C: CUDA failure %d\n", rc);
        fill_nan(stress, 6 * n);
        fill_nan(strain, 6 * n);
    }
}

// Replaces TDstressEachSourceAtReceiver_C (src/TDstressFS_C.cpp:2098-2143): one
// receiver, n_sources triangles given as flat xyz triplets.
PQ3D_EXPORT void TDstressEachSourceAtReceiver_C(double x, double y, double z, const double *P1_flat,
                                                const double *P2_flat, const double *P3_flat,
                                                size_t n_sources, double Ss, double Ds, double Ts,
                                                double mu, double lambda_, bool jud_halfspace,
                                                double *stress_out, double *strain_out)
{
    if (n_sources == 0) return;
    double *P9 = (double *)malloc(9 * n_sources * sizeof(double));
    if (!P9) {
        fill_nan(stress_out, 6 * n_sources);
        fill_nan(strain_out, 6 * n_sources);
        return;
    }
    for (size_t i = 0; i < n_sources; ++i) {
        for (int k = 0; k < 3; ++k) {
            P9[9 * i + k] = P1_flat[3 * i + k];
            P9[9 * i + 3 + k] = P2_flat[3 * i + k];
            P9[9 * i + 6 + k] = P3_flat[3 * i + k];
        }
        // the reference's warning, once per offending source (its TDstressHS runs per source)
        if (jud_halfspace && (z > 0 || P9[9 * i + 2] > 0 || P9[9 * i + 5] > 0 || P9[9 * i + 8] > 0))
            printf("Half-space solution: Z coordinates must be negative!\n");
    }
    int rc = stress_host(&x, &y, &z, 1, P9, n_sources, Ss, Ds, Ts, mu, lambda_, jud_halfspace, stress_out,
                         strain_out);
    free(P9);
    if (rc != PQ3D_OK) {
        fprintf(stderr, "pq3d TDstressEachSourceAtReceiver_C: CUDA failure %d\n", rc);
        fill_nan(stress_out, 6 * n_sources);
        fill_nan(strain_out, 6 * n_sources);
    }
}

// ---------------------------------------------------------------- dense near-field assembly
// One CTA per dense block (blocks listed largest first).  Entry (i, j) of block b is the
// traction at the element in tree position r0+i due to the element in tree position c0+j,
// written straight into the packed matvec layout (FP64 and/or FP32 copies).
template <bool HS>
__global__ void k_dense_assemble(const double *__restrict__ xg, const double *__restrict__ ev,
                                 const SrcRec *__restrict__ rec, const int32_t *__restrict__ perm,
                                 const DenseBlock *__restrict__ blocks, double mu, double lam,
                                 double *__restrict__ out64, float *__restrict__ out32,
                                 const HsRec *__restrict__ hs, int hs_mode)
{
    const DenseBlock B = blocks[blockIdx.x];
    const double nu = 1.0 / (1.0 + lam / mu) / 2.0;
    const int64_t npairs = (int64_t)B.m * B.n;
    for (int64_t p = threadIdx.x; p < npairs; p += blockDim.x) {
        int i = (int)(p % B.m), j = (int)(p / B.m);
        int r = perm[B.r0 + i], c = perm[B.c0 + j];
        double obs[3] = {xg[3 * r], xg[3 * r + 1], xg[3 * r + 2]};
        double f[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) f[k] = ev[9 * r + k];
        double t[6];
        if (HS) gf_traction_sd_hs(obs, f, rec[c], hs[c], hs_mode, mu, lam, nu, t);
        else gf_traction_sd(obs, f, rec[c], mu, lam, nu, t);
#pragma unroll
        for (int slip = 0; slip < 2; ++slip)
#pragma unroll
            for (int comp = 0; comp < 3; ++comp) {
                double v = t[3 * slip + comp];
                if (out64) out64[B.off64 + dense_index(B.m, i, j + B.c0 % kCW64, comp, slip, kCW64)] = v;
                if (out32) out32[B.off32 + dense_index(B.m, i, j + B.c0 % kCW32, comp, slip, kCW32)] = (float)v;
            }
    }
}

PQ3D_EXPORT int pq3d_dense_assemble(const double *d_xg, const double *d_ev, const void *d_rec,
                                    const int32_t *d_perm, const void *d_blocks, int64_t n_blocks,
                                    double mu, double lam, double *d_out64, float *d_out32,
                                    const void *d_hs, int hs_mode, cudaStream_t stream)
{
    if (n_blocks < 0 || !hs_args_ok(d_hs, hs_mode)) return PQ3D_ERR_ARG;
    if (n_blocks == 0) return PQ3D_OK;
    if (!d_xg || !d_ev || !d_rec || !d_perm || !d_blocks || (!d_out64 && !d_out32)) return PQ3D_ERR_ARG;
    for (int64_t b0 = 0; b0 < n_blocks; b0 += 65535) {
        int64_t nb = n_blocks - b0 < 65535 ? n_blocks - b0 : 65535;
        if (hs_mode)
            k_dense_assemble<true><<<(unsigned)nb, 256, 0, stream>>>(d_xg, d_ev, (const SrcRec *)d_rec, d_perm,
                                                                    (const DenseBlock *)d_blocks + b0, mu, lam,
                                                                    d_out64, d_out32, (const HsRec *)d_hs, hs_mode);
        else
            k_dense_assemble<false><<<(unsigned)nb, 256, 0, stream>>>(d_xg, d_ev, (const SrcRec *)d_rec, d_perm,
                                                                     (const DenseBlock *)d_blocks + b0, mu, lam,
                                                                     d_out64, d_out32, nullptr, 0);
    }
    return pq3d_launch_status();
}
