// Packing of the ACA factors into the mixed storage (storage code 3 of the
// H-matvec, hmatvec.cu): each ACA term of a low-rank block is stored as FP32,
// FP16 or INT8 according to how much of its rows' products it can carry.
//
// The reference applies every block in FP64 (blocks_process_MVM,
// src/Hmatrix.py:1445-1538); this storage is the project's own.  The
// classification rests on the size of the error a term can put into a row:
// quantising the term u v^T with a relative error e moves row i of the product
// by about e |u_i| ||v||_1 ||x||_inf, while FP32 storage of the row's operator
// entries already rounds at 2^-24 sum_j |K_ij| ||x||_inf.  The weight of a term is
//     w = max_i (|u_i| / R_i) * ||v||_1 ,   R_i = sum over the near-field (dense)
// blocks of row i of |K_ij| (both slips, largest of the three components), a
// lower bound of the row's absolute sum.  The host picks the class from w and a
// tolerance (hmatrix.py).
//
//   k_nearfield_rowabs   R3[c][i] += sum_j |K^c_ij| over the dense blocks
//   k_term_weights       w per (task, term): max over the three components
//   k_pack_mixed         normalised, quantised factors and per-row scales; an INT8
//                        entry b = round(127 v / max|v|) is stored as the byte b + 128
#include "pq3d_common.cuh"
#include "hm_layout.cuh"
#include <cuda_fp16.h>

using namespace pq3d;

namespace {

// One ACA task (block, slip pass) of the mixed packing.  tmap[tmap_off + q]
// holds the class of term q (bits 0-1) and its position among this pass's
// terms of that class (bits 2+).
struct PackTaskM {
    int64_t ws_off, rows_off, cols_off, tmap_off;
    int64_t u_off[3], v_off[3];    // block offsets in the FP32 / FP16 / INT8 arrays
    int32_t m, n, kmax, k, pass, r0, c0, zeroB;
    int32_t kS[3], kD[3], Q[3], K[3], sb[3];
    int32_t pad;
};

// The packing kernels give a warp one (term, component) vector pair of a task: 32 warps a task in
// PACK_SLICES CTAs, so that a task of 10 to 40 terms has them all in flight.  One CTA walking the
// terms with block reductions took 1.7 (weights) and 2.8 ms (packing) for the 20,480-element
// fault, now 0.61 and 0.99.
constexpr int PACK_SLICES = 4, PACK_THREADS = 256, PACK_WARPS = PACK_SLICES * PACK_THREADS / 32;

__device__ __forceinline__ int pack_warp() { return (int)(blockIdx.y * (PACK_THREADS / 32) + (threadIdx.x >> 5)); }

__device__ __forceinline__ double warp_max(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

__device__ __forceinline__ double warp_add(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// One CTA per dense block: threads over rows, each summing |K| over the block's
// columns for the three components (both slips).
__global__ void k_nearfield_rowabs(const float *__restrict__ D, const DenseBlock *__restrict__ blocks, int n,
                                   double *__restrict__ R3)
{
    const DenseBlock b = blocks[blockIdx.x];
    const int ng = (b.n + b.c0 % kCW32 + kCW32 - 1) / kCW32;
    for (int i = threadIdx.x; i < b.m; i += blockDim.x) {
        double a[3] = {0.0, 0.0, 0.0};
        for (int g = 0; g < ng; ++g)
            for (int c = 0; c < 3; ++c)
                for (int s = 0; s < 2; ++s) {
                    const float *p = D + b.off32 + (((int64_t)g * 6 + 2 * c + s) * b.m + i) * kCW32;
#pragma unroll
                    for (int t = 0; t < kCW32; ++t) a[c] += fabs((double)p[t]);
                }
        for (int c = 0; c < 3; ++c) atomicAdd(&R3[(int64_t)c * n + b.r0 + i], a[c]);
    }
}

// w of every term (largest over the components; the B factor is skipped when the packing drops it).
__global__ void __launch_bounds__(PACK_THREADS)
k_term_weights(const PackTaskM *__restrict__ tasks, const double *__restrict__ ws, const int32_t *__restrict__ rowlist,
               const int32_t *__restrict__ iperm, const double *__restrict__ R, double *__restrict__ w_out)
{
    const PackTaskM &P = tasks[blockIdx.x];
    const int m = P.m, n = P.n, lane = threadIdx.x & 31;
    const double *U = ws + P.ws_off;
    const double *V = U + (int64_t)P.kmax * 3 * m;
    const int32_t *rows = rowlist + P.rows_off;
    for (int q = pack_warp(); q < P.k; q += PACK_WARPS) {
        double um[3] = {0.0, 0.0, 0.0}, vs[3] = {0.0, 0.0, 0.0};
        const double *u = U + (int64_t)q * 3 * m, *v = V + (int64_t)q * 3 * n;
#pragma unroll 2
        for (int i = lane; i < m; i += 32) {
            const double r = R[iperm[rows[i]]];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const double a = fabs(u[(int64_t)c * m + i]);
                um[c] = fmax(um[c], r > 0.0 ? a / r : (a > 0.0 ? INFINITY : 0.0));
            }
        }
#pragma unroll 2
        for (int j = lane; j < n; j += 32)
#pragma unroll
            for (int c = 0; c < 3; ++c) vs[c] += fabs(v[(int64_t)c * n + j]);
        double w = 0.0;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double x = warp_max(um[c]) * warp_add(vs[c]);
            if (c < 2 || !P.zeroB) w = fmax(w, x);
        }
        if (lane == 0) w_out[P.tmap_off + q] = w;
    }
}

__global__ void __launch_bounds__(PACK_THREADS)
k_pack_mixed(const PackTaskM *__restrict__ tasks, const double *__restrict__ ws, const int32_t *__restrict__ rowlist,
             const int32_t *__restrict__ collist, const int32_t *__restrict__ iperm, const int32_t *__restrict__ tmap,
             float *__restrict__ U32, __half *__restrict__ U16, uint8_t *__restrict__ U8, float *__restrict__ V32,
             __half *__restrict__ V16, uint8_t *__restrict__ V8, float *__restrict__ scales)
{
    const PackTaskM &P = tasks[blockIdx.x];
    const int m = P.m, n = P.n, lane = threadIdx.x & 31;
    const double *U = ws + P.ws_off;
    const double *V = U + (int64_t)P.kmax * 3 * m;
    const int32_t *rows = rowlist + P.rows_off, *cols = collist + P.cols_off;
    for (int e = pack_warp(); e < 3 * P.k; e += PACK_WARPS) {
        const int q = e / 3, c = e - 3 * q;
        if (c == 2 && P.zeroB) continue;                                      // dropped B factor: zeros
        const int code = tmap[P.tmap_off + q];
        const int cls = code & 3, pos = code >> 2;
        const int col = P.pass == 0 ? pos : P.kS[cls] + pos;                 // U column within the class
        const int row = P.pass == 0 ? c * P.kS[cls] + pos : 3 * P.kS[cls] + c * P.kD[cls] + pos;  // V row
        const double *u = U + (int64_t)e * m;
        const double *v = V + (int64_t)e * n;
        if (cls == 0) {
#pragma unroll 4
            for (int i = lane; i < m; i += 32)
                U32[P.u_off[0] + u_index(m, iperm[rows[i]] - P.r0, c, col, 4)] = (float)u[i];
#pragma unroll 4
            for (int j = lane; j < n; j += 32)
                V32[P.v_off[0] + v_index(P.Q[0], row, P.c0 % 4 + iperm[cols[j]] - P.c0, 4)] = (float)v[j];
            continue;
        }
        double su = 0.0, sv = 0.0;
#pragma unroll 4
        for (int i = lane; i < m; i += 32) su = fmax(su, fabs(u[i]));
#pragma unroll 4
        for (int j = lane; j < n; j += 32) sv = fmax(sv, fabs(v[j]));
        su = warp_max(su);
        sv = warp_max(sv);
        if (!(su > 0.0) || !(sv > 0.0)) continue;                             // an all-zero term stays zero
        if (cls == 1) {
#pragma unroll 2
            for (int i = lane; i < m; i += 32)
                U16[P.u_off[1] + u_index(m, iperm[rows[i]] - P.r0, c, col, 8)] = __float2half_rn((float)(u[i] / su));
#pragma unroll 2
            for (int j = lane; j < n; j += 32)
                V16[P.v_off[1] + v_index(P.Q[1], row, P.c0 % 8 + iperm[cols[j]] - P.c0, 8)] =
                    __float2half_rn((float)(v[j] / sv));
            if (lane == 0) scales[P.sb[1] + row] = (float)(su * sv);
        } else {
#pragma unroll 2
            for (int i = lane; i < m; i += 32) {
                const double t = fmin(127.0, fmax(-127.0, rint(127.0 * u[i] / su)));
                U8[P.u_off[2] + u_index(m, iperm[rows[i]] - P.r0, c, col, 16)] = (uint8_t)(t + 128.0);
            }
#pragma unroll 2
            for (int j = lane; j < n; j += 32) {
                const double t = fmin(127.0, fmax(-127.0, rint(127.0 * v[j] / sv)));
                V8[P.v_off[2] + v_index(P.Q[2], row, P.c0 % 16 + iperm[cols[j]] - P.c0, 16)] = (uint8_t)(t + 128.0);
            }
            if (lane == 0) scales[P.sb[2] + row] = (float)(su * sv / (127.0 * 127.0));
        }
    }
}

}  // namespace

PQ3D_EXPORT size_t pq3d_pack_mixed_task_bytes(void) { return sizeof(PackTaskM); }

PQ3D_EXPORT int pq3d_nearfield_rowabs(const float *d_dense32, const void *d_blocks, int64_t n_blocks, int n,
                                      double *d_R3, cudaStream_t stream)
{
    if (n_blocks < 0 || n <= 0) return PQ3D_ERR_ARG;
    if (n_blocks == 0) return PQ3D_OK;
    if (!d_dense32 || !d_blocks || !d_R3) return PQ3D_ERR_ARG;
    for (int64_t b0 = 0; b0 < n_blocks; b0 += 65535) {
        const unsigned nb = (unsigned)(n_blocks - b0 < 65535 ? n_blocks - b0 : 65535);
        k_nearfield_rowabs<<<nb, 128, 0, stream>>>(d_dense32, (const DenseBlock *)d_blocks + b0, n, d_R3);
    }
    return pq3d_launch_status();
}

PQ3D_EXPORT int pq3d_aca_term_weights(const void *d_tasks, int64_t n_tasks, const double *d_ws,
                                      const int32_t *d_rowlist, const int32_t *d_iperm, const double *d_R,
                                      double *d_w, cudaStream_t stream)
{
    if (n_tasks < 0) return PQ3D_ERR_ARG;
    if (n_tasks == 0) return PQ3D_OK;
    if (!d_tasks || !d_ws || !d_rowlist || !d_iperm || !d_R || !d_w) return PQ3D_ERR_ARG;
    for (int64_t t0 = 0; t0 < n_tasks; t0 += 65535) {
        const unsigned nt = (unsigned)(n_tasks - t0 < 65535 ? n_tasks - t0 : 65535);
        k_term_weights<<<dim3(nt, PACK_SLICES), PACK_THREADS, 0, stream>>>((const PackTaskM *)d_tasks + t0, d_ws, d_rowlist, d_iperm, d_R, d_w);
    }
    return pq3d_launch_status();
}

PQ3D_EXPORT int pq3d_aca_pack_mixed(const void *d_tasks, int64_t n_tasks, const double *d_ws,
                                    const int32_t *d_rowlist, const int32_t *d_collist, const int32_t *d_iperm,
                                    const int32_t *d_tmap, float *d_U32, void *d_U16, void *d_U8, float *d_V32,
                                    void *d_V16, void *d_V8, float *d_scales, cudaStream_t stream)
{
    if (n_tasks < 0) return PQ3D_ERR_ARG;
    if (n_tasks == 0) return PQ3D_OK;
    if (!d_tasks || !d_ws || !d_rowlist || !d_collist || !d_iperm || !d_tmap || !d_U32 || !d_U16 || !d_U8 ||
        !d_V32 || !d_V16 || !d_V8 || !d_scales)
        return PQ3D_ERR_ARG;
    for (int64_t t0 = 0; t0 < n_tasks; t0 += 65535) {
        const unsigned nt = (unsigned)(n_tasks - t0 < 65535 ? n_tasks - t0 : 65535);
        k_pack_mixed<<<dim3(nt, PACK_SLICES), PACK_THREADS, 0, stream>>>((const PackTaskM *)d_tasks + t0, d_ws, d_rowlist, d_collist, d_iperm,
                                             d_tmap, d_U32, (__half *)d_U16, (uint8_t *)d_U8, d_V32, (__half *)d_V16,
                                             (uint8_t *)d_V8, d_scales);
    }
    return pq3d_launch_status();
}
