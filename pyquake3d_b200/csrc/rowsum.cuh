// The H-matvec's row reduction: y[3 i + c] = sum of row i's slots, fixed order.
//
// A row's slots are listed per leaf cluster (leaf_off; leaf_of_row, leaf_ptr), some 20 to
// 130 entries a row, and an entry's slots of consecutive rows are consecutive.  The sums
// are gathers of that list, bound by the latency of their rounds and, at 60k rows, by the
// 40 MB of FP32 slots.  Layout, for a CTA's R consecutive rows:
//  * lanes run over rows and a thread takes the three components of RS_BATCH entries at a
//    time, so 24 loads are in flight (lanes over the 3 R values, which read every sector
//    once instead of three times, had 16 and took 21 us instead of 12 at 60k rows);
//  * NT / R groups of threads share each list, so a short CTA still has all its warps'
//    loads in flight; the groups' sums meet in shared memory;
//  * the last batch is masked, not taken entry by entry.
// With rs_rows giving small problems 16-row CTAs (121 CTAs instead of 8 at 1,936 rows).
#pragma once
#include <stdint.h>

namespace pq3d {

constexpr int RS_STAGE = 2048;   // staged leaf_off entries per CTA (larger ranges read them from global)
constexpr int RS_BATCH = 8;

__device__ __forceinline__ float ld_slot(const float *p)
{
    float v;
    asm volatile("ld.global.cg.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ double ld_slot(const double *p)
{
    double v;
    asm volatile("ld.global.cg.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}

// Rows per CTA (a multiple of 16, at most nt) that spreads n rows over `grid` CTAs.
__host__ __device__ inline int rs_rows(int64_t n, int64_t grid, int nt)
{
    const int64_t r = 16 * ((n + 16 * grid - 1) / (16 * grid));
    return (int)(r < nt ? (r < 16 ? 16 : r) : nt);
}

// Sums of rows [base, min(base + R, end)), base < end: emit(r, sums) receives those of row
// base + r.  All NT threads of the CTA call; the caller synchronises before it reads what
// emit wrote.  R at most NT.
template <int NT, typename TA, class F>
__device__ __forceinline__ void rowsum_rows(const TA *__restrict__ slots, const int32_t *__restrict__ leaf_of_row,
                                            const int32_t *__restrict__ leaf_ptr, const int32_t *__restrict__ leaf_off,
                                            int64_t base, int64_t end, int R, F emit)
{
    __shared__ int s_off[RS_STAGE];
    __shared__ double s_part[3 * NT];
    const int rows = (int)(end - base < R ? end - base : R);
    const int G = NT / R, g = threadIdx.x / R, r = threadIdx.x - g * R;
    // the thread's list, read ahead of the staging: after it, its two round trips to L2 were 2 us
    // of a call (272 rows by CTAs of 256: 3.9 -> 2.1)
    int k = 0, k1 = 0;
    if (g < G && r < rows) {
        const int l = leaf_of_row[base + r];
        k = leaf_ptr[l] + g;
        k1 = leaf_ptr[l + 1];
    }
    // with leaves numbered in row order the CTA's lists are one range of leaf_off
    const int kb = leaf_ptr[leaf_of_row[base]], ke = leaf_ptr[leaf_of_row[base + rows - 1] + 1];
    const bool staged = (unsigned)(ke - kb) <= (unsigned)RS_STAGE;      // ke < kb: another numbering
    __syncthreads();             // s_off and s_part of the CTA's previous rows are no longer read
    if (staged)
        for (int e = kb + (int)threadIdx.x; e < ke; e += NT) s_off[e - kb] = __ldg(leaf_off + e);
    __syncthreads();
    double a[3] = {0.0, 0.0, 0.0};
    const TA *p = slots + 3 * (base + r);
    // unconditional loads (a masked entry repeats the list's last one), so that a batch's list
    // reads and then its slot reads are all in flight; a branch per entry made them a chain, which
    // the compiler also makes of a load it may move to its masked use (hence ld_slot).  The list
    // reads of the next batch go out with the slot reads of this one: from a list too long to
    // stage they are L2 reads.  Sums of 5,120 FP64 rows by CTAs of 256 (long lists), us: 31 with
    // the long lists entry by entry, 16.2 in batches, 12.0 with the list reads ahead.
    auto sum = [&](auto off) {
        int o[RS_BATCH];
        auto list = [&](int e) {
#pragma unroll
            for (int u = 0; u < RS_BATCH; ++u) {
                const int q = e + u * G;
                o[u] = off(q < k1 ? q : k1 - 1);
            }
        };
        if (k < k1) list(k);
#pragma unroll 1
        while (k < k1) {
            TA v[RS_BATCH][3];
#pragma unroll
            for (int u = 0; u < RS_BATCH; ++u) {
                const TA *s = p + 3 * (int64_t)o[u];
                v[u][0] = ld_slot(s);
                v[u][1] = ld_slot(s + 1);
                v[u][2] = ld_slot(s + 2);
            }
            const int kn = k + RS_BATCH * G;
            if (kn < k1) list(kn);
#pragma unroll
            for (int u = 0; u < RS_BATCH; ++u)
#pragma unroll
                for (int c = 0; c < 3; ++c) a[c] += k + u * G < k1 ? (double)v[u][c] : 0.0;
            k = kn;
        }
    };
    // a list outside the range, which another numbering of the leaves has, is read in place
    if (staged && k >= kb && k1 <= ke) sum([&](int e) { return s_off[e - kb]; });
    else sum([&](int e) { return __ldg(leaf_off + e); });
    if (G == 1) {
        if (g == 0 && r < rows) emit(r, a);      // threads R.. NT have no row (R = 208: 48 of them)
        return;
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) s_part[c * NT + threadIdx.x] = a[c];
    __syncthreads();
    if (threadIdx.x < rows) {
#pragma unroll 1
        for (int q = 1; q < G; ++q)
#pragma unroll
            for (int c = 0; c < 3; ++c) a[c] += s_part[c * NT + threadIdx.x + q * R];
        emit(threadIdx.x, a);
    }
}

}  // namespace pq3d
