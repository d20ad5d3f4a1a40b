// Element-wise pieces of the reference's rate-and-state DP5(4) step, shared by
// the single-fault step kernel (rk.cu) and the ensemble step kernel (ensemble.cu).
#pragma once
#include "pq3d_common.cuh"
#include "rowsum.cuh"

namespace pq3d_rk {

__device__ __forceinline__ double py_min(double a, double b) { return (b < a) ? b : a; }
__device__ __forceinline__ double py_max(double a, double b) { return (b > a) ? b : a; }
__device__ __forceinline__ double nanmax(double a, double b)
{
    if (a != a || b != b) return __longlong_as_double(0x7ff8000000000000ULL);
    return a > b ? a : b;
}

struct Deriv {
    double dpsi, dsig, dt1, dt2;
};

// derivative (src/QDsim.py:760-813); Tno, Tt in MPa, loads in Pa/s.  The same
// expressions, with the quotients shared through per-element (ia = 1/a,
// ib = 1/b, bdc = b/dc) and per-stage (1/(a Tno)) reciprocals.
__device__ __forceinline__ Deriv derivative(double Tno, double Tt1o, double Tt2o, double state, double ia,
                                            double ib, double bdc, double f0, double V0, double slipv,
                                            double AdotV1, double AdotV2, double dsigmadt, double shear,
                                            double eta)
{
    Tno = Tno * 1e6;
    Tt1o = Tt1o * 1e6;
    Tt2o = Tt2o * 1e6;
    const double iaT = ia / Tno;                  // 1 / (a Tno)
    const double sa = -state * ia;
    const double e1p = exp(sa + Tt1o * iaT), e1m = exp(sa - Tt1o * iaT);
    const double e2p = exp(sa + Tt2o * iaT), e2m = exp(sa - Tt2o * iaT);
    const double g1 = V0 * iaT * (e1p + e1m);     // 2 V0/(a Tno) * cosh-term
    const double g2 = V0 * iaT * (e2p + e2m);
    const double dV1dtau = g1, dV2dtau = g2;
    const double iTno = 1.0 / Tno;
    const double dV1dsigma = -g1 * Tt1o * iTno;
    const double dV2dsigma = -g2 * Tt2o * iTno;
    const double dV1dstate = -V0 * ia * (e1p - e1m);
    const double dV2dstate = -V0 * ia * (e2p - e2m);
    double arg = (f0 - state) * ib;
    arg = arg > 700.0 ? 700.0 : (arg < -700.0 ? -700.0 : arg);
    const double dstatedt = bdc * (V0 * exp(arg) - slipv);
    const double dtau1dt = (-AdotV1 + shear - eta * (dV1dsigma * dsigmadt + dV1dstate * dstatedt)) / (1.0 + eta * dV1dtau);
    const double dtau2dt = (-AdotV2 + shear - eta * (dV2dsigma * dsigmadt + dV2dstate * dstatedt)) / (1.0 + eta * dV2dtau);
    return Deriv{dstatedt, dsigmadt * 1e-6, dtau1dt * 1e-6, dtau2dt * 1e-6};
}

// Dormand-Prince 5(4) tableau (src/QDsim.py:1002-1032): rows 0..6 the stages' inputs (row 6 is
// the fifth-order solution), row 7 the embedded one.
static __constant__ double kDp[8][7] = {
    {0, 0, 0, 0, 0, 0, 0},
    {.2, 0, 0, 0, 0, 0, 0},
    {3. / 40, 9. / 40., 0, 0, 0, 0, 0},
    {44. / 45., -56. / 15, 32. / 9, 0, 0, 0, 0},
    {19372. / 6561., -25360 / 2187., 64448. / 6561., -212. / 729., 0, 0, 0},
    {9017. / 3168., -355. / 33., -46732. / 5247., 49. / 176., -5103. / 18656., 0, 0},
    {35. / 384., 0, 500. / 1113., 125. / 192., -2187. / 6784., 11. / 84., 0},
    {5179. / 57600., 0, 7571. / 16695., 393. / 640., -92097. / 339200., 187. / 2100., 1. / 40.}};

// The H-matvec's row reduction (rowsum.cuh) fused into the step kernels: y of the CTA's rows
// [base, min(base + R, end)), with all NT threads taking part.  Other threads of the CTA read
// y afterwards, hence the barrier.
template <int NT, typename TA, class A>
__device__ __forceinline__ void rowsum_cta(const A &S, int64_t base, int64_t end, int R)
{
    double *y = S.y + 3 * base;
    pq3d::rowsum_rows<NT>((const TA *)S.slots, S.leaf_of_row, S.leaf_ptr, S.leaf_off, base, end, R,
                          [y](int r, const double *v) {
                              y[3 * r] = v[0];
                              y[3 * r + 1] = v[1];
                              y[3 * r + 2] = v[2];
                          });
    __syncthreads();
}

// One DP5(4) attempt of size h for element i (RungeKutte_solve_Dormand_Prince,
// src/QDsim.py:1001-1134) with the frozen load y[i] and start-of-step slip rate:
// the 5th-order candidate goes to cand (Tno, Tt1o, Tt2o, psi planes of n), the
// relative error terms |dpsi/psi8|, |dTt1/Tt1_8|, |dTt2/Tt2_8|, |dTno/Tno8| to err.
// FLAT: straight-line stages.  The step kernels, short CTAs that meet at every attempt, take the
// rolled form; the row-range and lock-step kernels lose by it (see below).  Same bits.
template <bool FLAT = false, class A>
__device__ __forceinline__ void dp54_element(const A &S, int64_t i, double h, double err[4])
{
    const int64_t n = S.n;
    const double a = S.a[i], b = S.b[i], dc = S.dc[i], f0 = S.f0[i], sh = S.shear_loading[i];
    const double ia = 1.0 / a, ib = 1.0 / b, bdc = b / dc;
    const double sv = S.slipv[i];
    const double L1 = S.y[3 * i], L2 = S.y[3 * i + 1];
    const double dsg = S.fix_tn ? S.normal_loading[i] : S.y[3 * i + 2] + S.normal_loading[i];
    const double y0[4] = {S.Tno[i], S.Tt1o[i], S.Tt2o[i], S.psi[i]};
    // Rolled, the stages are one loop with the derivatives in local memory (L1).  Unrolled they made
    // k_rk_step 124 KB of code (57 KB rolled) that ran once per attempt, with spills.  An attempt of
    // the row-range kernel, rolled and unrolled, us: 15.2 and 13.2 at 784 rows, 19.1 and 17.1 at 5,120,
    // 43.8 and 41.3 at 60k.
    double k[7][4], y[4] = {y0[0], y0[1], y0[2], y0[3]};
    auto combine = [&](int s, double *o) {
        double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll (FLAT ? 7 : 1)
        for (int j = 0; j < (FLAT ? 7 : s < 7 ? s : 7); ++j) {
            const double w = kDp[s][j];
            if (FLAT ? j >= s || (j == 1 && s >= 6) : w == 0.0) continue;      // the tableau's zeros
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[q] += w * k[j][q];
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) o[q] = y0[q] + h * acc[q];
    };
#pragma unroll (FLAT ? 7 : 1)
    for (int s = 0; s < 7; ++s) {
        if (s > 0) combine(s, y);
        const Deriv d = derivative(y[0], y[1], y[2], y[3], ia, ib, bdc, f0, S.V0, sv, L1, L2, dsg, sh, S.eta);
        k[s][0] = d.dsig;
        k[s][1] = d.dt1;
        k[s][2] = d.dt2;
        k[s][3] = d.dpsi;
    }
    double z[4];
    combine(7, z);
#pragma unroll
    for (int q = 0; q < 4; ++q) S.cand[(int64_t)q * n + i] = y[q];
    err[0] = fabs(fabs(z[3] - y[3]) / z[3]);
    // Relerrormax2 = max(max|dTt1/Tt1|, max|dTt2/Tt2|, max|dTno/Tno|): the three
    // maxima are reduced separately and combined with Python max() afterwards.
    err[1] = fabs(fabs(z[1] - y[1]) / z[1]);
    err[2] = fabs(fabs(z[2] - y[2]) / z[2]);
    err[3] = fabs(fabs(z[0] - y[0]) / z[0]);
}

// Accepted step for element i (src/QDsim.py:960-993): state from cand, slip
// rates, rake, slip, friction, and the next slip-rate deficit in both x layouts
// (:902-903).  Returns the new slip rates (v1o, v2o).  FLAT as above.
template <bool FLAT = false, class A>
__device__ __forceinline__ void accept_element(const A &S, int64_t i, double h, double &v1o, double &v2o)
{
    const int64_t n = S.n;
    const double Tn = S.cand[i], T1 = S.cand[n + i], T2 = S.cand[2 * (int64_t)n + i],
                 ps = S.cand[3 * (int64_t)n + i];
    const double a = S.a[i];
    S.Tno[i] = Tn; S.Tt1o[i] = T1; S.Tt2o[i] = T2; S.psi[i] = ps;
    S.Tt[i] = sqrt(T1 * T1 + T2 * T2);
    const double ex = exp(-ps / a);
    double v1 = 0.0, v2 = 0.0;
#pragma unroll (FLAT ? 2 : 1)
    for (int c = 0; c < 2; ++c) {
        const double v = (2.0 * S.V0) * ex * sinh((c ? T2 : T1) / Tn / a);
        (c ? v2 : v1) = v;
    }
    S.slipv1[i] = v1;
    S.slipv2[i] = v2;
    double vv = sqrt(v1 * v1 + v2 * v2);
    S.rake[i] = atan2(T2, T1);
    if (vv < 1e-30) vv = 1e-30;
    S.slipv[i] = vv;
    const double s1 = S.slip1[i] + v1 * h, s2 = S.slip2[i] + v2 * h;
    S.slip1[i] = s1; S.slip2[i] = s2;
    S.slip[i] = sqrt(s1 * s1 + s2 * s2);
    S.fric[i] = S.Tt[i] / Tn;
    const double x1 = v1 - S.vplc[i] * S.cr0[i];
    const double x2 = v2 - S.vplc[i] * S.sr0[i];
    // interleaved copy (dense blocks) and strike / dip planes (V rows)
    const int64_t P = ((n + 16 + 7) / 8) * 8;
    if (S.x_fp32) {
        float *xf = (float *)S.x;
        xf[2 * i] = (float)x1;
        xf[2 * i + 1] = (float)x2;
        xf[2 * P + i] = (float)x1;
        xf[3 * P + i] = (float)x2;
    } else {
        double *xd = (double *)S.x;
        xd[2 * i] = x1;
        xd[2 * i + 1] = x2;
        xd[2 * P + i] = x1;
        xd[3 * P + i] = x2;
    }
    v1o = v1;
    v2o = v2;
}

// Step-size controller of the reference (src/QDsim.py:931-958) for one attempt
// with error maxima E (psi, Tt1, Tt2, Tno).  Returns true when the attempt ends
// the step (accepted, or given up: h < 1e-15 or more than 20 rejections).
struct StepCtl {
    double h, dtnext;
    int nrjct, attempt;
    bool accepted;
};

// The controller's sizes for error maxima E: the smaller of the two estimates.  The two powers
// one after the other (PAIR false: half the code, for the step kernels, where they run beside the
// state update) or overlapping.
template <bool PAIR>
__device__ __forceinline__ double controller_size(double h, const double E[4], double reltol)
{
    double hnew[2];
#pragma unroll (PAIR ? 2 : 1)
    for (int k = 0; k < 2; ++k) {
        const double R = (k ? py_max(py_max(E[1], E[2]), E[3]) : E[0]) + 1e-10;
        hnew[k] = h * 0.9 * pow(reltol / R, 0.2);
    }
    return py_min(hnew[0], hnew[1]);
}

// The size after an accepted attempt of size h.
template <bool PAIR = false>
__device__ __forceinline__ double controller_next(double h, const double E[4], double reltol)
{
    return py_min(controller_size<PAIR>(h, E, reltol), 1.5 * h);
}

// As controller(), but leaves dtnext of an accepted attempt to controller_next (two powers
// that only the thread that stores it needs).
template <bool PAIR = false>
__device__ __forceinline__ bool controller_decide(StepCtl &c, const double E[4], double reltol, bool forced)
{
    const double R1 = E[0] + 1e-10;
    const double R2 = py_max(py_max(E[1], E[2]), E[3]) + 1e-10;
    const double c1 = R1 / reltol, c2 = R2 / reltol;
    c.attempt++;
    if (forced || (py_max(c1, c2) < 1.0 && !(c1 != c1 || c2 != c2))) {
        c.accepted = true;
        return true;
    }
    c.nrjct++;
    c.dtnext = controller_size<PAIR>(c.h, E, reltol);
    c.h = py_max(0.5 * c.h, c.dtnext);
    return c.h < 1.e-15 || c.nrjct > 20;
}

__device__ __forceinline__ bool controller(StepCtl &c, const double E[4], double reltol, bool forced)
{
    const bool done = controller_decide<true>(c, E, reltol, forced);
    if (c.accepted) c.dtnext = controller_next<true>(c.h, E, reltol);
    return done;
}

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned *p)
{
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ unsigned atom_add_acq_rel_u32(unsigned *p, unsigned x)
{
    unsigned old;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(x) : "memory");
    return old;
}

__device__ __forceinline__ unsigned long long warp_max_u64(unsigned long long k)
{
    const unsigned hi = (unsigned)(k >> 32), mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? (unsigned)k : 0u);
    return ((unsigned long long)mh << 32) | ml;
}

// NaN-propagating max of four values that are >= 0 or +NaN over the `parties` CTAs that
// step one fault (the whole grid in k_rk_step), in one phase.  Every CTA folds its block maximum into a result slot with 64-bit
// atomicMax on the bit patterns (for such values the unsigned order of the
// bits is the order of the values, and +NaN lies above +inf, so the fold is
// nanmax), then arrives on bar with acquire-release semantics; a CTA goes on
// once bar reaches (attempt + 1) * parties and reads the slot.  Attempts
// rotate over three slots of four: the CTA that arrives last at attempt a
// clears slot (a + 2) % 3, which every CTA finished reading before it arrived
// at a and which no CTA touches before the next barrier.  The last CTA to
// finish the step clears bar and the slots.  All CTAs return the same four
// values.  Bounded spin: on timeout ctrl[4] = PQ3D_ERR_TIMEOUT and false is
// returned.
template <int NT>
__device__ __forceinline__ bool fault_max4(double *v, unsigned long long *slots3, unsigned *bar, unsigned parties,
                                           int attempt, double *ctrl)
{
    static_assert(NT == 256, "eight warps: lane 8 q + w reduces maximum q of warp w");
    __shared__ unsigned long long wred[4][NT / 32];
    __shared__ double s_res[4];
    __shared__ int s_ok;
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const unsigned long long m = warp_max_u64((unsigned long long)__double_as_longlong(v[q]));
        if (lane == 0) wred[q][threadIdx.x >> 5] = m;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        unsigned long long *r = slots3 + 4 * (attempt % 3);
        unsigned long long m = wred[lane >> 3][lane & 7];
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) {
            const unsigned long long x = __shfl_xor_sync(0xffffffffu, m, o);
            m = x > m ? x : m;
        }
        if ((lane & 7) == 0) atomicMax(r + (lane >> 3), m);
        __syncwarp();
        if (lane == 0) {
            const unsigned target = (unsigned)(attempt + 1) * parties;
            int ok = 1;
            if (atom_add_acq_rel_u32(bar, 1u) + 1u == target) {
                unsigned long long *z = slots3 + 4 * ((attempt + 2) % 3);
                for (int e = 0; e < 4; ++e) __stcg(z + e, 0ull);
            } else {
                long long it = 0;
                while (ld_acquire_u32(bar) < target) {
                    if (++it > (1LL << 24)) {
                        ctrl[4] = (double)PQ3D_ERR_TIMEOUT;
                        ok = 0;
                        break;
                    }
                    __nanosleep(32);
                }
            }
            s_ok = ok;
        }
        __syncwarp();
        if (lane < 4) s_res[lane] = __longlong_as_double((long long)__ldcg(r + lane));
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = s_res[q];
    return s_ok != 0;
}

// One time step after the load, by each of the fault's CTAs: elements first, first + stride, ...
// below end per thread, attempts from size c.h until the controller ends the step, state update.
// F gives what the CTAs of the fault share: ctrl(), hist() and ctrl_host() (may be null), slots3()
// (3 x 4 error maxima, then 2 slip-rate maxima), bar() and end() (arrivals of the attempts, CTAs
// done with the step), parties() (CTAs of the fault, all co-resident).  Words zeroed once, cleared
// by the last CTA.  Functions, and end in the type of the caller: as a struct of pointers formed up
// front with a 64-bit end, k_rk_step was 0.7 us slower at every size.
template <int NT, class A_, class F_, class I>
__device__ __forceinline__ void step_fault(const A_ &A, const F_ &F, StepCtl c, bool forced, int64_t first, I end,
                                           int64_t stride)
{
    double E[4];

    while (true) {
        double m1 = 0.0, g1 = 0.0, g2 = 0.0, g3 = 0.0;  // max relative errors, NaN-propagating
        for (int64_t i = first; i < end; i += stride) {
            double e[4];
            dp54_element(A, i, c.h, e);
            m1 = nanmax(m1, e[0]);
            g1 = nanmax(g1, e[1]);
            g2 = nanmax(g2, e[2]);
            g3 = nanmax(g3, e[3]);
        }
        // maxima over the fault of (m1, g1, g2, g3); identical in every CTA
        E[0] = m1; E[1] = g1; E[2] = g2; E[3] = g3;
        if (!fault_max4<NT>(E, F.slots3(), F.bar(), F.parties(), c.attempt, F.ctrl())) return;
        if (controller_decide(c, E, A.reltol, forced)) break;
    }
    const double h = c.h;
    // the size after this step: two powers, by a thread of the last warp (idle when R <= 224)
    // while the others update the state
    __shared__ double s_next;
    if (threadIdx.x == NT - 1 && c.accepted) s_next = controller_next(h, E, A.reltol);
    const bool accepted = c.accepted;
    const int nrjct = c.nrjct, attempt = c.attempt;

    // accepted step: state update (src/QDsim.py:960-993) and next deficit (:902-903)
    double mv1 = 0.0, mv2 = 0.0;
    if (accepted) {
        for (int64_t i = first; i < end; i += stride) {
            double v1, v2;
            accept_element(A, i, h, v1, v2);
            mv1 = fmax(mv1, fabs(v1));
            mv2 = fmax(mv2, fabs(v2));
        }
    }
    __shared__ unsigned long long vred[2][NT / 32];
    {
        // >= 0 and never NaN: ordered bits
        const unsigned long long m1 = warp_max_u64((unsigned long long)__double_as_longlong(mv1)),
                                 m2 = warp_max_u64((unsigned long long)__double_as_longlong(mv2));
        if ((threadIdx.x & 31) == 0) {
            vred[0][threadIdx.x >> 5] = m1;
            vred[1][threadIdx.x >> 5] = m2;
        }
    }
    __syncthreads();
    // every CTA folds its slip-rate maxima (>= 0, never NaN) into two words; the last one to
    // finish the step updates ctrl, read ahead of its arrival
    if (threadIdx.x == 0) {
        unsigned long long u1 = vred[0][0], u2 = vred[1][0];
#pragma unroll
        for (int k = 1; k < NT / 32; ++k) {
            u1 = vred[0][k] > u1 ? vred[0][k] : u1;
            u2 = vred[1][k] > u2 ? vred[1][k] : u2;
        }
        const double c2 = F.ctrl()[2], c4 = F.ctrl()[4], c8 = F.ctrl()[8], c9 = F.ctrl()[9], c10 = F.ctrl()[10];
        atomicMax(F.slots3() + 12, u1);
        atomicMax(F.slots3() + 13, u2);
        __threadfence();
        if (atomicAdd(F.end(), 1u) != F.parties() - 1) return;
        __threadfence();
        const double w1 = __longlong_as_double((long long)__ldcg(F.slots3() + 12));
        const double w2 = __longlong_as_double((long long)__ldcg(F.slots3() + 13));
        *F.end() = 0u;
        *F.bar() = 0u;
        for (int q = 0; q < 14; ++q) F.slots3()[q] = 0ull;
        if (accepted) {
            const double t = c2 + h, dtnext = s_next;
            F.ctrl()[2] = t;
            F.ctrl()[0] = dtnext;   // next dttry
            F.ctrl()[1] = h;        // accepted step
            F.ctrl()[3] = nrjct;
            F.ctrl()[5] = w1;
            F.ctrl()[6] = w2;
            F.ctrl()[8] = c8 + 1.0;
            F.ctrl()[9] = c9 + nrjct;
            F.ctrl()[10] = c10 + attempt;
            if (F.hist()) {
                double *hh = F.hist();
                hh[0] = h; hh[1] = dtnext; hh[2] = t; hh[3] = w1; hh[4] = w2; hh[5] = nrjct;
            }
        } else {
            F.ctrl()[1] = h;
            F.ctrl()[3] = nrjct;
            if (c4 == 0.0) F.ctrl()[4] = (double)PQ3D_ERR_DT;
        }
        if (F.ctrl_host()) {
            // the host's copy, sequence number last (a step that ended early leaves it stale)
            for (int k = 0; k < 11; ++k) F.ctrl_host()[k] = F.ctrl()[k];
            __threadfence_system();
            F.ctrl_host()[15] = (double)A.step_index + 1.0;
        }
    }
}

}  // namespace pq3d_rk
