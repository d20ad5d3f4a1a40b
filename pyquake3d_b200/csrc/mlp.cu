// Training and inference of the Newton-seeding MLP (5 -> 64 -> 64 -> 1, tanh, FP32).
// No counterpart in the reference.  Samples come from the V-mode stepper's own
// Newton solves (vmode.cu logs 5 features + the logit of the solution); the
// stepper evaluates the trained network in its stage kernel.
//
// Parameter layout (4609 floats): W1[64][5], b1[64], W2[64][64], b2[64], W3[64], b3.
// Loss: 0.5 * mean((y - t)^2) over a batch.  One step of training is two launches:
//   k_mlp_grad    tiles of 32 samples per CTA: forward, backward and the CTA's share of
//                 every parameter's gradient, all in shared memory and registers
//   k_mlp_reduce  per parameter: the CTAs' shares in a fixed order (deterministic), then
//                 the Adam update
// Bound: 24.6 kFLOP a sample in FP32 (100 MFLOP = 1.4 us for 4,096 samples); the batch has
// to be spread over the SMs, since each layer is a chain of 64 dependent FMAs.  B = 4,096 on
// B200: 8.4 + 3.4 us, against 110 + 55 + 14 + 2 us for separate forward, backward, weight
// gradient and Adam kernels with one thread a sample (32 CTAs, the hidden vector in local
// memory, activations through HBM); an epoch of 65,536 samples 3.42 -> 0.42 ms.
#include "pq3d_common.cuh"
#include <math.h>

namespace {
constexpr int H = 64, NIN = 5;
constexpr int OFF_W1 = 0, OFF_B1 = 320, OFF_W2 = 384, OFF_B2 = 4480, OFF_W3 = 4544, OFF_B3 = 4608, NP = 4609;

constexpr int TS = 32;            // samples per tile
constexpr int MT = 256;           // threads per CTA
constexpr int WST = H + 4;        // row stride of W2 in shared memory (16-byte rows, rows 4 banks apart)
constexpr int SST = TS + 4;       // row stride of the activations: [unit][sample]
constexpr int NPP = 4612;         // floats per CTA share: NP gradients, [NP] the loss, padding
constexpr int MAX_CTAS = 296;     // two CTAs per SM; more tiles loop

struct Weights {
    float W2[H * WST], W1[H * NIN], b1[H], b2[H], W3[H], b3;
};

// Thread roles.  Layer 1: sample = lane, units 8 * warp + 0..7.  Layers 2 and 3 and the
// backward product: units u0 = 8 * warp + 4 * (lane / 16) + 0..3, samples 2 * (lane % 16) + 0..1
// (per column of W2: one broadcast 16-byte and one 8-byte shared load for eight FMAs).
// All loads of a thread in flight at once, then the stores: in loops they were eight round trips
// to L2, 8,800 of the gradient kernel's 20,000 cycles (11.4 -> 8.4 us).  Scalar, since P has any
// alignment.
__device__ __forceinline__ void load_weights(Weights &w, const float *__restrict__ P)
{
    static_assert(OFF_B1 + H <= 2 * MT && NP - OFF_B2 <= MT, "W1, b1 in two loads; b2, W3, b3 in one");
    const int t = threadIdx.x;
    float q[H * H / MT];
#pragma unroll
    for (int k = 0; k < H * H / MT; ++k) q[k] = P[OFF_W2 + k * MT + t];
    const float head0 = P[OFF_W1 + t], head1 = MT + t < OFF_W2 ? P[OFF_W1 + MT + t] : 0.0f;
    const float tail = OFF_B2 + t < NP ? P[OFF_B2 + t] : 0.0f;
#pragma unroll
    for (int k = 0; k < H * H / MT; ++k) {
        const int e = k * MT + t;
        w.W2[(e >> 6) * WST + (e & 63)] = q[k];
    }
    w.W1[t] = head0;
    if (MT + t < OFF_B1) w.W1[MT + t] = head1;
    else if (MT + t < OFF_W2) w.b1[MT + t - OFF_B1] = head1;
    if (t < H) w.b2[t] = tail;
    else if (t < 2 * H) w.W3[t - H] = tail;
    else if (t == 2 * H) w.b3 = tail;
}

// Samples b0.. of X (0 beyond B) into xs[sample][NIN].
__device__ __forceinline__ void load_tile(float *xs, const float *__restrict__ X, int xstride, int b0, int B)
{
    if (threadIdx.x < TS * NIN) {
        const int s = threadIdx.x / NIN, i = threadIdx.x % NIN;
        xs[threadIdx.x] = b0 + s < B ? X[(int64_t)(b0 + s) * xstride + i] : 0.0f;
    }
}

__device__ __forceinline__ void layer1(const Weights &w, const float *xs, float *h1)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float x[NIN];
#pragma unroll
    for (int i = 0; i < NIN; ++i) x[i] = xs[lane * NIN + i];
#pragma unroll
    for (int k = 0; k < H / 8; ++k) {
        const int j = 8 * warp + k;
        float s = w.b1[j];
#pragma unroll
        for (int i = 0; i < NIN; ++i) s += w.W1[NIN * j + i] * x[i];
        h1[j * SST + lane] = tanhf(s);
    }
}

// h2[a][t] of units u0 + a, samples s0 + t: bias first, then inputs in order.
__device__ __forceinline__ void layer2(const Weights &w, const float *h1, int u0, int s0, float h2[4][2])
{
#pragma unroll
    for (int a = 0; a < 4; ++a) h2[a][0] = h2[a][1] = w.b2[u0 + a];
#pragma unroll 4
    for (int i = 0; i < H; i += 4) {
        float4 q[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) q[a] = *reinterpret_cast<const float4 *>(w.W2 + (u0 + a) * WST + i);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            const float2 h = *reinterpret_cast<const float2 *>(h1 + (i + t) * SST + s0);
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                const float c = t == 0 ? q[a].x : (t == 1 ? q[a].y : (t == 2 ? q[a].z : q[a].w));
                h2[a][0] += c * h.x;
                h2[a][1] += c * h.y;
            }
        }
    }
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        h2[a][0] = tanhf(h2[a][0]);
        h2[a][1] = tanhf(h2[a][1]);
    }
}

// The thread's four units' part of the output, summed over the warp's eight units:
// yp[warp][sample].
__device__ __forceinline__ void output_part(const Weights &w, const float h2[4][2], int u0, int s0, float *yp)
{
    float y0 = 0.0f, y1 = 0.0f;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        y0 += w.W3[u0 + a] * h2[a][0];
        y1 += w.W3[u0 + a] * h2[a][1];
    }
    y0 += __shfl_xor_sync(0xffffffffu, y0, 16);
    y1 += __shfl_xor_sync(0xffffffffu, y1, 16);
    if ((threadIdx.x & 31) < 16) {
        float *o = yp + (threadIdx.x >> 5) * TS + s0;
        o[0] = y0;
        o[1] = y1;
    }
}

__device__ __forceinline__ float output_sum(const Weights &w, const float *yp, int s)
{
    float y = w.b3;
#pragma unroll
    for (int k = 0; k < MT / 32; ++k) y += yp[k * TS + s];
    return y;
}

// Inference: persistent CTAs, the weights loaded once (65,536 samples in 28 us).
__global__ void __launch_bounds__(MT) k_mlp_fwd(const float *__restrict__ P, const float *__restrict__ X, int xstride,
                                                int B, float *__restrict__ Y)
{
    __shared__ __align__(16) Weights w;
    __shared__ __align__(16) float h1[H * SST];
    __shared__ float xs[TS * NIN], yp[MT / 32 * TS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int u0 = 8 * warp + 4 * (lane >> 4), s0 = 2 * (lane & 15);
    load_weights(w, P);
    for (int64_t b0 = (int64_t)blockIdx.x * TS; b0 < B; b0 += (int64_t)gridDim.x * TS) {
        load_tile(xs, X, xstride, (int)b0, B);
        __syncthreads();
        layer1(w, xs, h1);
        __syncthreads();
        float h2[4][2];
        layer2(w, h1, u0, s0, h2);
        output_part(w, h2, u0, s0, yp);
        __syncthreads();
        if (threadIdx.x < TS && b0 + threadIdx.x < B) Y[b0 + threadIdx.x] = output_sum(w, yp, threadIdx.x);
    }
}

// part[blockIdx.x][NPP]: this CTA's share of every gradient over its tiles; loss_part, with the
// same stride, its share of the loss.
// The W2 gradient (64 x 64, a sum over the tile's samples) is 4 x 4 per thread, units
// threadIdx / 16 + 16 a and inputs threadIdx % 16 + 16 b, so the 16-byte reads along the
// samples fall in different banks; the other gradients stay with the thread that holds the
// unit and are summed over its 16 lanes at the end.
__global__ void __launch_bounds__(MT, 2) k_mlp_grad(const float *__restrict__ P, const float *__restrict__ X, int xstride,
                                                    const float *__restrict__ T, int tstride, int B,
                                                    float *__restrict__ part, float *__restrict__ loss_part)
{
    __shared__ __align__(16) Weights w;
    __shared__ __align__(16) float h1[H * SST];
    __shared__ __align__(16) float d2[H * SST];
    __shared__ float xs[TS * NIN], yp[MT / 32 * TS], d3s[TS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int u0 = 8 * warp + 4 * (lane >> 4), s0 = 2 * (lane & 15);
    const int tj = threadIdx.x >> 4, ti = threadIdx.x & 15;
    float gW2[4][4] = {}, gW1[4][NIN] = {}, gb1[4] = {}, gb2[4] = {}, gW3[4] = {}, gb3 = 0.0f, gl = 0.0f;
    load_weights(w, P);
    for (int64_t b0 = (int64_t)blockIdx.x * TS; b0 < B; b0 += (int64_t)gridDim.x * TS) {
        load_tile(xs, X, xstride, (int)b0, B);
        const bool mine = threadIdx.x < TS && b0 + threadIdx.x < B;
        const float target = mine ? T[(b0 + threadIdx.x) * tstride] : 0.0f;   // ahead of its use
        __syncthreads();
        layer1(w, xs, h1);
        __syncthreads();
        float h2[4][2];
        layer2(w, h1, u0, s0, h2);
        output_part(w, h2, u0, s0, yp);
        __syncthreads();
        if (threadIdx.x < TS) {
            float d3 = 0.0f;
            if (mine) {
                const float r = output_sum(w, yp, threadIdx.x) - target;
                d3 = r / (float)B;
                gl += 0.5f * r * r / (float)B;
            }
            d3s[threadIdx.x] = d3;
            gb3 += d3;
        }
        __syncthreads();
        const float e0 = d3s[s0], e1 = d3s[s0 + 1];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const float p = e0 * w.W3[u0 + a] * (1.0f - h2[a][0] * h2[a][0]);
            const float q = e1 * w.W3[u0 + a] * (1.0f - h2[a][1] * h2[a][1]);
            *reinterpret_cast<float2 *>(d2 + (u0 + a) * SST + s0) = make_float2(p, q);
            gb2[a] += p + q;
            gW3[a] += e0 * h2[a][0] + e1 * h2[a][1];
        }
        __syncthreads();
        // d1 of units u0 + a (inputs of layer 2), samples s0, s0 + 1
        float d1[4][2] = {};
#pragma unroll 8
        for (int j = 0; j < H; ++j) {
            const float4 c = *reinterpret_cast<const float4 *>(w.W2 + j * WST + u0);
            const float2 d = *reinterpret_cast<const float2 *>(d2 + j * SST + s0);
            d1[0][0] += c.x * d.x; d1[0][1] += c.x * d.y;
            d1[1][0] += c.y * d.x; d1[1][1] += c.y * d.y;
            d1[2][0] += c.z * d.x; d1[2][1] += c.z * d.y;
            d1[3][0] += c.w * d.x; d1[3][1] += c.w * d.y;
        }
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const float2 h = *reinterpret_cast<const float2 *>(h1 + (u0 + a) * SST + s0);
            const float p = d1[a][0] * (1.0f - h.x * h.x), q = d1[a][1] * (1.0f - h.y * h.y);
            gb1[a] += p + q;
#pragma unroll
            for (int i = 0; i < NIN; ++i) gW1[a][i] += p * xs[s0 * NIN + i] + q * xs[(s0 + 1) * NIN + i];
        }
#pragma unroll 2
        for (int s = 0; s < TS; s += 4) {
            float4 d[4], h[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                d[a] = *reinterpret_cast<const float4 *>(d2 + (tj + 16 * a) * SST + s);
                h[a] = *reinterpret_cast<const float4 *>(h1 + (ti + 16 * a) * SST + s);
            }
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    gW2[a][b] += d[a].x * h[b].x;
                    gW2[a][b] += d[a].y * h[b].y;
                    gW2[a][b] += d[a].z * h[b].z;
                    gW2[a][b] += d[a].w * h[b].w;
                }
        }
        __syncthreads();      // xs, h1 and d2 are rewritten by the next tile
    }
    float *o = part + (int64_t)blockIdx.x * NPP;
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) o[OFF_W2 + H * (tj + 16 * a) + ti + 16 * b] = gW2[a][b];
    auto lanes16 = [](float v) {
#pragma unroll
        for (int m = 8; m > 0; m >>= 1) v += __shfl_xor_sync(0xffffffffu, v, m);
        return v;
    };
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        const float b1 = lanes16(gb1[a]), b2 = lanes16(gb2[a]), w3 = lanes16(gW3[a]);
        float w1[NIN];
#pragma unroll
        for (int i = 0; i < NIN; ++i) w1[i] = lanes16(gW1[a][i]);
        if ((lane & 15) == 0) {
            o[OFF_B1 + u0 + a] = b1;
            o[OFF_B2 + u0 + a] = b2;
            o[OFF_W3 + u0 + a] = w3;
#pragma unroll
            for (int i = 0; i < NIN; ++i) o[OFF_W1 + NIN * (u0 + a) + i] = w1[i];
        }
    }
    if (warp == 0) {
        gb3 = lanes16(gb3);
        gl = lanes16(gl);
        gb3 += __shfl_xor_sync(0xffffffffu, gb3, 16);
        gl += __shfl_xor_sync(0xffffffffu, gl, 16);
        if (lane == 0) {
            o[OFF_B3] = gb3;
            loss_part[(int64_t)blockIdx.x * NPP] = gl;
        }
    }
}

struct Adam {
    float *P, *M, *V;      // P null: no update
    float lr, b1, b2, eps;
    int step;
};

// G[p] = sum of the CTAs' shares: 32 parameters per CTA, eight threads a parameter, each
// over every eighth share in order, so all loads are in flight at once; then Adam.  A single
// share may stand in G itself, so the shares are not read through the read-only path; past L1 (they
// come from other SMs) they take no longer by it (296 shares: 6 us, 8 through L1).
__global__ void __launch_bounds__(256) k_mlp_reduce(const float *part, const float *loss_part, int nblk, float *G,
                                                    float *__restrict__ loss, Adam A)
{
    __shared__ float red[8][33];
    const int c = threadIdx.x & 31, r = threadIdx.x >> 5;
    const int p = blockIdx.x * 32 + c;
    float s = 0.0f;
    if (p <= NP) {
        const float *q = p < NP ? part + p : loss_part;
#pragma unroll 8
        for (int k = r; k < nblk; k += 8) s += __ldcg(q + (int64_t)k * NPP);
    }
    red[r][c] = s;
    __syncthreads();
    if (r != 0 || p > NP) return;
    s = 0.0f;
#pragma unroll
    for (int k = 0; k < 8; ++k) s += red[k][c];
    if (p == NP) {
        if (loss) atomicAdd(loss, s);      // batches of several streams may share the sum
        return;
    }
    G[p] = s;
    if (!A.P) return;
    const float m = A.b1 * A.M[p] + (1.0f - A.b1) * s;
    const float v = A.b2 * A.V[p] + (1.0f - A.b2) * s * s;
    A.M[p] = m;
    A.V[p] = v;
    const float mh = m / (1.0f - powf(A.b1, (float)A.step));
    const float vh = v / (1.0f - powf(A.b2, (float)A.step));
    A.P[p] -= A.lr * mh / (sqrtf(vh) + A.eps);
}

// 258 floats a sample, which callers have always allocated: shares for one CTA per tile from 36
// samples on.
int64_t scratch_floats(int B) { return (int64_t)4 * H * B + 2 * (int64_t)B; }

// CTAs of a gradient over B samples: one per tile, as many as the scratch holds shares for.  One
// CTA needs no scratch but for the loss: its share is the gradient.
int grad_ctas(int B)
{
    int64_t n = ((int64_t)B + TS - 1) / TS;
    const int64_t fit = scratch_floats(B) / NPP;
    n = n < fit ? n : fit;
    n = n < MAX_CTAS ? n : MAX_CTAS;
    return (int)(n > 1 ? n : 1);
}

int gradient(const float *P, const float *X, int xstride, const float *T, int tstride, int B, float *scratch, float *G,
             float *loss, const Adam &A, cudaStream_t stream)
{
    const int n = grad_ctas(B);
    float *part = n > 1 ? scratch : G, *loss_part = n > 1 ? scratch + NP : scratch;
    k_mlp_grad<<<n, MT, 0, stream>>>(P, X, xstride, T, tstride, B, part, loss_part);
    k_mlp_reduce<<<(NP + 32) / 32, 256, 0, stream>>>(part, loss_part, n, G, loss, A);
    return pq3d_launch_status();
}
}  // namespace

PQ3D_EXPORT int pq3d_mlp_param_count(void) { return NP; }

// Scratch for a batch of B samples.
PQ3D_EXPORT int64_t pq3d_mlp_scratch_floats(int B) { return scratch_floats(B); }

// y = MLP(X) for B samples (X rows of xstride floats, the first 5 used).
PQ3D_EXPORT int pq3d_mlp_forward(const float *d_P, const float *d_X, int xstride, int B, float *d_Y,
                                 cudaStream_t stream)
{
    if (!d_P || !d_X || !d_Y || B < 0 || xstride < NIN) return PQ3D_ERR_ARG;
    if (B == 0) return PQ3D_OK;
    const int64_t tiles = ((int64_t)B + TS - 1) / TS;
    k_mlp_fwd<<<(unsigned)(tiles < 4 * 148 ? tiles : 4 * 148), MT, 0, stream>>>(d_P, d_X, xstride, B, d_Y);
    return pq3d_launch_status();
}

// Gradient of 0.5 mean((MLP(X) - T)^2) into d_G (4609 floats); loss added to *d_loss if non-null.
PQ3D_EXPORT int pq3d_mlp_grad(const float *d_P, const float *d_X, int xstride, const float *d_T, int tstride, int B,
                              float *d_scratch, float *d_G, float *d_loss, cudaStream_t stream)
{
    if (!d_P || !d_X || !d_T || !d_scratch || !d_G || B <= 0 || xstride < NIN) return PQ3D_ERR_ARG;
    return gradient(d_P, d_X, xstride, d_T, tstride, B, d_scratch, d_G, d_loss, Adam{}, stream);
}

// One Adam step (gradient of the batch, then the update); step counts from 1.
PQ3D_EXPORT int pq3d_mlp_train_step(float *d_P, float *d_M, float *d_V, const float *d_X, int xstride,
                                    const float *d_T, int tstride, int B, float *d_scratch, float *d_G,
                                    float lr, float beta1, float beta2, float eps, int step, float *d_loss,
                                    cudaStream_t stream)
{
    if (!d_M || !d_V || step < 1) return PQ3D_ERR_ARG;
    if (!d_P || !d_X || !d_T || !d_scratch || !d_G || B <= 0 || xstride < NIN) return PQ3D_ERR_ARG;
    return gradient(d_P, d_X, xstride, d_T, tstride, B, d_scratch, d_G, d_loss,
                    Adam{d_P, d_M, d_V, lr, beta1, beta2, eps, step}, stream);
}
