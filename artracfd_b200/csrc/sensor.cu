// Learned smoothness sensor (no counterpart in the reference).
//
// A small MLP, 10 -> 32 -> 32 -> 1 (ReLU, ReLU, sigmoid), looks at the
// density and pressure on the 5-point stencil i-2..i+2 along a sweep axis and
// predicts whether the WENO5 nonlinear weights (weno5.c:41-55) at the node's
// two interfaces depart from the linear weights C = (0.1, 0.6, 0.3) enough to
// change the reconstruction.  Nodes the network does not flag use the
// linear-weight limit of the same characteristic scheme in the hybrid sweep.
//
// Features: 10 * (q_m - mean(q)) / mean(q) for q = rho then p, m = i-2..i+2.
// Label (training): max over the node's two interfaces, both split fluxes and
// the five characteristic fields of |sum_k (omega_k - C_k) q_k|, the change of
// the reconstruction caused by the departure of the weights, divided by the
// interface's flux scale (|u_s| + c) * max|W|; computed from the method's own
// characteristic fluxes (Roe average, LLF splitting).  A node is non-smooth
// where it exceeds the training threshold.
//
// Kernels: feature/label extraction, MLP forward, MLP loss gradient (tiles of
// 64 samples in shared memory, the weight gradients as products over the tile),
// Adam update, and flag inference for the three sweep axes: a pass that
// stores (rho, p) of every node as float2, then a warp-per-32-nodes pass that
// runs layers 1 and 2 as f16 tensor-core MMAs with f32 accumulation.
#include <algorithm>
#include <cstdint>

#include <cooperative_groups.h>
#include <cuda_fp16.h>

#include "acfd_internal.cuh"
#include "fast_div.h"
#include "flux_math.cuh"

namespace acfd {
namespace sensor {

constexpr int kIn = 10, kH = 32;
constexpr int oW1 = 0, oB1 = kH * kIn, oW2 = oB1 + kH, oB2 = oW2 + kH * kH, oW3 = oB2 + kH, oB3 = oW3 + kH;
constexpr int kParams = oB3 + 1;  // 1441

__device__ __forceinline__ long long node_of(const Grid &g, int i, int j, int k)
{
    return ((long long)k * g.n[1] + j) * g.pitch + i;
}

__device__ __forceinline__ long long stride(const Grid &g, int s)
{
    return s == 0 ? 1LL : (s == 1 ? (long long)g.pitch : (long long)g.pitch * g.n[1]);
}

__device__ __forceinline__ void features(const double *U, long long nn, long long id, long long st, double gm1,
                                         float f[kIn])
{
    double rho[5], p[5], mr = 0.0, mp = 0.0;
#pragma unroll
    for (int m = 0; m < 5; ++m) {
        const long long q = id + (m - 2) * st;
        const double r = U[q];
        const double mx = U[nn + q], my = U[2 * nn + q], mz = U[3 * nn + q], e = U[4 * nn + q];
        rho[m] = r;
        p[m] = (e - 0.5 * (mx * mx + my * my + mz * mz) / r) * gm1;
        mr += r;
        mp += p[m];
    }
    const double ir = 5.0 / mr, ip = 5.0 / mp;
#pragma unroll
    for (int m = 0; m < 5; ++m) {
        f[m] = (float)(10.0 * (rho[m] * ir - 1.0));
        f[5 + m] = (float)(10.0 * (p[m] * ip - 1.0));
    }
}

// WENO5 weights of one stencil (weno5.c:41-55) and how far their departure
// from C moves the reconstruction: |sum_k (omega_k - C_k) q_k| (divided by
// the interface's flux scale by the caller).  At smooth extrema the weights of
// WENO-JS depart from C although the three candidates q_k agree, which this
// measure ignores.
__device__ __forceinline__ double weight_departure(double f0, double f1, double f2, double f3, double f4)
{
    const double eps = 1.0e-6;
    const double t0 = f0 - 2.0 * f1 + f2, u0 = f0 - 4.0 * f1 + 3.0 * f2;
    const double t1 = f1 - 2.0 * f2 + f3, u1 = f1 - f3;
    const double t2 = f2 - 2.0 * f3 + f4, u2 = 3.0 * f2 - 4.0 * f3 + f4;
    const double is0 = (13.0 / 12.0) * t0 * t0 + 0.25 * u0 * u0;
    const double is1 = (13.0 / 12.0) * t1 * t1 + 0.25 * u1 * u1;
    const double is2 = (13.0 / 12.0) * t2 * t2 + 0.25 * u2 * u2;
    const double a0 = 0.1 / ((eps + is0) * (eps + is0));
    const double a1 = 0.6 / ((eps + is1) * (eps + is1));
    const double a2 = 0.3 / ((eps + is2) * (eps + is2));
    const double s = a0 + a1 + a2;
    const double q0 = (2.0 * f0 - 7.0 * f1 + 11.0 * f2) / 6.0;
    const double q1 = (-f1 + 5.0 * f2 + 2.0 * f3) / 6.0;
    const double q2 = (2.0 * f2 + 5.0 * f3 - f4) / 6.0;
    return fabs((a0 / s - 0.1) * q0 + (a1 / s - 0.6) * q1 + (a2 / s - 0.3) * q2);
}

// departure at the interface between node c and c + st (6-point stencil c-2..c+3)
__device__ double interface_departure(const double *U, long long nn, long long c, long long st, int s,
                                      const ModelParams &mp)
{
    double Ust[6][5];
#pragma unroll
    for (int m = 0; m < 6; ++m) {
#pragma unroll
        for (int v = 0; v < 5; ++v) {
            Ust[m][v] = U[v * nn + c + (m - 2) * st];
        }
    }
    double Uo[6];
    fast::interface_state<double>(mp.jacobMean, mp.gamma, Ust[2], Ust[3], Uo);
    const double V[3] = {Uo[1], Uo[2], Uo[3]};
    const double cs = Uo[5];
    const double q = 0.5 * (V[0] * V[0] + V[1] * V[1] + V[2] * V[2]);
    const double d = 1.0 / (2.0 * cs);
    const double b = (mp.gamma - 1.0) * (2.0 * d * d);
    double lam[5] = {V[s] - cs, V[s], V[s], V[s], V[s] + cs};
    const double ls = fabs(V[s]) + cs;
    double W[6][5];
#pragma unroll
    for (int m = 0; m < 6; ++m) {
        const double *u = Ust[m];
        const double A = q * u[0] - V[0] * u[1] - V[1] * u[2] - V[2] * u[3] + u[4];
        const double B = V[s] * u[0] - u[s + 1];
        W[m][0] = b * A + d * B;
        W[m][4] = b * A - d * B;
        for (int t = 0; t < 3; ++t) {
            W[m][t + 1] = (t == s) ? u[0] - 2.0 * b * A : u[t + 1] - 2.0 * b * V[t] * A;
        }
    }
    // flux scale of the interface: (|u_s| + c) times the largest
    // characteristic variable of the stencil
    double wmax = 0.0;
#pragma unroll
    for (int m = 0; m < 6; ++m) {
#pragma unroll
        for (int r = 0; r < 5; ++r) wmax = fmax(wmax, fabs(W[m][r]));
    }
    double dep = 0.0;
#pragma unroll
    for (int r = 0; r < 5; ++r) {
        const double lp = 0.5 * (lam[r] + ls), ln = 0.5 * (lam[r] - ls);
        dep = fmax(dep, weight_departure(lp * W[0][r], lp * W[1][r], lp * W[2][r], lp * W[3][r], lp * W[4][r]));
        dep = fmax(dep, weight_departure(ln * W[5][r], ln * W[4][r], ln * W[3][r], ln * W[2][r], ln * W[1][r]));
    }
    return dep / (ls * wmax + 1.0e-300);
}

__global__ void features_kernel(Grid g, ModelParams mp, const double *U, const int *did, int s, float *feat,
                                float *dep)
{
    const int Lx = g.hi[0] - g.lo[0], Ly = g.hi[1] - g.lo[1], Lz = g.hi[2] - g.lo[2];
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)Lx * Ly * Lz) return;
    const int i = g.lo[0] + (int)(t % Lx);
    const long long rest = t / Lx;
    const int j = g.lo[1] + (int)(rest % Ly);
    const int k = g.lo[2] + (int)(rest / Ly);
    const long long id = node_of(g, i, j, k);
    const long long st = stride(g, s);
    float f[kIn];
    features(U, g.nn, id, st, mp.gamma - 1.0, f);
#pragma unroll
    for (int q = 0; q < kIn; ++q) feat[t * kIn + q] = f[q];
    if (did[id] != 0) {
        dep[t] = -1.0f;  // not a fluid node: no label
        return;
    }
    const double d0 = interface_departure(U, g.nn, id - st, st, s, mp);
    const double d1 = interface_departure(U, g.nn, id, st, s, mp);
    dep[t] = (float)fmax(d0, d1);
}

// ---------------------------------------------------------------------------
// the MLP
// ---------------------------------------------------------------------------
__device__ __forceinline__ float mlp_logit(const float *P, const float x[kIn], float h1[kH], float h2[kH])
{
#pragma unroll 4
    for (int a = 0; a < kH; ++a) {
        float z = P[oB1 + a];
#pragma unroll
        for (int q = 0; q < kIn; ++q) z = fmaf(P[oW1 + a * kIn + q], x[q], z);
        h1[a] = fmaxf(z, 0.0f);
    }
#pragma unroll 4
    for (int a = 0; a < kH; ++a) {
        float z = P[oB2 + a];
#pragma unroll
        for (int q = 0; q < kH; ++q) z = fmaf(P[oW2 + a * kH + q], h1[q], z);
        h2[a] = fmaxf(z, 0.0f);
    }
    float z = P[oB3];
#pragma unroll
    for (int q = 0; q < kH; ++q) z = fmaf(P[oW3 + q], h2[q], z);
    return z;
}

__global__ void mlp_forward_kernel(const float *params, const float *X, int n, float *prob)
{
    __shared__ float P[kParams];
    for (int q = threadIdx.x; q < kParams; q += blockDim.x) P[q] = params[q];
    __syncthreads();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    float x[kIn], h1[kH], h2[kH];
#pragma unroll
    for (int q = 0; q < kIn; ++q) x[q] = X[(long long)t * kIn + q];
    const float z = mlp_logit(P, x, h1, h2);
    prob[t] = 1.0f / (1.0f + expf(-z));
}

__device__ __forceinline__ float warp_sum(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sum over the samples of the weighted binary cross-entropy and of its
// gradient: loss = w*(softplus(z) - y*z), dL/dz = w*(sigmoid(z) - y), with
// w = pos_weight for y = 1.  grad and loss are accumulated (the caller
// zeroes them).
//
// A block takes tiles of 64 samples.  Every layer is a small product over the
// tile in shared memory (rows of one hidden unit, kRow floats apart so that
// float4 reads of consecutive rows do not collide): thread (s, rg) computes the
// units 8 rg .. 8 rg + 7 of sample s forward and backward, then the weight
// gradients -- sums over the samples -- are products of the stored rows, a
// 2 x 2 patch of dW2 per thread, all in FP32.  The sums stay in registers over a
// block's tiles; a cluster of eight blocks adds its sums through distributed
// shared memory and brings them to memory in one atomic per parameter.  (The
// atomics of a parameter follow one another, and each rounds the running sum: one
// per block, 256 of them for 16,384 samples, gave twice the error.)  What bounds
// it is the latency of its six phases (16,384 samples: 256 blocks of one tile); a
// warp reduction per weight and warp, with one thread per sample, took 395 us for
// 16,384 samples.
namespace cg = cooperative_groups;
constexpr int kTile = 64, kRow = kTile + 4, kGradThreads = 256;
constexpr int kGradBlocks = 2 * 148, kGradCluster = 8;
static_assert(kGradBlocks % kGradCluster == 0 && kParams + 1 <= kGradCluster * kGradThreads, "grid of whole clusters");

__device__ __forceinline__ float sum8(float v)
{
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    return v;
}

__device__ __forceinline__ float dot4(float4 a, float4 b, float c)
{
    return fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, fmaf(a.w, b.w, c))));
}

__global__ void __cluster_dims__(kGradCluster, 1, 1) __launch_bounds__(kGradThreads) mlp_grad_kernel(const float *params, const float *X, const float *Y,
                                                                int n, float pos_weight, float *grad, float *loss)
{
    __shared__ __align__(16) float P[(kParams + 4) / 4 * 4];  // then the block's sums and its loss
    __shared__ __align__(16) float sX[kIn * kRow], sH1[kH * kRow], sD2[kH * kRow];
    __shared__ __align__(16) float sQ[kH * kRow];  // H2, then D1
    __shared__ __align__(16) float sdz[kTile];
    __shared__ float sz[4][kTile];
    const int tid = threadIdx.x;
    for (int q = tid; q < kParams; q += kGradThreads) P[q] = params[q];
    const int s = tid & (kTile - 1), rg = tid / kTile, r0 = 8 * rg;  // sample, first unit
    const int row = tid >> 3, part = tid & 7;                        // bias and w3 sums
    const int a0 = tid >> 4, q0 = tid & 15;                          // dW2: rows a0, a0 + 16, columns q0, q0 + 16
    float g2[2][2] = {{0.0f, 0.0f}, {0.0f, 0.0f}}, g1[2] = {0.0f, 0.0f};
    float gb1 = 0.0f, gb2 = 0.0f, gw3 = 0.0f, gb3 = 0.0f, gl = 0.0f;
    const long long tiles = ((long long)n + kTile - 1) / kTile;
    for (long long tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const long long first = tile * kTile;
        const int m = (int)min((long long)kTile, n - first);  // samples of the tile
        __syncthreads();
        for (int q = tid; q < kTile * kIn; q += kGradThreads) {
            const int i = q / kIn;
            sX[(q - i * kIn) * kRow + i] = i < m ? X[first * kIn + q] : 0.0f;
        }
        __syncthreads();
        // layer 1
        float h1[8], h2[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) h1[r] = P[oB1 + r0 + r];
#pragma unroll
        for (int q = 0; q < kIn; ++q) {
            const float x = sX[q * kRow + s];
#pragma unroll
            for (int r = 0; r < 8; ++r) h1[r] = fmaf(P[oW1 + (r0 + r) * kIn + q], x, h1[r]);
        }
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            h1[r] = fmaxf(h1[r], 0.0f);
            sH1[(r0 + r) * kRow + s] = h1[r];
            h2[r] = P[oB2 + r0 + r];
        }
        __syncthreads();
        // layer 2 and this thread's share of the output layer
#pragma unroll 2
        for (int q = 0; q < kH; q += 4) {
            const float x0 = sH1[q * kRow + s], x1 = sH1[(q + 1) * kRow + s];
            const float x2 = sH1[(q + 2) * kRow + s], x3 = sH1[(q + 3) * kRow + s];
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const float4 w = *reinterpret_cast<const float4 *>(P + oW2 + (r0 + r) * kH + q);
                h2[r] = fmaf(w.w, x3, fmaf(w.z, x2, fmaf(w.y, x1, fmaf(w.x, x0, h2[r]))));
            }
        }
        float z = 0.0f;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            h2[r] = fmaxf(h2[r], 0.0f);
            sQ[(r0 + r) * kRow + s] = h2[r];
            z = fmaf(P[oW3 + r0 + r], h2[r], z);
        }
        sz[rg][s] = z;
        __syncthreads();
        if (tid < kTile) {
            const bool valid = s < m;
            const float zz = P[oB3] + ((sz[0][s] + sz[1][s]) + (sz[2][s] + sz[3][s]));
            const float y = valid ? Y[first + s] : 0.0f;
            const float w = valid ? (y > 0.5f ? pos_weight : 1.0f) : 0.0f;
            const float ex = expf(-fabsf(zz));
            const float sp = fmaxf(zz, 0.0f) + log1pf(ex);
            const float sg = zz >= 0.0f ? 1.0f / (1.0f + ex) : ex / (1.0f + ex);
            const float dz = w * (sg - y);
            sdz[s] = dz;
            gl += w * (sp - y * zz);
            gb3 += dz;
        }
        __syncthreads();
        {
            const float dz = sdz[s];
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                sD2[(r0 + r) * kRow + s] = h2[r] > 0.0f ? dz * P[oW3 + r0 + r] : 0.0f;
            }
            // w3: eight samples a thread of this thread's row
            const float4 *h = reinterpret_cast<const float4 *>(sQ + row * kRow + 8 * part);
            const float4 *d = reinterpret_cast<const float4 *>(sdz + 8 * part);
            gw3 += sum8(dot4(h[0], d[0], dot4(h[1], d[1], 0.0f)));
        }
        __syncthreads();
        // layer 2 backward: D1 = (W2^T D2) where layer 1 is active
        float d1[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) d1[r] = 0.0f;
#pragma unroll 4
        for (int a = 0; a < kH; ++a) {
            const float d = sD2[a * kRow + s];
            const float4 w0 = *reinterpret_cast<const float4 *>(P + oW2 + a * kH + r0);
            const float4 w1 = *reinterpret_cast<const float4 *>(P + oW2 + a * kH + r0 + 4);
            d1[0] = fmaf(w0.x, d, d1[0]);
            d1[1] = fmaf(w0.y, d, d1[1]);
            d1[2] = fmaf(w0.z, d, d1[2]);
            d1[3] = fmaf(w0.w, d, d1[3]);
            d1[4] = fmaf(w1.x, d, d1[4]);
            d1[5] = fmaf(w1.y, d, d1[5]);
            d1[6] = fmaf(w1.z, d, d1[6]);
            d1[7] = fmaf(w1.w, d, d1[7]);
        }
#pragma unroll
        for (int r = 0; r < 8; ++r) sQ[(r0 + r) * kRow + s] = h1[r] > 0.0f ? d1[r] : 0.0f;
        // dW2 and the bias of layer 2 (D2 and H1 are complete)
        float p2[2][2] = {{0.0f, 0.0f}, {0.0f, 0.0f}};  // of 16 samples
        for (int t = 0; t < kTile; t += 4) {
            const float4 u0 = *reinterpret_cast<const float4 *>(sD2 + a0 * kRow + t);
            const float4 u1 = *reinterpret_cast<const float4 *>(sD2 + (a0 + 16) * kRow + t);
            const float4 v0 = *reinterpret_cast<const float4 *>(sH1 + q0 * kRow + t);
            const float4 v1 = *reinterpret_cast<const float4 *>(sH1 + (q0 + 16) * kRow + t);
            p2[0][0] = dot4(u0, v0, p2[0][0]);
            p2[0][1] = dot4(u0, v1, p2[0][1]);
            p2[1][0] = dot4(u1, v0, p2[1][0]);
            p2[1][1] = dot4(u1, v1, p2[1][1]);
            if ((t & 12) == 12) {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    g2[i >> 1][i & 1] += p2[i >> 1][i & 1];
                    p2[i >> 1][i & 1] = 0.0f;
                }
            }
        }
        const float4 one = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
        {
            const float4 *d = reinterpret_cast<const float4 *>(sD2 + row * kRow + 8 * part);
            gb2 += sum8(dot4(d[0], one, dot4(d[1], one, 0.0f)));
        }
        __syncthreads();
        // dW1 and the bias of layer 1
        {
            const float4 *d = reinterpret_cast<const float4 *>(sQ + row * kRow + 8 * part);
            gb1 += sum8(dot4(d[0], one, dot4(d[1], one, 0.0f)));
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int w = tid + e * kGradThreads;  // weight a * kIn + q
            if (w < kH * kIn) {
                const int a = w / kIn, q = w - a * kIn;
                for (int t0 = 0; t0 < kTile; t0 += 16) {
                    float acc = 0.0f;
                    for (int t = t0; t < t0 + 16; t += 4) {
                        acc = dot4(*reinterpret_cast<const float4 *>(sQ + a * kRow + t),
                                   *reinterpret_cast<const float4 *>(sX + q * kRow + t), acc);
                    }
                    g1[e] += acc;
                }
            }
        }
    }
    if (tid < kTile) {
        gl = warp_sum(gl);
        gb3 = warp_sum(gb3);
    }
    __syncthreads();
    // every parameter's sum over the block's tiles in the place of the parameter
#pragma unroll
    for (int i = 0; i < 2; ++i) {
#pragma unroll
        for (int j = 0; j < 2; ++j) P[oW2 + (a0 + 16 * i) * kH + q0 + 16 * j] = g2[i][j];
        const int w = tid + i * kGradThreads;
        if (w < kH * kIn) P[oW1 + w] = g1[i];
    }
    if (part == 0) {
        P[oB1 + row] = gb1;
        P[oB2 + row] = gb2;
        P[oW3 + row] = gw3;
    }
    if (tid == 32) {
        sz[0][0] = gl;
        sz[0][1] = gb3;
    }
    __syncthreads();
    if (tid == 0) {
        P[kParams] = gl + sz[0][0];
        P[oB3] = gb3 + sz[0][1];
    }
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    const int q = (int)cluster.block_rank() * kGradThreads + tid;
    if (q <= kParams) {
        float v[kGradCluster];
#pragma unroll
        for (int r = 0; r < kGradCluster; ++r) v[r] = cluster.map_shared_rank(P, r)[q];
        atomicAdd(q < kParams ? &grad[q] : loss,
                  ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7])));
    }
    cluster.sync();  // a block's shared memory stays until the others have read it
}

// Adam (Kingma & Ba 2015) on the summed gradient times `scale`
__global__ void mlp_adam_kernel(float *params, const float *grad, float *m, float *v, int step, float lr, float scale,
                                float b1, float b2, float eps)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= kParams) return;
    const float gq = grad[q] * scale;
    const float mq = b1 * m[q] + (1.0f - b1) * gq;
    const float vq = b2 * v[q] + (1.0f - b2) * gq * gq;
    m[q] = mq;
    v[q] = vq;
    const float mh = mq / (1.0f - powf(b1, (float)step));
    const float vh = vq / (1.0f - powf(b2, (float)step));
    params[q] -= lr * mh / (sqrtf(vh) + eps);
}

// ---------------------------------------------------------------------------
// tensor-core inference
// ---------------------------------------------------------------------------
// pass 1: density and pressure of every node, as float2
__global__ void rho_p_kernel(long long nn, double gm1, const double *U, float2 *rp)
{
    pdl_wait();
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= nn) return;
    const double r = U[id];
    const double mx = U[nn + id], my = U[2 * nn + id], mz = U[3 * nn + id], e = U[4 * nn + id];
    const double p = (e - 0.5 * (mx * mx + my * my + mz * mz) / r) * gm1;
    rp[id] = make_float2((float)r, (float)p);
}

__device__ __forceinline__ uint32_t pack_half2(float lo, float hi)
{
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&h);
}

// D = A (16x16, f16, row) * B (16x8, f16, col) + C (f32)
__device__ __forceinline__ void mma_16816(float d[4], const uint32_t a[4], const uint32_t b[2], const float c[4])
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%10,%11,%12,%13};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(c[0]), "f"(c[1]), "f"(c[2]),
          "f"(c[3]));
}

constexpr int kFlagWarps = 8;

// pass 2: each warp takes 32 consecutive PIN nodes of one sweep axis at a
// time; lane l builds the features of node l into shared memory, then the
// warp runs layer 1 (16x16 . 16x32) and layer 2 (16x32 . 32x32) on tensor
// cores for two 16-row tiles; the output layer is a dot product finished by
// quad shuffles.  Layer-1 accumulators are reused as layer-2 A fragments.
// Flags: flags[s][node] = 1 where the network's logit exceeds the threshold
// or the node is not a fluid node, 0 elsewhere; nodes outside PIN keep the 1
// written when the sensor was loaded.  count (optional) accumulates the flags set.
// div_x, div_y: division by the PIN extents along x and y.
__global__ void __launch_bounds__(kFlagWarps * 32) flags_mma_kernel(Grid g, const float2 *rp, const int *did,
                                                                    const float *params, float logit_threshold,
                                                                    uint8_t *flags, unsigned long long *count,
                                                                    FastDiv div_x, FastDiv div_y)
{
    pdl_wait();
    // one 32 x 16 f16 feature tile per warp, rows padded to 12 words so that
    // the fragment loads (8 rows x 4 words) hit 32 distinct banks
    constexpr int kRow = 12;
    __shared__ uint32_t Xs[kFlagWarps][32 * kRow];
    __shared__ float Zs[kFlagWarps][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int gq = lane >> 2, t = lane & 3;
    // weights as B fragments (k >= 10 of layer 1 are zero padding)
    uint32_t B1[4][2], B2[2][4][2];
    float bias1[4][2], bias2[4][2], w3[4][2];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int n = 8 * j + gq;
        const float *W1 = params + oW1 + n * kIn;
        B1[j][0] = pack_half2(W1[2 * t], W1[2 * t + 1]);
        B1[j][1] = (2 * t + 8 < kIn) ? pack_half2(W1[2 * t + 8], W1[2 * t + 9]) : 0u;
#pragma unroll
        for (int kk = 0; kk < 2; ++kk) {
            const float *W2 = params + oW2 + n * kH + 16 * kk;
            B2[kk][j][0] = pack_half2(W2[2 * t], W2[2 * t + 1]);
            B2[kk][j][1] = pack_half2(W2[2 * t + 8], W2[2 * t + 9]);
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            bias1[j][c] = params[oB1 + 8 * j + 2 * t + c];
            bias2[j][c] = params[oB2 + 8 * j + 2 * t + c];
            w3[j][c] = params[oW3 + 8 * j + 2 * t + c];
        }
    }
    const float b3 = params[oB3];
    // 32-bit work indices (the launcher checks that 3 * PIN and the node
    // count fit): 64-bit divisions would cost more than the network
    const int Lx = g.hi[0] - g.lo[0], Ly = g.hi[1] - g.lo[1], Lz = g.hi[2] - g.lo[2];
    const int pin = Lx * Ly * Lz;
    const int ngroups = ((pin + 31) / 32) * 3;
    const int nwarps = (int)gridDim.x * kFlagWarps;
    const int sy = g.pitch, sz = g.pitch * g.n[1];
    unsigned nflag = 0;
    for (int grp = (int)blockIdx.x * kFlagWarps + w; grp < ngroups; grp += nwarps) {
        const int gq3 = grp / 3;
        const int s = grp - 3 * gq3;
        const int q = gq3 * 32 + lane;
        const bool valid = q < pin;
        long long id = 0;
        float f[kIn];
#pragma unroll
        for (int m = 0; m < kIn; ++m) f[m] = 0.0f;
        if (valid) {
            const int rest = (int)fast_div((uint32_t)q, div_x);
            const int i = g.lo[0] + (q - rest * Lx);
            const int kk = (int)fast_div((uint32_t)rest, div_y);
            const int j = g.lo[1] + (rest - kk * Ly);
            const int k = g.lo[2] + kk;
            id = (long long)(k * sz + j * sy + i);
            const long long st = (s == 0) ? 1 : (s == 1 ? sy : sz);
            float2 v[5];
            float mr = 0.0f, mp = 0.0f;
#pragma unroll
            for (int m = 0; m < 5; ++m) {
                v[m] = rp[id + (m - 2) * st];
                mr += v[m].x;
                mp += v[m].y;
            }
            // 5 / mean, with the approximate division (2 ulp): the features
            // go to f16 next
            const float ir = __fdividef(5.0f, mr), ip = __fdividef(5.0f, mp);
#pragma unroll
            for (int m = 0; m < 5; ++m) {
                f[m] = 10.0f * (v[m].x * ir - 1.0f);
                f[5 + m] = 10.0f * (v[m].y * ip - 1.0f);
            }
        }
        uint32_t *row = &Xs[w][lane * kRow];
#pragma unroll
        for (int m = 0; m < kIn / 2; ++m) row[m] = pack_half2(f[2 * m], f[2 * m + 1]);
#pragma unroll
        for (int m = kIn / 2; m < 8; ++m) row[m] = 0u;
        __syncwarp();
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
            const int r0 = 16 * mt + gq, r1 = r0 + 8;
            uint32_t A[4];
            A[0] = Xs[w][r0 * kRow + t];
            A[1] = Xs[w][r1 * kRow + t];
            A[2] = Xs[w][r0 * kRow + t + 4];
            A[3] = Xs[w][r1 * kRow + t + 4];
            float H1[4][4];
            const float zero[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                mma_16816(H1[j], A, B1[j], zero);
                H1[j][0] = fmaxf(H1[j][0] + bias1[j][0], 0.0f);
                H1[j][1] = fmaxf(H1[j][1] + bias1[j][1], 0.0f);
                H1[j][2] = fmaxf(H1[j][2] + bias1[j][0], 0.0f);
                H1[j][3] = fmaxf(H1[j][3] + bias1[j][1], 0.0f);
            }
            uint32_t A2[2][4];
#pragma unroll
            for (int kk = 0; kk < 2; ++kk) {
                A2[kk][0] = pack_half2(H1[2 * kk][0], H1[2 * kk][1]);
                A2[kk][1] = pack_half2(H1[2 * kk][2], H1[2 * kk][3]);
                A2[kk][2] = pack_half2(H1[2 * kk + 1][0], H1[2 * kk + 1][1]);
                A2[kk][3] = pack_half2(H1[2 * kk + 1][2], H1[2 * kk + 1][3]);
            }
            float z0 = 0.0f, z1 = 0.0f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float H2[4];
                mma_16816(H2, A2[0], B2[0][j], zero);
                mma_16816(H2, A2[1], B2[1][j], H2);
                z0 += fmaxf(H2[0] + bias2[j][0], 0.0f) * w3[j][0] + fmaxf(H2[1] + bias2[j][1], 0.0f) * w3[j][1];
                z1 += fmaxf(H2[2] + bias2[j][0], 0.0f) * w3[j][0] + fmaxf(H2[3] + bias2[j][1], 0.0f) * w3[j][1];
            }
            z0 += __shfl_xor_sync(0xffffffffu, z0, 1);
            z0 += __shfl_xor_sync(0xffffffffu, z0, 2);
            z1 += __shfl_xor_sync(0xffffffffu, z1, 1);
            z1 += __shfl_xor_sync(0xffffffffu, z1, 2);
            if (t == 0) {
                Zs[w][r0] = z0 + b3;
                Zs[w][r1] = z1 + b3;
            }
        }
        __syncwarp();
        if (valid) {
            // a logit that is not a number (a non-physical state) flags the node
            const uint8_t fl = (did[id] != 0 || !(Zs[w][lane] <= logit_threshold)) ? 1 : 0;
            flags[s * g.nn + id] = fl;
            nflag += fl;
        }
        __syncwarp();
    }
    if (count) {
        const unsigned c = __reduce_add_sync(0xffffffffu, nflag);
        if (lane == 0 && c) atomicAdd(count, (unsigned long long)c);
    }
}

}  // namespace sensor

int sensor_param_count()
{
    return sensor::kParams;
}

int launch_sensor_flags(const Grid &g, const ModelParams &m, const double *U, const int *did, const float *params,
                        float logit_threshold, float2 *rho_p, uint8_t *flags, unsigned long long *count,
                        cudaStream_t st)
{
    const long long pin = (long long)(g.hi[0] - g.lo[0]) * (g.hi[1] - g.lo[1]) * (g.hi[2] - g.lo[2]);
    if (pin <= 0) return ACFD_OK;
    if (3 * pin + 96 > (long long)INT32_MAX || g.nn > (long long)INT32_MAX) {
        set_error("sensor flags: case of %lld computed nodes exceeds the 32-bit work indices", pin);
        return ACFD_ERR_ARG;
    }
    ACFD_CUDA(launch_k(sensor::rho_p_kernel, dim3((unsigned)((g.nn + 255) / 256)), dim3(256), 0, st, g.nn,
                       m.gamma - 1.0, U, rho_p));
    const long long groups = ((pin + 31) / 32) * 3;
    // as many blocks as are resident at once: a block loads the weights once and
    // walks its groups (flags of 65^3 nodes 33 -> 27 us, of 129^3 145 -> 139 us, from eight
    // blocks per SM of which three are resident)
    static int resident[64] = {0};
    int dev = 0;
    ACFD_CUDA(cudaGetDevice(&dev));
    int per_chip = dev >= 0 && dev < 64 ? resident[dev] : 0;
    if (per_chip == 0) {
        int per_sm = 0, sms = 0;
        ACFD_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, sensor::flags_mma_kernel,
                                                                sensor::kFlagWarps * 32, 0));
        ACFD_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        per_chip = std::max(1, per_sm * sms);
        if (dev >= 0 && dev < 64) resident[dev] = per_chip;
    }
    const long long blocks =
        std::min<long long>((groups + sensor::kFlagWarps - 1) / sensor::kFlagWarps, per_chip);
    const FastDiv div_x = make_fast_div((uint32_t)(g.hi[0] - g.lo[0]));
    const FastDiv div_y = make_fast_div((uint32_t)(g.hi[1] - g.lo[1]));
    ACFD_CUDA(launch_k(sensor::flags_mma_kernel, dim3((unsigned)blocks), dim3(sensor::kFlagWarps * 32), 0, st, g,
                       (const float2 *)rho_p, did, params, logit_threshold, flags, count, div_x, div_y));
    return ACFD_OK;
}

int launch_sensor_features(const Grid &g, const ModelParams &m, const double *U, const int *did, int s, float *feat,
                           float *dep, cudaStream_t st)
{
    const long long pin = (long long)(g.hi[0] - g.lo[0]) * (g.hi[1] - g.lo[1]) * (g.hi[2] - g.lo[2]);
    if (pin <= 0) return ACFD_OK;
    sensor::features_kernel<<<(unsigned)((pin + 127) / 128), 128, 0, st>>>(g, m, U, did, s, feat, dep);
    ACFD_CUDA(cudaGetLastError());
    return ACFD_OK;
}

}  // namespace acfd

extern "C" {

int acfd_mlp_param_count(void)
{
    return acfd::sensor::kParams;
}

int acfd_mlp_forward(const float *params, const float *X, int n, float *prob, void *stream)
{
    if (!params || !X || !prob || n < 0) {
        acfd::set_error("acfd_mlp_forward: bad arguments");
        return ACFD_ERR_ARG;
    }
    if (n == 0) return ACFD_OK;
    acfd::sensor::mlp_forward_kernel<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(params, X, n, prob);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? ACFD_OK : acfd::cuda_status(e, "mlp_forward launch");
}

int acfd_mlp_grad(const float *params, const float *X, const float *Y, int n, float pos_weight, float *grad,
                  float *loss, void *stream)
{
    if (!params || !X || !Y || !grad || !loss || n < 0) {
        acfd::set_error("acfd_mlp_grad: bad arguments");
        return ACFD_ERR_ARG;
    }
    if (n == 0) return ACFD_OK;
    namespace sn = acfd::sensor;
    const int tiles = (n - 1) / sn::kTile + 1;
    const int clusters = (std::min(tiles, sn::kGradBlocks) + sn::kGradCluster - 1) / sn::kGradCluster;
    sn::mlp_grad_kernel<<<clusters * sn::kGradCluster, sn::kGradThreads, 0, (cudaStream_t)stream>>>(params, X, Y, n, pos_weight, grad, loss);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? ACFD_OK : acfd::cuda_status(e, "mlp_grad launch");
}

int acfd_mlp_adam(float *params, const float *grad, float *m, float *v, int step, float lr, float scale,
                  void *stream)
{
    if (!params || !grad || !m || !v || step < 1) {
        acfd::set_error("acfd_mlp_adam: bad arguments");
        return ACFD_ERR_ARG;
    }
    const int n = acfd::sensor::kParams;
    acfd::sensor::mlp_adam_kernel<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(
        params, grad, m, v, step, lr, scale, 0.9f, 0.999f, 1.0e-8f);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? ACFD_OK : acfd::cuda_status(e, "mlp_adam launch");
}

}  // extern "C"
