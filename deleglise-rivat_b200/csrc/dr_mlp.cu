// dr_mlp.cu -- the learned parameter tuner: a 4-64-64-4 FP32 MLP with
// hand-written forward, backward and Adam kernels, and the proposal path that
// turns its outputs into engine parameters (with the endpoint-coverage check
// and the fallback to the reference heuristic).  No counterpart in the
// reference, which picks its parameters by fixed heuristics
// (mertens_dr.hpp:914-962, 1401-1419).
//
// Features (inputs):  log10 X, log2 HBM budget (bytes), SM count, batch size.
// Outputs:            cx, log2 fx, log2 u_cap, log2 segment length, where
//                     u = min(fx * (X / ln ln X)^(2/3), u_cap).
// Inputs and outputs are normalised by fixed affine maps (kIn*, kOut*) so the
// network works on O(1) values.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "../../include/dr_engine.h"
#include "dr_kernels.cuh"
#include "dr_params.hpp"

using namespace drb;

namespace {

constexpr int kIn = 4, kHid = 64, kOut = 4;
// parameter layout: W1[64][4] b1[64] W2[64][64] b2[64] W3[4][64] b3[4]
constexpr int oW1 = 0, oB1 = oW1 + kHid * kIn, oW2 = oB1 + kHid, oB2 = oW2 + kHid * kHid, oW3 = oB2 + kHid,
              oB3 = oW3 + kOut * kHid, kParams = oB3 + kOut;  // 4740
constexpr int kMaxBatch = 4096;

// feature / target normalisation (shared with the numpy oracle in oracle/mlp_oracle.py)
constexpr float kInMean[kIn] = {13.0f, 35.0f, 148.0f, 0.0f};
constexpr float kInScale[kIn] = {3.0f, 3.0f, 64.0f, 8.0f};
constexpr float kOutMean[kOut] = {1.2f, 0.0f, 34.0f, 16.0f};
constexpr float kOutScale[kOut] = {0.5f, 1.5f, 4.0f, 1.5f};

// ---------------------------------------------------------------------------
// kernels: one 64-thread CTA per example
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(64) mlp_forward_kernel(const float* __restrict__ P, const float* __restrict__ x,
                                                         int B, float* __restrict__ h1, float* __restrict__ h2,
                                                         float* __restrict__ y) {
    __shared__ float s_x[kIn], s_h1[kHid], s_h2[kHid];
    const int b = blockIdx.x, j = threadIdx.x;
    if (b >= B) return;
    if (j < kIn) s_x[j] = x[b * kIn + j];
    __syncthreads();
    float a = P[oB1 + j];
#pragma unroll
    for (int i = 0; i < kIn; ++i) a = fmaf(P[oW1 + j * kIn + i], s_x[i], a);
    a = fmaxf(a, 0.f);
    s_h1[j] = a;
    if (h1) h1[b * kHid + j] = a;
    __syncthreads();
    float c = P[oB2 + j];
    for (int k = 0; k < kHid; ++k) c = fmaf(P[oW2 + j * kHid + k], s_h1[k], c);
    c = fmaxf(c, 0.f);
    s_h2[j] = c;
    if (h2) h2[b * kHid + j] = c;
    __syncthreads();
    if (j < kOut) {
        float o = P[oB3 + j];
        for (int k = 0; k < kHid; ++k) o = fmaf(P[oW3 + j * kHid + k], s_h2[k], o);
        y[b * kOut + j] = o;
    }
}

// Per-example gradient of L = mean over B*4 of (y - t)^2 into G[b][kParams];
// sq[b] = sum of squared errors of example b.
__global__ void __launch_bounds__(64) mlp_backward_kernel(const float* __restrict__ P, const float* __restrict__ x,
                                                          const float* __restrict__ t, const float* __restrict__ h1,
                                                          const float* __restrict__ h2, const float* __restrict__ y,
                                                          int B, float* __restrict__ G, float* __restrict__ sq) {
    __shared__ float s_x[kIn], s_h1[kHid], s_h2[kHid], s_dy[kOut], s_d2[kHid];
    const int b = blockIdx.x, j = threadIdx.x;
    if (b >= B) return;
    float* g = G + (size_t)b * kParams;
    if (j < kIn) s_x[j] = x[b * kIn + j];
    s_h1[j] = h1[b * kHid + j];
    s_h2[j] = h2[b * kHid + j];
    if (j < kOut) {
        const float e = y[b * kOut + j] - t[b * kOut + j];
        s_dy[j] = 2.f * e / (float)(B * kOut);
    }
    __syncthreads();
    if (j == 0) {
        float s = 0.f;
        for (int o = 0; o < kOut; ++o) {
            const float e = y[b * kOut + o] - t[b * kOut + o];
            s += e * e;
        }
        sq[b] = s;
    }
    // layer 3: dW3[o][j] = dy[o] * h2[j], db3 = dy
#pragma unroll
    for (int o = 0; o < kOut; ++o) g[oW3 + o * kHid + j] = s_dy[o] * s_h2[j];
    if (j < kOut) g[oB3 + j] = s_dy[j];
    // dh2[j] = sum_o W3[o][j] dy[o], through the ReLU
    float d2 = 0.f;
#pragma unroll
    for (int o = 0; o < kOut; ++o) d2 = fmaf(P[oW3 + o * kHid + j], s_dy[o], d2);
    d2 = s_h2[j] > 0.f ? d2 : 0.f;
    s_d2[j] = d2;
    __syncthreads();
    // layer 2: dW2[j][k] = d2[j] * h1[k], db2 = d2
    for (int k = 0; k < kHid; ++k) g[oW2 + j * kHid + k] = d2 * s_h1[k];
    g[oB2 + j] = d2;
    // dh1[j] = sum_r W2[r][j] d2[r], through the ReLU
    float d1 = 0.f;
    for (int r = 0; r < kHid; ++r) d1 = fmaf(P[oW2 + r * kHid + j], s_d2[r], d1);
    d1 = s_h1[j] > 0.f ? d1 : 0.f;
#pragma unroll
    for (int i = 0; i < kIn; ++i) g[oW1 + j * kIn + i] = d1 * s_x[i];
    g[oB1 + j] = d1;
}

// grad[p] = sum_b G[b][p] in a fixed order (deterministic); loss = sum sq / (B*4)
__global__ void mlp_reduce_kernel(const float* __restrict__ G, const float* __restrict__ sq, int B,
                                  float* __restrict__ grad, float* __restrict__ loss) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < kParams) {
        float s = 0.f;
        for (int b = 0; b < B; ++b) s += G[(size_t)b * kParams + p];
        grad[p] = s;
    }
    if (p == 0 && loss) {
        float s = 0.f;
        for (int b = 0; b < B; ++b) s += sq[b];
        *loss = s / (float)(B * kOut);
    }
}

// Full-batch Adam (Kingma & Ba 2015, with bias correction), all `steps` updates in one
// launch of one cluster of kTrainCtas CTAs.  A step is two halves with a cluster barrier
// after each:
//   1. examples: CTA c takes the examples c, c + 16, ...; 64 threads per example hold a row
//      of W2 each in registers and run the forward pass and the back-propagated d2, d1, dy,
//      which go to global memory (L2);
//   2. parameters: CTA c owns a 16 x 16 tile of W2 and 4 rows of the small arrays.  Each
//      parameter's gradient is the sum over the examples in order, its moments stay in the
//      thread's registers for the whole call, and the updated weight goes to L2 for everyone.
// The sums run in the order of mlp_forward_kernel, mlp_backward_kernel and
// mlp_reduce_kernel, so a step's weights equal theirs bit for bit.  100 steps on 305
// examples, call and copies included: 3.97 ms as five launches a step (forward, backward, the
// reduction of 305 gradients of 19 KB each, Adam, step counter), 1.42 ms here.  The bound is
// latency: by timing with a half left out, 4.9 us a step for the examples (chains of 64
// dependent FMAs), 5.3 us for the parameters (exchange through L2 and the chain of B
// additions), 0.5 us for a barrier.
//
// Chunk and side-by-side count were chosen at a tuner's training set of 305 examples (one chunk,
// one round of 16 x 8 x 3); larger sets take several of each.  100 steps, five launches a step ->
// here: 1 example 1.66 -> 0.62 ms, 32 2.03 -> 0.70, 385 4.33 -> 1.72, 1000 9.27 -> 3.41, 4096
// 34.8 -> 11.8.  Where a device has no room for the cluster, dr_mlp_train runs the launches.
constexpr int kTrainCtas = 16, kTrainThreads = 512, kTrainSlots = kTrainThreads / kHid;
constexpr int kTrainChunk = 320;  // examples staged at a time in the second half
constexpr int kTrainIlp = 3;      // examples a slot runs side by side (independent FMA chains)
static_assert(kTrainCtas == 16 && kHid == 64 && kIn == 4 && kOut == 4, "tiles of the parameter half");

struct TrainShared {
    float w2[kHid][kHid + 1];  // padded: rows and columns are both read
    float w1[kHid][kIn], b1[kHid], b2[kHid], w3[kOut][kHid], b3[kOut];
    float h1[kTrainSlots][kTrainIlp][kHid], h2[kTrainSlots][kTrainIlp][kHid], d2[kTrainSlots][kTrainIlp][kHid];
    float dy[kTrainSlots][kTrainIlp][kOut];
    // the W2 tile's columns and rows and the small arrays' 4, examples along the rows (a pitch
    // of 4 mod 32 words: 8 rows of 16-byte reads fall on distinct banks)
    float th1[16][kTrainChunk + 4], td2[16][kTrainChunk + 4];
    float sd1[4][kTrainChunk + 4], sd2[4][kTrainChunk + 4], sh2[4][kTrainChunk + 4], sdy[4][kTrainChunk + 4];
    float sx[4][kTrainChunk + 4], one[kTrainChunk + 4];
    float c1, c2;  // bias corrections of the step
};

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ void slot_barrier(int slot) {  // the 64 threads of one example
    asm volatile("bar.sync %0, 64;" ::"r"(1 + slot) : "memory");
}

struct AdamState {
    float p, m, v;
};

__device__ __forceinline__ void adam_step(AdamState& a, float g, float lr, float c1, float c2) {
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    // the roundings of `b1 * m + (1 - b1) * g` and `b2 * v + (1 - b2) * g * g` spelled out
    const float mm = fmaf(1.f - b1, g, __fmul_rn(b1, a.m));
    const float vv = fmaf(__fmul_rn(1.f - b2, g), g, __fmul_rn(b2, a.v));
    a.m = mm;
    a.v = vv;
    const float mh = mm / c1, vh = vv / c2;
    a.p -= lr * mh / (sqrtf(vh) + eps);
}

__global__ void __launch_bounds__(kTrainThreads, 1)
    mlp_train_kernel(float* __restrict__ P, float* __restrict__ gm, float* __restrict__ gv, float* __restrict__ step,
                     const float* __restrict__ x, const float* __restrict__ t, float* __restrict__ gh1,
                     float* __restrict__ gh2, float* __restrict__ gd1, float* __restrict__ gd2,
                     float* __restrict__ gdy, float* __restrict__ sq, float* __restrict__ loss, int B, int steps,
                     float lr) {
    extern __shared__ __align__(16) unsigned char train_smem[];
    TrainShared& S = *reinterpret_cast<TrainShared*>(train_smem);
    const int c = blockIdx.x, tid = threadIdx.x, j = tid & (kHid - 1), slot = tid >> 6;
    // this thread's parameters of the second half: two neighbours of a W2 row (tid < 128), or
    // one of the CTA's 40 (44 in CTA 0) others: W1 rows, b1, b2, W3 columns 4c .. 4c+3, b3
    const int jr = (c >> 2) * 16 + (tid >> 3), kr = (c & 3) * 16 + 2 * (tid & 7);
    const int o = tid - 128;
    int pi = -1;
    if (o >= 0 && o < 16) pi = oW1 + (4 * c + (o >> 2)) * kIn + (o & 3);
    else if (o >= 16 && o < 20) pi = oB1 + 4 * c + (o - 16);
    else if (o >= 20 && o < 24) pi = oB2 + 4 * c + (o - 20);
    else if (o >= 24 && o < 40) pi = oW3 + ((o - 24) >> 2) * kHid + 4 * c + ((o - 24) & 3);
    else if (o >= 40 && o < 44 && c == 0) pi = oB3 + (o - 40);
    AdamState A0 = {0.f, 0.f, 0.f}, A1 = {0.f, 0.f, 0.f};
    const int p0 = tid < 128 ? oW2 + jr * kHid + kr : pi;
    if (p0 >= 0) A0 = {P[p0], gm[p0], gv[p0]};
    if (tid < 128) A1 = {P[p0 + 1], gm[p0 + 1], gv[p0 + 1]};
    float st = *step;
    for (int s = 0; s < steps; ++s) {
        // the weights (written by every CTA in the step before: read past L1), every load in
        // flight before the first is used
        {
            const float4* W2 = reinterpret_cast<const float4*>(P + oW2);
            const float4 wa = __ldcg(W2 + tid), wb = __ldcg(W2 + tid + kTrainThreads);
            float r[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int i = tid + q * kTrainThreads;
                r[q] = i < kParams - kHid * kHid ? __ldcg(P + (i < oW2 ? i : i + kHid * kHid)) : 0.f;
            }
            float* d = &S.w2[tid >> 4][4 * (tid & 15)];
            d[0] = wa.x, d[1] = wa.y, d[2] = wa.z, d[3] = wa.w;
            d = &S.w2[32 + (tid >> 4)][4 * (tid & 15)];
            d[0] = wb.x, d[1] = wb.y, d[2] = wb.z, d[3] = wb.w;
            float* rest = &S.w1[0][0];  // w1, b1, b2, w3, b3 lie one after another, as in P without W2
            if (tid < kParams - kHid * kHid) rest[tid] = r[0];
            if (tid + kTrainThreads < kParams - kHid * kHid) rest[tid + kTrainThreads] = r[1];
        }
        st += 1.f;
        if (tid == 0) S.c1 = 1.f - powf(0.9f, st);
        if (tid == 32) S.c2 = 1.f - powf(0.999f, st);
        __syncthreads();
        float row[kHid];
#pragma unroll
        for (int k = 0; k < kHid; ++k) row[k] = S.w2[j][k];
        const int bstep = kTrainCtas * kTrainSlots;
        for (int bb = c + kTrainCtas * slot; bb < B; bb += kTrainIlp * bstep) {
            float a[kTrainIlp], h[kTrainIlp], d[kTrainIlp];
#pragma unroll
            for (int u = 0; u < kTrainIlp; ++u) {
                const float4 xb = __ldg(reinterpret_cast<const float4*>(x) + min(bb + u * bstep, B - 1));
                a[u] = S.b1[j];
                a[u] = fmaf(S.w1[j][0], xb.x, a[u]);
                a[u] = fmaf(S.w1[j][1], xb.y, a[u]);
                a[u] = fmaf(S.w1[j][2], xb.z, a[u]);
                a[u] = fmaf(S.w1[j][3], xb.w, a[u]);
                a[u] = fmaxf(a[u], 0.f);
                S.h1[slot][u][j] = a[u];
                h[u] = S.b2[j];
            }
            slot_barrier(slot);
#pragma unroll
            for (int k = 0; k < kHid; k += 4)
#pragma unroll
                for (int u = 0; u < kTrainIlp; ++u) {
                    const float4 q = *reinterpret_cast<const float4*>(&S.h1[slot][u][k]);
                    h[u] = fmaf(row[k], q.x, h[u]);
                    h[u] = fmaf(row[k + 1], q.y, h[u]);
                    h[u] = fmaf(row[k + 2], q.z, h[u]);
                    h[u] = fmaf(row[k + 3], q.w, h[u]);
                }
#pragma unroll
            for (int u = 0; u < kTrainIlp; ++u) {
                h[u] = fmaxf(h[u], 0.f);
                S.h2[slot][u][j] = h[u];
            }
            slot_barrier(slot);
            // outputs: one thread per example and output
            if (j < kOut * kTrainIlp) {
                const int u = j >> 2, oo = j & 3;
                const int b = bb + u * bstep;
                float y = S.b3[oo];
#pragma unroll
                for (int k = 0; k < kHid; k += 4) {
                    const float4 q = *reinterpret_cast<const float4*>(&S.h2[slot][u][k]);
                    const float4 w = *reinterpret_cast<const float4*>(&S.w3[oo][k]);
                    y = fmaf(w.x, q.x, y);
                    y = fmaf(w.y, q.y, y);
                    y = fmaf(w.z, q.z, y);
                    y = fmaf(w.w, q.w, y);
                }
                const float e = y - __ldg(t + min(b, B - 1) * kOut + oo);
                const float g = 2.f * e / (float)(B * kOut);
                S.dy[slot][u][oo] = g;
                if (b < B) __stcg(gdy + b * kOut + oo, g);
                if (s == steps - 1) {  // squared errors in output order, as mlp_backward_kernel
                    float q = 0.f;
#pragma unroll
                    for (int i = 0; i < kOut; ++i) {
                        const float ei = __shfl_sync((1u << (kOut * kTrainIlp)) - 1u, e, 4 * u + i);
                        q += ei * ei;
                    }
                    if (oo == 0 && b < B) __stcg(sq + b, q);
                }
            }
            slot_barrier(slot);
#pragma unroll
            for (int u = 0; u < kTrainIlp; ++u) {
                float g = 0.f;
#pragma unroll
                for (int k = 0; k < kOut; ++k) g = fmaf(S.w3[k][j], S.dy[slot][u][k], g);
                g = h[u] > 0.f ? g : 0.f;
                S.d2[slot][u][j] = g;
                d[u] = 0.f;
                const int b = bb + u * bstep;
                if (b < B) {
                    __stcg(gh1 + b * kHid + j, a[u]);
                    __stcg(gh2 + b * kHid + j, h[u]);
                    __stcg(gd2 + b * kHid + j, g);
                }
            }
            slot_barrier(slot);
#pragma unroll
            for (int r = 0; r < kHid; r += 4) {
                const float w0 = S.w2[r][j], w1 = S.w2[r + 1][j], w2 = S.w2[r + 2][j], w3 = S.w2[r + 3][j];
#pragma unroll
                for (int u = 0; u < kTrainIlp; ++u) {
                    const float4 q = *reinterpret_cast<const float4*>(&S.d2[slot][u][r]);
                    d[u] = fmaf(w0, q.x, d[u]);
                    d[u] = fmaf(w1, q.y, d[u]);
                    d[u] = fmaf(w2, q.z, d[u]);
                    d[u] = fmaf(w3, q.w, d[u]);
                }
            }
#pragma unroll
            for (int u = 0; u < kTrainIlp; ++u)
                if (bb + u * bstep < B) __stcg(gd1 + (bb + u * bstep) * kHid + j, a[u] > 0.f ? d[u] : 0.f);
        }
        cluster_barrier();
        // gradients of this thread's parameters, example after example
        float g0 = 0.f, g1 = 0.f;
        for (int b0 = 0; b0 < B; b0 += kTrainChunk) {
            const int n = min(kTrainChunk, B - b0);
            __syncthreads();  // the chunk before has been read
#pragma unroll 3
            for (int i = tid; i < 4 * n; i += kTrainThreads) {
                const int b = i >> 2, q = 4 * (i & 3);
                const size_t at = (size_t)(b0 + b) * kHid;
                const float4 h = __ldcg(reinterpret_cast<const float4*>(gh1 + at + (c & 3) * 16 + q));
                const float4 d = __ldcg(reinterpret_cast<const float4*>(gd2 + at + (c >> 2) * 16 + q));
                S.th1[q][b] = h.x, S.th1[q + 1][b] = h.y, S.th1[q + 2][b] = h.z, S.th1[q + 3][b] = h.w;
                S.td2[q][b] = d.x, S.td2[q + 1][b] = d.y, S.td2[q + 2][b] = d.z, S.td2[q + 3][b] = d.w;
            }
            for (int b = tid; b < n; b += kTrainThreads) {
                const size_t at = (size_t)(b0 + b) * kHid + 4 * c;
                const float4 d1 = __ldcg(reinterpret_cast<const float4*>(gd1 + at));
                const float4 d2 = __ldcg(reinterpret_cast<const float4*>(gd2 + at));
                const float4 h2 = __ldcg(reinterpret_cast<const float4*>(gh2 + at));
                const float4 dy = __ldcg(reinterpret_cast<const float4*>(gdy) + b0 + b);
                const float4 xb = __ldg(reinterpret_cast<const float4*>(x) + b0 + b);
                S.sd1[0][b] = d1.x, S.sd1[1][b] = d1.y, S.sd1[2][b] = d1.z, S.sd1[3][b] = d1.w;
                S.sd2[0][b] = d2.x, S.sd2[1][b] = d2.y, S.sd2[2][b] = d2.z, S.sd2[3][b] = d2.w;
                S.sh2[0][b] = h2.x, S.sh2[1][b] = h2.y, S.sh2[2][b] = h2.z, S.sh2[3][b] = h2.w;
                S.sdy[0][b] = dy.x, S.sdy[1][b] = dy.y, S.sdy[2][b] = dy.z, S.sdy[3][b] = dy.w;
                S.sx[0][b] = xb.x, S.sx[1][b] = xb.y, S.sx[2][b] = xb.z, S.sx[3][b] = xb.w;
                S.one[b] = 1.f;
            }
            __syncthreads();
            // g0 += u * w0 (and g1 += u * w1), one product after another
            if (p0 >= 0) {
                const float *u, *w0, *w1;
                if (tid < 128) u = S.td2[jr & 15], w0 = S.th1[kr & 15], w1 = S.th1[(kr & 15) + 1];
                else {
                    u = o < 16 ? S.sd1[o >> 2] : o < 20 ? S.sd1[o - 16] : o < 24 ? S.sd2[o - 20]
                        : o < 40 ? S.sdy[(o - 24) >> 2] : S.sdy[o - 40];
                    w0 = o < 16 ? S.sx[o & 3] : o >= 24 && o < 40 ? S.sh2[(o - 24) & 3] : S.one;
                    w1 = w0;
                }
                int b = 0;
#pragma unroll 4
                for (; b + 4 <= n; b += 4) {
                    const float4 q = *reinterpret_cast<const float4*>(u + b);
                    const float4 h = *reinterpret_cast<const float4*>(w0 + b);
                    const float4 k = *reinterpret_cast<const float4*>(w1 + b);
                    g0 = __fadd_rn(g0, __fmul_rn(q.x, h.x));
                    g1 = __fadd_rn(g1, __fmul_rn(q.x, k.x));
                    g0 = __fadd_rn(g0, __fmul_rn(q.y, h.y));
                    g1 = __fadd_rn(g1, __fmul_rn(q.y, k.y));
                    g0 = __fadd_rn(g0, __fmul_rn(q.z, h.z));
                    g1 = __fadd_rn(g1, __fmul_rn(q.z, k.z));
                    g0 = __fadd_rn(g0, __fmul_rn(q.w, h.w));
                    g1 = __fadd_rn(g1, __fmul_rn(q.w, k.w));
                }
                for (; b < n; ++b) {
                    g0 = __fadd_rn(g0, __fmul_rn(u[b], w0[b]));
                    g1 = __fadd_rn(g1, __fmul_rn(u[b], w1[b]));
                }
            }
        }
        if (p0 >= 0) {
            adam_step(A0, g0, lr, S.c1, S.c2);
            __stcg(P + p0, A0.p);
        }
        if (tid < 128) {
            adam_step(A1, g1, lr, S.c1, S.c2);
            __stcg(P + p0 + 1, A1.p);
        }
        cluster_barrier();
    }
    if (p0 >= 0) {
        gm[p0] = A0.m;
        gv[p0] = A0.v;
    }
    if (tid < 128) {
        gm[p0 + 1] = A1.m;
        gv[p0 + 1] = A1.v;
    }
    if (c == 0 && tid == 0) {
        *step = st;
        float q = 0.f;
        for (int b = 0; b < B; ++b) q += __ldcg(sq + b);
        *loss = q / (float)(B * kOut);
    }
}

// The same update step by step, after mlp_forward_kernel, mlp_backward_kernel and
// mlp_reduce_kernel: step s of a call (the counter on the device moves when the call ends).
__global__ void mlp_adam_kernel(float* __restrict__ P, const float* __restrict__ grad, float* __restrict__ m,
                                float* __restrict__ v, const float* __restrict__ step, int s, float lr) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= kParams) return;
    const float t = *step + (float)(s + 1);
    AdamState a = {P[p], m[p], v[p]};
    adam_step(a, grad[p], lr, 1.f - powf(0.9f, t), 1.f - powf(0.999f, t));
    P[p] = a.p;
    m[p] = a.m;
    v[p] = a.v;
}

__global__ void mlp_step_advance(float* step, int steps) { *step += (float)steps; }

}  // namespace

struct dr_mlp {
    dr_ctx* ctx = nullptr;
    cudaStream_t stream = nullptr;
    float* P = nullptr;  // device parameters
    float* m = nullptr;
    float* v = nullptr;
    float* grad = nullptr;
    float* step = nullptr;
    float* loss = nullptr;
    float *x = nullptr, *t = nullptr, *h1 = nullptr, *h2 = nullptr, *y = nullptr, *G = nullptr, *sq = nullptr;
    int cap = 0;  // examples the work buffers hold
    int clusters = -1;  // clusters of mlp_train_kernel the device holds at once (-1: not asked yet)
};

namespace {

int mlp_fail(int code, const char* msg) { return record_error(code, msg); }

#define MCU(call)                                                 \
    do {                                                          \
        cudaError_t e_ = (call);                                  \
        if (e_ != cudaSuccess) return mlp_fail(DR_ERR_CUDA, #call); \
    } while (0)

int mlp_reserve(dr_mlp* n, int B) {
    if (B <= n->cap) return DR_OK;
    float** bufs[] = {&n->x, &n->t, &n->h1, &n->h2, &n->y, &n->G, &n->sq};
    for (float** b : bufs)
        if (*b) cudaFree(*b), *b = nullptr;
    const size_t sz[] = {(size_t)B * kIn, (size_t)B * kOut, (size_t)B * kHid, (size_t)B * kHid,
                         (size_t)B * kOut, (size_t)B * kParams, (size_t)B};
    for (int i = 0; i < 7; ++i) MCU(cudaMalloc(bufs[i], sz[i] * sizeof(float)));
    n->cap = B;
    return DR_OK;
}

// Launch configuration of mlp_train_kernel.  False where the device does not hold a cluster of 16
// such CTAs at once (a slice of a GPU, no GPC with 16 free SMs): training then runs step by step.
bool mlp_train_config(dr_mlp* n, cudaLaunchConfig_t* cfg, cudaLaunchAttribute* at) {
    cfg->gridDim = dim3(kTrainCtas);
    cfg->blockDim = dim3(kTrainThreads);
    cfg->dynamicSmemBytes = sizeof(TrainShared);
    cfg->stream = n->stream;
    at->id = cudaLaunchAttributeClusterDimension;
    at->val.clusterDim.x = kTrainCtas;
    at->val.clusterDim.y = at->val.clusterDim.z = 1;
    cfg->attrs = at;
    cfg->numAttrs = 1;
    if (n->clusters < 0) {
        const bool ok = cudaFuncSetAttribute(mlp_train_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)sizeof(TrainShared)) == cudaSuccess &&
                        cudaFuncSetAttribute(mlp_train_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
                            cudaSuccess &&
                        cudaOccupancyMaxActiveClusters(&n->clusters, mlp_train_kernel, cfg) == cudaSuccess;
        if (!ok) {
            n->clusters = 0;
            cudaGetLastError();
        }
    }
    return n->clusters > 0;
}

// Training domain of the shipped network: X in [10^10, 10^16], budgets of
// 8..160 GiB.  Inputs outside it are clamped to its boundary: the outputs are
// already relative to the (X / ln ln X)^(2/3) law (fx, cx), so a proposal
// carried to a larger X keeps the scale-free part the network learned instead
// of extrapolating a ReLU network linearly.
constexpr double kLog10XMin = 10.0, kLog10XMax = 16.0, kLog2BudgetMin = 33.0, kLog2BudgetMax = 37.33;

void features(int64_t X, uint64_t budget, int sms, int batch, float out[kIn]) {
    const double lx = std::min(kLog10XMax, std::max(kLog10XMin, std::log10((double)std::max<int64_t>(X, 2))));
    const double lb = std::min(kLog2BudgetMax, std::max(kLog2BudgetMin, std::log2((double)std::max<uint64_t>(budget, 1))));
    const float raw[kIn] = {(float)lx, (float)lb, (float)sms, (float)std::log2((double)std::max(batch, 1))};
    for (int i = 0; i < kIn; ++i) out[i] = (raw[i] - kInMean[i]) / kInScale[i];
}

}  // namespace

// Host-side map from network outputs to engine parameters (exported for tests
// through dr_tuner_params).
static void outputs_to_params(int64_t X, const float yn[kOut], dr_params* p) {
    float o[kOut];
    for (int i = 0; i < kOut; ++i) o[i] = yn[i] * kOutScale[i] + kOutMean[i];
    const double cx = std::min(4.0, std::max(0.3, (double)o[0]));
    const double fx = std::exp2(std::min(4.0, std::max(-4.0, (double)o[1])));
    // the cap is an absolute size learned inside the training domain; for an X
    // outside it (whose features were clamped) it is carried along the same
    // X^(2/3) law as the rest of the proposal
    const double lx = std::log10((double)std::max<int64_t>(X, 2));
    const double lxc = std::min(kLog10XMax, std::max(kLog10XMin, lx));
    const double cap = std::exp2(std::min(41.0, std::max(20.0, (double)o[2]))) * std::pow(10.0, (2.0 / 3.0) * (lx - lxc));
    int seg = (int)std::lround(o[3]);
    seg = std::max(12, std::min(seg, 18));
    params_clear(p);
    const double loglogX = std::log(std::max(2.0, std::log((double)X)));
    int64_t u = (int64_t)std::min(cap, fx * std::pow((double)X / loglogX, 2.0 / 3.0));
    const int64_t S = isqrt_i64(X);
    const int64_t endpoint = (int64_t)(cx * std::sqrt((double)X)) + 1000;
    u = std::max(u, std::max(S + 1000, endpoint));
    u = ((u + 255) / 256) * 256;
    const int64_t e256 = (endpoint + 255) & ~255LL;
    p->u_total = u;
    // dense int16 tier as in the B200 policy: max(1.28e8, u/16) values, at most 4e9
    const int64_t dense_target = std::min<int64_t>(4000000000LL, std::max<int64_t>(128000000LL, u / 16));
    p->u_dense = std::min<int64_t>(u, std::max<int64_t>(e256, (dense_target + 255) & ~255LL));
    p->cx = cx;
    p->mu_limit = std::min(u, std::max(endpoint, X / u + 1000));
    p->segment_log2 = seg;
}

extern "C" {

int dr_mlp_create(dr_ctx* ctx, uint64_t seed, dr_mlp** out) {
    if (!out) return mlp_fail(DR_ERR_ARG, "out is NULL");
    *out = nullptr;
    dr_mlp* n = new dr_mlp();
    n->ctx = ctx;
    if (cudaStreamCreateWithFlags(&n->stream, cudaStreamNonBlocking) != cudaSuccess) {
        delete n;
        return mlp_fail(DR_ERR_CUDA, "cudaStreamCreate failed");
    }
    float** bufs[] = {&n->P, &n->m, &n->v, &n->grad};
    for (float** b : bufs)
        if (cudaMalloc(b, kParams * sizeof(float)) != cudaSuccess) {
            dr_mlp_destroy(n);
            return mlp_fail(DR_ERR_NOMEM, "cudaMalloc failed");
        }
    if (cudaMalloc(&n->step, 2 * sizeof(float)) != cudaSuccess) {
        dr_mlp_destroy(n);
        return mlp_fail(DR_ERR_NOMEM, "cudaMalloc failed");
    }
    n->loss = n->step + 1;
    // He-uniform initialisation from a 64-bit LCG (host), biases zero
    std::vector<float> w(kParams, 0.f);
    uint64_t s = seed * 6364136223846793005ULL + 1442695040888963407ULL;
    auto uni = [&]() {
        s = s * 6364136223846793005ULL + 1442695040888963407ULL;
        return (float)((double)(s >> 11) * (1.0 / 9007199254740992.0)) * 2.f - 1.f;
    };
    const float a1 = std::sqrt(6.f / kIn), a2 = std::sqrt(6.f / kHid), a3 = std::sqrt(6.f / kHid) * 0.1f;
    for (int i = 0; i < kHid * kIn; ++i) w[oW1 + i] = a1 * uni();
    for (int i = 0; i < kHid * kHid; ++i) w[oW2 + i] = a2 * uni();
    for (int i = 0; i < kOut * kHid; ++i) w[oW3 + i] = a3 * uni();
    int rc = dr_mlp_set_weights(n, w.data(), kParams);
    if (rc) {
        dr_mlp_destroy(n);
        return rc;
    }
    *out = n;
    return DR_OK;
}

int dr_mlp_destroy(dr_mlp* n) {
    if (!n) return DR_OK;
    float* bufs[] = {n->P, n->m, n->v, n->grad, n->step, n->x, n->t, n->h1, n->h2, n->y, n->G, n->sq};
    for (float* b : bufs)
        if (b) cudaFree(b);
    if (n->stream) cudaStreamDestroy(n->stream);
    delete n;
    return DR_OK;
}

int64_t dr_mlp_num_params(void) { return kParams; }

int dr_mlp_set_weights(dr_mlp* n, const float* w, int64_t count) {
    if (!n || !w || count != kParams) return mlp_fail(DR_ERR_ARG, "dr_mlp_set_weights: need 4740 floats");
    MCU(cudaMemcpy(n->P, w, kParams * sizeof(float), cudaMemcpyHostToDevice));
    MCU(cudaMemset(n->m, 0, kParams * sizeof(float)));
    MCU(cudaMemset(n->v, 0, kParams * sizeof(float)));
    MCU(cudaMemset(n->step, 0, 2 * sizeof(float)));
    return DR_OK;
}

int dr_mlp_get_weights(dr_mlp* n, float* w, int64_t count) {
    if (!n || !w || count != kParams) return mlp_fail(DR_ERR_ARG, "dr_mlp_get_weights: need 4740 floats");
    MCU(cudaMemcpy(w, n->P, kParams * sizeof(float), cudaMemcpyDeviceToHost));
    return DR_OK;
}

// y = f(x) for B normalised feature rows (host arrays B x 4 -> B x 4).
int dr_mlp_forward(dr_mlp* n, const float* x, int64_t B, float* y) {
    if (!n || !x || !y || B < 1 || B > kMaxBatch) return mlp_fail(DR_ERR_ARG, "dr_mlp_forward: bad argument");
    int rc = mlp_reserve(n, (int)B);
    if (rc) return rc;
    MCU(cudaMemcpyAsync(n->x, x, B * kIn * sizeof(float), cudaMemcpyHostToDevice, n->stream));
    mlp_forward_kernel<<<(unsigned)B, 64, 0, n->stream>>>(n->P, n->x, (int)B, nullptr, nullptr, n->y);
    MCU(cudaGetLastError());
    MCU(cudaMemcpyAsync(y, n->y, B * kOut * sizeof(float), cudaMemcpyDeviceToHost, n->stream));
    MCU(cudaStreamSynchronize(n->stream));
    return DR_OK;
}

// Gradient of the mean squared error over B examples (host arrays), no update.
int dr_mlp_grad(dr_mlp* n, const float* x, const float* t, int64_t B, float* grad, float* loss) {
    if (!n || !x || !t || !grad || B < 1 || B > kMaxBatch) return mlp_fail(DR_ERR_ARG, "dr_mlp_grad: bad argument");
    int rc = mlp_reserve(n, (int)B);
    if (rc) return rc;
    MCU(cudaMemcpyAsync(n->x, x, B * kIn * sizeof(float), cudaMemcpyHostToDevice, n->stream));
    MCU(cudaMemcpyAsync(n->t, t, B * kOut * sizeof(float), cudaMemcpyHostToDevice, n->stream));
    mlp_forward_kernel<<<(unsigned)B, 64, 0, n->stream>>>(n->P, n->x, (int)B, n->h1, n->h2, n->y);
    mlp_backward_kernel<<<(unsigned)B, 64, 0, n->stream>>>(n->P, n->x, n->t, n->h1, n->h2, n->y, (int)B, n->G, n->sq);
    mlp_reduce_kernel<<<(kParams + 255) / 256, 256, 0, n->stream>>>(n->G, n->sq, (int)B, n->grad, n->loss);
    MCU(cudaGetLastError());
    MCU(cudaMemcpyAsync(grad, n->grad, kParams * sizeof(float), cudaMemcpyDeviceToHost, n->stream));
    float l = 0.f;
    MCU(cudaMemcpyAsync(&l, n->loss, sizeof(float), cudaMemcpyDeviceToHost, n->stream));
    MCU(cudaStreamSynchronize(n->stream));
    if (loss) *loss = l;
    return DR_OK;
}

}  // extern "C"

// Full-batch Adam: `steps` updates on the B examples, in one cluster launch or step by step.
static int mlp_train(dr_mlp* n, const float* x, const float* t, int64_t B, int steps, float lr, float* final_loss,
                     bool one_launch) {
    if (!n || !x || !t || B < 1 || B > kMaxBatch || steps < 0) return mlp_fail(DR_ERR_ARG, "dr_mlp_train: bad argument");
    int rc = mlp_reserve(n, (int)B);
    if (rc) return rc;
    MCU(cudaMemcpyAsync(n->x, x, B * kIn * sizeof(float), cudaMemcpyHostToDevice, n->stream));
    MCU(cudaMemcpyAsync(n->t, t, B * kOut * sizeof(float), cudaMemcpyHostToDevice, n->stream));
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    if (steps > 0 && one_launch) one_launch = mlp_train_config(n, &cfg, at);
    if (steps > 0 && !one_launch) {
        for (int s = 0; s < steps; ++s) {
            mlp_forward_kernel<<<(unsigned)B, 64, 0, n->stream>>>(n->P, n->x, (int)B, n->h1, n->h2, n->y);
            mlp_backward_kernel<<<(unsigned)B, 64, 0, n->stream>>>(n->P, n->x, n->t, n->h1, n->h2, n->y, (int)B, n->G,
                                                                    n->sq);
            mlp_reduce_kernel<<<(kParams + 255) / 256, 256, 0, n->stream>>>(n->G, n->sq, (int)B, n->grad, n->loss);
            mlp_adam_kernel<<<(kParams + 255) / 256, 256, 0, n->stream>>>(n->P, n->grad, n->m, n->v, n->step, s, lr);
        }
        mlp_step_advance<<<1, 1, 0, n->stream>>>(n->step, steps);
        MCU(cudaGetLastError());
    }
    if (steps > 0 && one_launch) {
        // the per-example gradients' buffer (B x kParams) holds d1, d2 and dy here
        float *d1 = n->G, *d2 = n->G + (size_t)B * kHid, *dy = n->G + 2 * (size_t)B * kHid;
        MCU(cudaLaunchKernelEx(&cfg, mlp_train_kernel, n->P, n->m, n->v, n->step, (const float*)n->x,
                               (const float*)n->t, n->h1, n->h2, d1, d2, dy, n->sq, n->loss, (int)B, steps, lr));
    }
    float l = 0.f;
    MCU(cudaMemcpyAsync(&l, n->loss, sizeof(float), cudaMemcpyDeviceToHost, n->stream));
    MCU(cudaStreamSynchronize(n->stream));
    if (final_loss) *final_loss = l;
    return DR_OK;
}

extern "C" {

int dr_mlp_train(dr_mlp* n, const float* x, const float* t, int64_t B, int steps, float lr, float* final_loss) {
    return mlp_train(n, x, t, B, steps, lr, final_loss, true);
}

int dr_debug_mlp_train_steps(dr_mlp* n, const float* x, const float* t, int64_t B, int steps, float lr,
                             float* final_loss) {
    return mlp_train(n, x, t, B, steps, lr, final_loss, false);
}

// Engine parameters for X from the network's outputs (no check, no fallback).
int dr_tuner_params(int64_t X, const float* y_normalised, dr_params* out) {
    if (!y_normalised || !out || X < 1) return mlp_fail(DR_ERR_ARG, "dr_tuner_params: bad argument");
    outputs_to_params(X, y_normalised, out);
    return DR_OK;
}

// Normalised features of one query (the network's input row).
int dr_tuner_features(int64_t X, uint64_t hbm_budget, int sm_count, int batch, float* out4) {
    if (!out4) return mlp_fail(DR_ERR_ARG, "dr_tuner_features: out is NULL");
    features(X, hbm_budget, sm_count, batch, out4);
    return DR_OK;
}

// Shrink u (keeping cx, the dense tier and the endpoints) until the query's
// device footprint fits 90% of the budget: the budget is a hard constraint of
// the proposal, not a reason to discard it.
static void project_to_budget(int64_t X, uint64_t budget, dr_params* p) {
    if (!budget) return;
    for (int it = 0; it < 64 && dr_query_bytes(X, p) > budget / 10 * 9; ++it) {
        const int64_t S = isqrt_i64(X);
        const int64_t endpoint = (int64_t)(p->cx * std::sqrt((double)X)) + 1000;
        const int64_t floor_u = std::max(S + 1000, std::max(endpoint, p->u_dense));
        int64_t u = std::max(floor_u, (int64_t)((double)p->u_total * 0.9));
        u = ((u + 255) / 256) * 256;
        if (u >= p->u_total) break;
        p->u_total = u;
        p->mu_limit = std::min(u, std::max(endpoint, X / u + 1000));
    }
}

// The learned tuner's proposal for X: network inference on the device, mapped
// to parameters and projected onto the device budget, then the endpoint-
// coverage check; a proposal that fails it is replaced by the reference's
// default heuristic (*fallback = 1).
int dr_tuner_propose(dr_mlp* n, int64_t X, uint64_t hbm_budget, int sm_count, int batch, dr_params* out,
                     int* fallback) {
    if (!n || !out) return mlp_fail(DR_ERR_ARG, "dr_tuner_propose: bad argument");
    float f[kIn], y[kOut];
    features(X, hbm_budget, sm_count, batch, f);
    int rc = dr_mlp_forward(n, f, 1, y);
    if (rc) return rc;
    outputs_to_params(X, y, out);
    if (X > 0) project_to_budget(X, hbm_budget, out);
    int fb = 0;
    if (X < 1 || dr_check_params(X, out, hbm_budget) != DR_OK) {
        fb = 1;
        rc = dr_default_params(X, DR_POLICY_REFERENCE, out);
        if (rc) return rc;
    }
    if (fallback) *fallback = fb;
    return DR_OK;
}

}  // extern "C"
