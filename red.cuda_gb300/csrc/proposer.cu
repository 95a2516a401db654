// proposer.cu -- learned step-size proposals for the adaptive integrators.
//
// After every accepted step, a per-system feature vector is formed on the
// device from the new state.  A small MLP (12 -> 64 -> 64 -> 1, SiLU, BF16
// weights, FP32 accumulation) maps the normalised features to the log of the
// next step size.  The embedded error estimate still judges every try: a
// rejected proposal is retried with the classical controller's step, so only
// the number of rejected tries can change, never the accuracy test.
//
// Training runs on the GPU with the kernels below: a forward / backward pass
// over 16-row tiles writing per-CTA gradients, a fixed-order reduction of the
// CTAs (deterministic), and Adam on FP32 master weights that refreshes the
// BF16 copy used by inference.  The network is far too small for tensor cores
// to pay (a 16 x 64 x 64 tile per CTA): the kernels are latency-bound FMA code.
//
// Features (per system, from the accepted state; FP32 from the truncated FP64
// state -- they steer the step size only):
//   0 log|dt| of the accepted step      6 mean e      9 mean i
//   1 log(err / tol) of that step       7 rms e      10 rms i
//   2 log min over protoplanet-body pairs of distance / Hill radius
//   3 log max |a|                       8 max e      11 max i
//   4 max |v| / v_kep                   (e, i: osculating heliocentric elements
//   5 log N (active bodies)              of the active non-star bodies)
#include <cuda_bf16.h>
#include <algorithm>
#include <cfloat>
#include <cstdio>
#include <cstring>
#include <mutex>

#include "common.cuh"
#include "proposer.cuh"
#include "redgb.h"

namespace redgb {

// FP64 -> FP32 by truncation of the bits (no FP64 instruction; within 1 ulp of
// FP32 of the rounded conversion).  Zero, denormals and values outside FP32's
// range are clamped.
__device__ __forceinline__ float d2f_trunc(double x)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const int e = (int)((b >> 52) & 0x7FF) - 1023 + 127;
    const unsigned sign = (unsigned)(b >> 32) & 0x80000000u;
    if (e <= 0) return __uint_as_float(sign);
    if (e >= 255) return __uint_as_float(sign | 0x7F7FFFFFu);
    return __uint_as_float(sign | ((unsigned)e << 23) | (unsigned)((b >> 29) & 0x7FFFFFu));
}

__device__ __forceinline__ float silu(float z) { return z / (1.0f + expf(-z)); }
__device__ __forceinline__ float silu_grad(float z)
{
    const float s = 1.0f / (1.0f + expf(-z));
    return s * (1.0f + z * (1.0f - s));
}
__device__ __forceinline__ float bf(const __nv_bfloat16* w, int i) { return __bfloat162float(w[i]); }

// partial q is combined by max (3, 6, 7, 8), min (9) or sum (the rest)
__device__ __forceinline__ float combine_part(int q, float a, float b)
{
    return (q == 3 || q == 6 || q == 7 || q == 8) ? fmaxf(a, b) : (q == 9 ? fminf(a, b) : a + b);
}

// ---------------------------------------------------------------------------
// features: per-segment partial sums, then per system in a fixed order
// ---------------------------------------------------------------------------
constexpr int kMaxHill = 64;   // protoplanet-class bodies tested for the Hill-radius feature

__global__ void __launch_bounds__(kSegment) k_feat_seg(const FeatParams P)
{
    __shared__ float hx[kMaxHill], hy[kMaxHill], hz[kMaxHill], hr[kMaxHill];
    __shared__ float red[kNPart][kSegment / 32];
    pdl_wait();
    pdl_trigger();
    const Segment sg = P.segs[blockIdx.x];
    const DevSys& S = P.sys[sg.sys];
    if (!S.accepted) return;   // uniform
    const SysInfo si = P.sinfo[sg.sys];
    const float mstar = si.n_star > 0 ? d2f_trunc(P.mass[si.off]) : 0.f;
    // the protoplanet-class bodies (SI bodies after the stars) and their Hill radii
    const int nh = min(kMaxHill, si.n_SI - si.n_star);
    for (int k = threadIdx.x; k < nh; k += blockDim.x) {
        const int i = si.off + si.n_star + k;
        const float4 p = P.pos[i];
        hx[k] = p.x;
        hy[k] = p.y;
        hz[k] = p.z;
        const float rr = sqrtf(p.x * p.x + p.y * p.y + p.z * p.z);
        const float m = P.id[i] >= 0 ? d2f_trunc(P.mass[i]) : 0.f;
        hr[k] = (m > 0.f && mstar > 0.f) ? rr * cbrtf(m / (3.0f * mstar)) : 0.f;
    }
    __syncthreads();
    float part[kNPart];
#pragma unroll
    for (int q = 0; q < kNPart; q++) part[q] = q == 9 ? FLT_MAX : 0.f;
    const int j = sg.b0 + threadIdx.x;
    if (j < sg.b1 && j >= si.off + si.n_star && P.id[j] >= 0) {
        const float4 p = P.pos[j];
        const float vx = d2f_trunc(P.y_v[3 * j]), vy = d2f_trunc(P.y_v[3 * j + 1]), vz = d2f_trunc(P.y_v[3 * j + 2]);
        const float ax = d2f_trunc(P.acc[3 * j]), ay = d2f_trunc(P.acc[3 * j + 1]), az = d2f_trunc(P.acc[3 * j + 2]);
        const float mu = mstar + d2f_trunc(P.mass[j]);
        const float r = sqrtf(p.x * p.x + p.y * p.y + p.z * p.z);
        const float v2 = vx * vx + vy * vy + vz * vz;
        // angular momentum h = r x v, eccentricity vector (v x h) / mu - r / |r|
        const float hxv = p.y * vz - p.z * vy, hyv = p.z * vx - p.x * vz, hzv = p.x * vy - p.y * vx;
        const float h = sqrtf(hxv * hxv + hyv * hyv + hzv * hzv);
        float e = 0.f, inc = 0.f, vr = 0.f;
        if (mu > 0.f && r > 0.f) {
            const float ex = (vy * hzv - vz * hyv) / mu - p.x / r;
            const float ey = (vz * hxv - vx * hzv) / mu - p.y / r;
            const float ez = (vx * hyv - vy * hxv) / mu - p.z / r;
            e = sqrtf(ex * ex + ey * ey + ez * ez);
            inc = h > 0.f ? acosf(fminf(1.f, fmaxf(-1.f, hzv / h))) : 0.f;
            vr = sqrtf(v2 * r / mu);
        }
        part[0] = 1.f;
        part[1] = e;
        part[2] = e * e;
        part[3] = e;
        part[4] = inc;
        part[5] = inc * inc;
        part[6] = inc;
        part[7] = vr;
        part[8] = sqrtf(ax * ax + ay * ay + az * az);
        const int self = j - (si.off + si.n_star);
        for (int k = 0; k < nh; k++) {
            if (k == self || !(hr[k] > 0.f)) continue;
            const float dx = p.x - hx[k], dy = p.y - hy[k], dz = p.z - hz[k];
            part[9] = fminf(part[9], sqrtf(dx * dx + dy * dy + dz * dz) / hr[k]);
        }
    }
    // block reduction in a fixed order: warp trees, then one thread per partial over the warps
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < kNPart; q++) {
        float v = part[q];
        for (int o = 16; o > 0; o >>= 1) v = combine_part(q, v, __shfl_xor_sync(0xffffffffu, v, o));
        if (lane == 0) red[q][w] = v;
    }
    __syncthreads();
    if (threadIdx.x < kNPart) {
        const int q = threadIdx.x;
        float v = red[q][0];
        for (int k = 1; k < (int)(blockDim.x >> 5); k++) v = combine_part(q, v, red[q][k]);
        P.part[(size_t)blockIdx.x * kNPart + q] = v;
    }
}

// ---------------------------------------------------------------------------
// the MLP on one warp: hidden units lane and lane + 32 of both layers
// ---------------------------------------------------------------------------
__device__ __forceinline__ float mlp_warp(const __nv_bfloat16* w, const float (&xn)[kFeat], int lane)
{
    float h1[2], h2[2];
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const int u = lane + 32 * q;
        float z = bf(w, oB1 + u);
#pragma unroll
        for (int c = 0; c < kFeat; c++) z = fmaf(bf(w, oW1 + u * kFeat + c), xn[c], z);
        h1[q] = silu(z);
    }
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const int u = lane + 32 * q;
        float z = bf(w, oB2 + u);
#pragma unroll
        for (int k = 0; k < kHid; k++) z = fmaf(bf(w, oW2 + u * kHid + k), __shfl_sync(0xffffffffu, h1[k >> 5], k & 31), z);
        h2[q] = silu(z);
    }
    float y = fmaf(bf(w, oW3 + lane), h2[0], bf(w, oW3 + lane + 32) * h2[1]);
    for (int o = 16; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
    return y + bf(w, oB3);
}

__device__ __forceinline__ void normalise(const MlpNorm& nm, const float (&f)[kFeat], float (&xn)[kFeat])
{
#pragma unroll
    for (int c = 0; c < kFeat; c++) xn[c] = (f[c] - nm.x_mean[c]) / nm.x_std[c];
}

// One warp per system that accepted its try: the features from the segment
// partials (fixed order), the log record, the proposal.
__global__ void k_propose(const ProposeParams P)
{
    pdl_wait();
    pdl_trigger();
    const int lane = threadIdx.x & 31;
    const int s = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (s >= P.n_sys) return;
    DevSys& S = P.sys[s];
    if (!S.accepted) return;   // uniform over the warp
    float part[kNPart];
#pragma unroll
    for (int q = 0; q < kNPart; q++) part[q] = q == 9 ? FLT_MAX : 0.f;
    for (int k = lane; k < P.nseg[s]; k += 32) {
        const float* p = P.part + (size_t)(P.seg0[s] + k) * kNPart;
#pragma unroll
        for (int q = 0; q < kNPart; q++) part[q] = combine_part(q, part[q], p[q]);
    }
#pragma unroll
    for (int q = 0; q < kNPart; q++)
        for (int o = 16; o > 0; o >>= 1) part[q] = combine_part(q, part[q], __shfl_xor_sync(0xffffffffu, part[q], o));
    const double dt_did = S.dt_did;
    const float cnt = fmaxf(part[0], 1.f);
    float f[kFeat];
    f[0] = logf(fmaxf(d2f_trunc(fabs(dt_did)), 1e-30f));
    f[1] = logf(fmaxf(d2f_trunc(S.err_last / P.tolerance), 1e-30f));
    f[2] = part[9] < FLT_MAX ? logf(fmaxf(part[9], 1e-30f)) : 0.f;
    f[3] = logf(fmaxf(part[8], 1e-30f));
    f[4] = part[7];
    f[5] = logf(cnt);
    f[6] = part[1] / cnt;
    f[7] = sqrtf(part[2] / cnt);
    f[8] = part[3];
    f[9] = part[4] / cnt;
    f[10] = sqrtf(part[5] / cnt);
    f[11] = part[6];
    if (P.log && lane == 0) {
        if (P.has_prev[s]) {
            const unsigned k = atomicAdd(P.log_n, 1u);
            if (k < P.log_cap) {
                float* r = P.log_buf + (size_t)k * kLogRec;
                for (int c = 0; c < kFeat; c++) r[c] = P.feat_prev[s * kFeat + c];
                r[kFeat] = f[0];       // log|dt| of the step accepted after those features
                r[kFeat + 1] = f[1];   // log(err / tol) of that step
            }
        }
        for (int c = 0; c < kFeat; c++) P.feat_prev[s * kFeat + c] = f[c];
        P.has_prev[s] = 1;
    }
    if (!P.propose) return;
    float xn[kFeat];
    normalise(P.norm, f, xn);
    const float y = mlp_warp(P.w, xn, lane);
    if (lane != 0) return;
    const double log_dt = (double)y * P.norm.y_std + P.norm.y_mean;
    const double mag = fabs(dt_did);
    double ratio = exp(log_dt) * P.safety / mag;
    ratio = fmin(fmax(ratio, P.ratio_lo), P.ratio_hi);
    if (!(ratio == ratio)) return;   // keep the classical step
    double dt = (dt_did < 0.0 ? -mag : mag) * ratio;
    if (P.output_interval != 0.0 && fabs(P.output_interval) < fabs(dt))
        dt = 0.0 < dt ? fabs(P.output_interval) : -fabs(P.output_interval);
    S.dt_next = dt;
    S.dt_try = dt;
}

// Inference on rows of raw features (warp per row): out = predicted log|dt|.
__global__ void k_mlp_rows(const __nv_bfloat16* w, const MlpNorm nm, const float* x, float* out, int n)
{
    const int lane = threadIdx.x & 31;
    const int r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (r >= n) return;
    float f[kFeat], xn[kFeat];
#pragma unroll
    for (int c = 0; c < kFeat; c++) f[c] = x[(size_t)r * kFeat + c];
    normalise(nm, f, xn);
    const float y = mlp_warp(w, xn, lane);
    if (lane == 0) out[r] = y * nm.y_std + nm.y_mean;
}

// ---------------------------------------------------------------------------
// training: loss = sum over rows of (y - t)^2 / (2 n), normalised inputs and
// targets.  A CTA takes tiles of kTrainRows rows (tile b, b + grid, ...) and
// keeps its gradient in registers over them; it writes the gradient (kNParam
// floats) and loss once, and k_mlp_sum adds the CTAs in a fixed order.
//
// Bound by latency: 16 rows are a chain of seven small products between
// barriers.  256 threads split each product by unit (t % 64) and by four rows
// (or 16 of the other index) per group t / 64; activations lie unit-major with
// rows of kRS floats, so that a warp reads its own units conflict-free as
// float4 and the other operand as one broadcast, and W2 has an odd row stride
// for its two uses.  One thread per unit over all 16 rows, with W2 read in a
// 32-way bank conflict, and a sum of one thread per parameter over all CTAs took
// 36.2 us per training step (gradient and Adam) of 2048 rows; this takes 17.2 us.
// ---------------------------------------------------------------------------
constexpr int kTrainThreads = 4 * kHid;
constexpr int kRS = kTrainRows + 4;     // row stride of the activations, floats
constexpr int kW2S = kHid + 1;          // row stride of W2 transposed
static_assert(kTrainRows == 16, "four groups of four rows");

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void fma4(float4& a, float w, float4 v)
{
    a.x = fmaf(w, v.x, a.x);
    a.y = fmaf(w, v.y, a.y);
    a.z = fmaf(w, v.z, a.z);
    a.w = fmaf(w, v.w, a.w);
}
__device__ __forceinline__ float dot4(float4 a, float4 b, float c)
{
    return fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, fmaf(a.w, b.w, c))));
}
__device__ __forceinline__ float4 map4(float4 v, float (*f)(float))
{
    return make_float4(f(v.x), f(v.y), f(v.z), f(v.w));
}

__global__ void __launch_bounds__(kTrainThreads) k_mlp_train(const __nv_bfloat16* w, const float* xn, const float* tn,
                                                            int n, float* part)
{
    constexpr int R = kTrainRows;
    __shared__ float W1[kFeat * kHid], W2[kHid * kW2S], w3[kHid];   // W1 and W2 transposed: [input][unit]
    __shared__ __align__(16) float x[kFeat * kRS], h1[kHid * kRS], h2[kHid * kRS], dz2[kHid * kRS], dz1[kHid * kRS];
    __shared__ __align__(16) float ye[R], dy[R];
    pdl_wait();
    pdl_trigger();
    const int t = threadIdx.x, u = t % kHid, g = t / kHid;
    const int lane = t & 31, wp = t >> 5;
    for (int k = t; k < kHid * kFeat; k += kTrainThreads) W1[(k % kFeat) * kHid + k / kFeat] = bf(w, oW1 + k);
    for (int k = t; k < kHid * kHid; k += kTrainThreads) W2[(k % kHid) * kW2S + k / kHid] = bf(w, oW2 + k);
    if (t < kHid) w3[t] = bf(w, oW3 + t);
    const float b1 = bf(w, oB1 + u), b2 = bf(w, oB2 + u), b3 = bf(w, oB3);
    float gw2[16], gw1[3] = {0.f, 0.f, 0.f}, gb = 0.f, gout = 0.f;
#pragma unroll
    for (int q = 0; q < 16; q++) gw2[q] = 0.f;
    const int tiles = (n + R - 1) / R;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int r0 = tile * R;
        __syncthreads();   // the previous tile's activations are read
        if (t < R * kFeat) {
            const int r = t / kFeat, c = t % kFeat;
            x[c * kRS + r] = r0 + r < n ? xn[(size_t)r0 * kFeat + t] : 0.f;
        }
        __syncthreads();
        // forward: unit u, rows 4 g .. 4 g + 3
        float4 z1 = make_float4(b1, b1, b1, b1), z2 = make_float4(b2, b2, b2, b2);
#pragma unroll
        for (int c = 0; c < kFeat; c++) fma4(z1, W1[c * kHid + u], ld4(x + c * kRS + 4 * g));
        st4(h1 + u * kRS + 4 * g, map4(z1, silu));
        __syncthreads();
#pragma unroll 16
        for (int k = 0; k < kHid; k++) fma4(z2, W2[k * kW2S + u], ld4(h1 + k * kRS + 4 * g));
        st4(h2 + u * kRS + 4 * g, map4(z2, silu));
        __syncthreads();
        // output: warp wp takes rows wp and wp + 8
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int r = wp + 8 * q;
            float y = fmaf(w3[lane], h2[lane * kRS + r], w3[lane + 32] * h2[(lane + 32) * kRS + r]);
            for (int o = 16; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
            if (lane == 0) {
                const float e = r0 + r < n ? y + b3 - tn[r0 + r] : 0.f;
                ye[r] = e;
                dy[r] = e / (float)n;
            }
        }
        __syncthreads();
        const float4 d4 = ld4(dy + 4 * g);
        const float4 s2 = map4(z2, silu_grad);
        st4(dz2 + u * kRS + 4 * g, make_float4(d4.x * w3[u] * s2.x, d4.y * w3[u] * s2.y, d4.z * w3[u] * s2.z,
                                               d4.w * w3[u] * s2.w));
        __syncthreads();
        // hidden layer 2: column u (input unit) of W2's rows 16 g .. 16 g + 15
        const float4 a0 = ld4(h1 + u * kRS), a1 = ld4(h1 + u * kRS + 4), a2 = ld4(h1 + u * kRS + 8),
                     a3 = ld4(h1 + u * kRS + 12);
#pragma unroll
        for (int q = 0; q < 16; q++) {
            const float* d = dz2 + (16 * g + q) * kRS;
            gw2[q] = dot4(ld4(d), a0, dot4(ld4(d + 4), a1, dot4(ld4(d + 8), a2, dot4(ld4(d + 12), a3, gw2[q]))));
        }
        // hidden layer 1: unit u, rows 4 g .. 4 g + 3
        float4 dh = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 16
        for (int k = 0; k < kHid; k++) fma4(dh, W2[u * kW2S + k], ld4(dz2 + k * kRS + 4 * g));
        const float4 s1 = map4(z1, silu_grad);
        st4(dz1 + u * kRS + 4 * g, make_float4(dh.x * s1.x, dh.y * s1.y, dh.z * s1.z, dh.w * s1.w));
        __syncthreads();
        // W1[u][3 g .. 3 g + 2]; the biases and the output layer by one group each
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const float4 d = ld4(dz1 + u * kRS + 4 * q);
#pragma unroll
            for (int c = 0; c < 3; c++) gw1[c] = dot4(d, ld4(x + (3 * g + c) * kRS + 4 * q), gw1[c]);
            if (g == 0) gb += d.x + d.y + d.z + d.w;
            if (g == 1) {
                const float4 e = ld4(dz2 + u * kRS + 4 * q);
                gb += e.x + e.y + e.z + e.w;
            }
            if (g == 2) gb = dot4(ld4(dy + 4 * q), ld4(h2 + u * kRS + 4 * q), gb);
        }
        if (g == 3 && u == 0)
            for (int r = 0; r < R; r++) gout += dy[r];
        if (g == 3 && u == 32)
            for (int r = 0; r < R; r++) gout += ye[r] * ye[r] / (2.0f * (float)n);
    }
    float* o = part + (size_t)blockIdx.x * (kNParam + 1);
#pragma unroll
    for (int q = 0; q < 16; q++) o[oW2 + (16 * g + q) * kHid + u] = gw2[q];
#pragma unroll
    for (int c = 0; c < 3; c++) o[oW1 + u * kFeat + 3 * g + c] = gw1[c];
    if (g < 3) o[(g == 0 ? oB1 : (g == 1 ? oB2 : oW3)) + u] = gb;
    if (g == 3 && u == 0) o[oB3] = gout;
    if (g == 3 && u == 32) o[kNParam] = gout;
}

// Sum of the CTAs' gradients and losses: 32 parameters per CTA, eight warps over
// the partial gradients (w, w + 8, ...), their sums added in warp order.
constexpr int kSumWarps = 8;
__global__ void __launch_bounds__(32 * kSumWarps) k_mlp_sum(const float* part, int nblk, float* grad, float* loss)
{
    __shared__ float sh[kSumWarps][32];
    pdl_wait();
    pdl_trigger();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int p = blockIdx.x * 32 + lane;
    float a = 0.f;
    if (p <= kNParam) {
#pragma unroll 8
        for (int b = w; b < nblk; b += kSumWarps) a += part[(size_t)b * (kNParam + 1) + p];
    }
    sh[w][lane] = a;
    __syncthreads();
    if (w != 0 || p > kNParam) return;
#pragma unroll
    for (int k = 1; k < kSumWarps; k++) a += sh[k][lane];
    if (p < kNParam) grad[p] = a;
    else *loss = a;
}

// Adam (Kingma & Ba 2015) on the FP32 master weights; refreshes the BF16 copy.
__global__ void k_adam(float* master, __nv_bfloat16* w, float* m, float* v, const float* grad, float lr, float b1,
                       float b2, float eps, float c1, float c2)
{
    pdl_wait();
    pdl_trigger();
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= kNParam) return;
    const float g = grad[p];
    const float mm = b1 * m[p] + (1.f - b1) * g;
    const float vv = b2 * v[p] + (1.f - b2) * g * g;
    m[p] = mm;
    v[p] = vv;
    const float x = master[p] - lr * (mm / c1) / (sqrtf(vv / c2) + eps);
    master[p] = x;
    w[p] = __float2bfloat16_rn(x);
}

void launch_features(const FeatParams& F, int n_segs, cudaStream_t s)
{
    if (n_segs > 0) launch_k(k_feat_seg, (unsigned)n_segs, (unsigned)kSegment, s, F);
}

void launch_propose(const ProposeParams& P, cudaStream_t s)
{
    if (P.n_sys > 0) launch_k(k_propose, (unsigned)((P.n_sys + 3) / 4), 128u, s, P);
}

}  // namespace redgb

// ---------------------------------------------------------------------------
// C ABI: the network on its own (training and evaluation on device buffers)
// ---------------------------------------------------------------------------
using namespace redgb;

int redgb_set_error(int code, const char* msg);

static_assert(sizeof(red_mlp_norm_t) == sizeof(MlpNorm), "red_mlp_norm_t mirrors MlpNorm");

namespace {
// The per-CTA gradients of red_mlp_grad: allocated and freed in the order of the
// caller's stream, so calls on several streams and threads have memory of their own (and
// a captured call has the graph's).  A pool per device keeps kWorkKept bytes for the
// next calls and gives back the rest whenever a stream is waited for.
constexpr int kMaxDevices = 64;
constexpr unsigned long long kWorkKept = 32ull << 20;   // two calls' largest workspaces
std::mutex g_pool_mu;
cudaMemPool_t g_pool[kMaxDevices] = {nullptr};

cudaError_t work_pool(cudaMemPool_t* pool)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lk(g_pool_mu);
    if (!g_pool[dev]) {
        cudaMemPoolProps p = {};
        p.allocType = cudaMemAllocationTypePinned;
        p.location.type = cudaMemLocationTypeDevice;
        p.location.id = dev;
        unsigned long long keep = kWorkKept;
        cudaMemPool_t q = nullptr;
        if ((e = cudaMemPoolCreate(&q, &p)) != cudaSuccess) return e;
        if ((e = cudaMemPoolSetAttribute(q, cudaMemPoolAttrReleaseThreshold, &keep)) != cudaSuccess) {
            cudaMemPoolDestroy(q);
            return e;
        }
        g_pool[dev] = q;
    }
    *pool = g_pool[dev];
    return cudaSuccess;
}

// The training kernels follow each other by programmatic dependent launch:
// each waits for its predecessor before it reads anything.
struct PdlScope {
    bool was = pdl_on();
    PdlScope() { set_pdl(true); }
    ~PdlScope() { set_pdl(was); }
};

int cuda_fail(cudaError_t e, const char* what)
{
    char buf[256];
    snprintf(buf, sizeof(buf), "%s: %s", what, cudaGetErrorString(e));
    return redgb_set_error(RED_ERR_CUDA, buf);
}
}  // namespace

extern "C" {

uint32_t red_mlp_param_count(void) { return (uint32_t)kNParam; }

int red_mlp_predict(const void* w_bf16, const red_mlp_norm_t* norm, const float* x, float* out, uint32_t n,
                    void* stream)
{
    if (!w_bf16 || !norm || (n && (!x || !out))) return redgb_set_error(RED_ERR_ARG, "red_mlp_predict: null argument");
    if (n == 0) return RED_OK;
    MlpNorm nm;
    memcpy(&nm, norm, sizeof(nm));
    k_mlp_rows<<<(n + 3) / 4, 128, 0, (cudaStream_t)stream>>>((const __nv_bfloat16*)w_bf16, nm, x, out, (int)n);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? RED_OK : cuda_fail(e, "red_mlp_predict");
}

int red_mlp_grad(const void* w_bf16, const float* xn, const float* tn, uint32_t n, float* grad, float* loss,
                 void* stream)
{
    if (!w_bf16 || !xn || !tn || !grad || !loss || n == 0)
        return redgb_set_error(RED_ERR_ARG, "red_mlp_grad: bad argument");
    const int nblk = (int)std::min<uint32_t>((n - 1) / kTrainRows + 1, kTrainCtas);
    cudaStream_t s = (cudaStream_t)stream;
    cudaMemPool_t pool = nullptr;
    float* work = nullptr;
    cudaError_t e = work_pool(&pool);
    if (e == cudaSuccess) e = cudaMallocFromPoolAsync(&work, (size_t)nblk * (kNParam + 1) * sizeof(float), pool, s);
    if (e != cudaSuccess) return cuda_fail(e, "red_mlp_grad: workspace");
    const PdlScope pdl;
    launch_k(k_mlp_train, (unsigned)nblk, (unsigned)kTrainThreads, s, (const __nv_bfloat16*)w_bf16, xn, tn, (int)n, work);
    launch_k(k_mlp_sum, (unsigned)(kNParam / 32 + 1), 32u * kSumWarps, s, (const float*)work, nblk, grad, loss);
    e = cudaGetLastError();
    const cudaError_t f = cudaFreeAsync(work, s);
    if (e == cudaSuccess) e = f;
    return e == cudaSuccess ? RED_OK : cuda_fail(e, "red_mlp_grad");
}

int red_mlp_adam(float* master, void* w_bf16, float* m, float* v, const float* grad, uint32_t step, float lr,
                 float beta1, float beta2, float eps, void* stream)
{
    if (!master || !w_bf16 || !m || !v || !grad || step == 0)
        return redgb_set_error(RED_ERR_ARG, "red_mlp_adam: bad argument");
    const float c1 = 1.0f - powf(beta1, (float)step), c2 = 1.0f - powf(beta2, (float)step);
    const PdlScope pdl;
    launch_k(k_adam, (unsigned)((kNParam + 127) / 128), 128u, (cudaStream_t)stream, master, (__nv_bfloat16*)w_bf16, m, v,
             grad, lr, beta1, beta2, eps, c1, c2);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? RED_OK : cuda_fail(e, "red_mlp_adam");
}

}  // extern "C"
