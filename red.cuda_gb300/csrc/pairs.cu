// pairs.cu -- k_pairs: gravity with each pair formed once (pairs.cuh).
#include "common.cuh"
#include "pairs.cuh"

namespace redgb {

namespace {

__device__ __forceinline__ float2 dup(float a) { return make_float2(a, a); }

// One body j (h, l: its double-single position, h.w its mass) against the
// thread's four sinks, held as two pairs: packed FP32, one instruction for two
// pair terms.  With SYM the terms go both ways: (jx, jy, jz) += m_i d / |d|^3,
// the negative of j's acceleration.  The terms are the stage kernel's
// (gravity_f32).
template <int MODE, bool SYM>
__device__ __forceinline__ void pair_step(float4 h, float4 l, const float2 (&nH)[2][3], const float2 (&nL)[2][3],
                                          const float2 (&mi)[2], float2 (&a)[2][3], float& jx, float& jy, float& jz)
{
    const float2 hx = dup(h.x), hy = dup(h.y), hz = dup(h.z), mj = dup(h.w);
    float2 sx = make_float2(jx, 0.f), sy = make_float2(jy, 0.f), sz = make_float2(jz, 0.f);
#pragma unroll
    for (int p = 0; p < 2; p++) {
        float2 dx = __fadd2_rn(hx, nH[p][0]), dy = __fadd2_rn(hy, nH[p][1]), dz = __fadd2_rn(hz, nH[p][2]);
        if (MODE == MODE_MIXED) {
            dx = __fadd2_rn(dx, __fadd2_rn(dup(l.x), nL[p][0]));
            dy = __fadd2_rn(dy, __fadd2_rn(dup(l.y), nL[p][1]));
            dz = __fadd2_rn(dz, __fadd2_rn(dup(l.z), nL[p][2]));
        }
        float2 r2 = __ffma2_rn(dx, dx, dup(kEps2));
        r2 = __ffma2_rn(dy, dy, r2);
        r2 = __ffma2_rn(dz, dz, r2);
        const float2 ri = make_float2(rsqrtf(r2.x), rsqrtf(r2.y));
        const float2 ri3 = __fmul2_rn(ri, __fmul2_rn(ri, ri));   // at most 1e36 (kEps2)
        const float2 si = __fmul2_rn(mj, ri3);
        a[p][0] = __ffma2_rn(si, dx, a[p][0]);
        a[p][1] = __ffma2_rn(si, dy, a[p][1]);
        a[p][2] = __ffma2_rn(si, dz, a[p][2]);
        if (SYM) {
            const float2 sj = __fmul2_rn(mi[p], ri3);
            sx = __ffma2_rn(sj, dx, sx);
            sy = __ffma2_rn(sj, dy, sy);
            sz = __ffma2_rn(sj, dz, sz);
        }
    }
    if (SYM) {
        jx = sx.x + sx.y;
        jy = sy.x + sy.y;
        jz = sz.x + sz.y;
    }
}

struct PairSmem {
    float4 h[kTile], l[kTile];                // the sub-block's bodies
    float2 j[kTile / 32][3][kTile];           // per warp: their sums over the warp's sinks
};

}  // namespace

// Lane l of a warp takes body (l + s) mod 32 of a group of 32 in step s, so the
// 32 bodies are read without bank conflicts and each meets every sink of the warp
// once; the running sum of a body moves one lane down per step.  FP32 sums of at
// most 32 terms (two packed halves of 16) go into double-single ones: a body's
// every 8 steps, a sink's every 32.
//
// Bound by the FP32 pipe (76 % busy): 22 operations a pair in MIXED and 16 in FP32
// mode, where one-sided terms take 36 and 24; the other per-step work (two loads,
// three shuffles, three adds, the packed copies of the body) issues beside it.
// 16384 bodies, adaptive RKF7(8) in MIXED: 2.74 -> 1.79 ms per try against the
// one-sided tiles (1.70 with the packed collision filter); 65536 bodies, RK4 in FP32: 8.17 -> 5.58 ms.
template <int MODE>
__global__ void __launch_bounds__(kTile, 4) k_pairs(const PairParams P)
{
    __shared__ PairSmem sm;
    const PairJob job = P.jobs[blockIdx.x];
    pdl_wait();
    pdl_trigger();
    if (!runnable(*P.sys)) return;   // uniform over the grid
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    // sinks: 32 p + lane of the warp's 128
    const int i0 = job.block * kPairBlock + w * 128;
    float2 nH[2][3], nL[2][3], mi[2], acc_h[2][3], acc_l[2][3];
#pragma unroll
    for (int p = 0; p < 2; p++) {
        float4 H[2], L[2];
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int i = i0 + 32 * (2 * p + q) + lane;
            H[q] = i < P.n ? P.pos_hi[P.b0 + i] : make_float4(1.0e9f, 0.f, 0.f, 0.f);   // no body: no mass
            L[q] = MODE == MODE_MIXED && i < P.n ? P.pos_lo[P.b0 + i] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        nH[p][0] = make_float2(-H[0].x, -H[1].x);
        nH[p][1] = make_float2(-H[0].y, -H[1].y);
        nH[p][2] = make_float2(-H[0].z, -H[1].z);
        nL[p][0] = make_float2(-L[0].x, -L[1].x);
        nL[p][1] = make_float2(-L[0].y, -L[1].y);
        nL[p][2] = make_float2(-L[0].z, -L[1].z);
        mi[p] = make_float2(H[0].w, H[1].w);
#pragma unroll
        for (int c = 0; c < 3; c++) acc_h[p][c] = acc_l[p][c] = make_float2(0.f, 0.f);
    }
    float4 h, l = make_float4(0.f, 0.f, 0.f, 0.f);
    auto fetch = [&](int sub) {
        const int j = sub * kTile + t;
        h = j < P.n ? P.pos_hi[P.b0 + j] : make_float4(-1.0e9f, 0.f, 0.f, 0.f);
        if (MODE == MODE_MIXED) l = j < P.n ? P.pos_lo[P.b0 + j] : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    fetch(job.sub0);
    for (int sub = job.sub0; sub < job.sub1; sub++) {
        const bool sym = sub >= (job.block + 1) * kPairSinks;   // not the block itself; uniform
        __syncthreads();   // the previous sub-block is done with
        sm.h[t] = h;
        if (MODE == MODE_MIXED) sm.l[t] = l;
        __syncthreads();
        if (sub + 1 < job.sub1) fetch(sub + 1);
        for (int g = 0; g < kTile; g += 32) {
            float2 a[2][3];
#pragma unroll
            for (int p = 0; p < 2; p++)
#pragma unroll
                for (int c = 0; c < 3; c++) a[p][c] = make_float2(0.f, 0.f);
            if (sym) {
#pragma unroll 1
                for (int s0 = 0; s0 < 32; s0 += 8) {
                    float jx = 0.f, jy = 0.f, jz = 0.f;
#pragma unroll
                    for (int s = 0; s < 8; s++) {
                        if (s > 0) {
                            const int from = (lane + 1) & 31;
                            jx = __shfl_sync(0xffffffffu, jx, from);
                            jy = __shfl_sync(0xffffffffu, jy, from);
                            jz = __shfl_sync(0xffffffffu, jz, from);
                        }
                        const int jj = g + ((lane + s0 + s) & 31);
                        pair_step<MODE, true>(sm.h[jj], MODE == MODE_MIXED ? sm.l[jj] : l, nH, nL, mi, a, jx, jy, jz);
                    }
                    const int jj = g + ((lane + s0 + 7) & 31);
                    const float v[3] = {jx, jy, jz};
#pragma unroll
                    for (int c = 0; c < 3; c++) {
                        float2 d = s0 > 0 ? sm.j[w][c][jj] : make_float2(0.f, 0.f);
                        ds_add(d.x, d.y, v[c]);
                        sm.j[w][c][jj] = d;
                    }
                    __syncwarp();   // the next eight steps add to the same sums from other lanes
                }
            } else {
                float jx = 0.f, jy = 0.f, jz = 0.f;
#pragma unroll 4
                for (int s = 0; s < 32; s++) {
                    const int jj = g + ((lane + s) & 31);
                    pair_step<MODE, false>(sm.h[jj], MODE == MODE_MIXED ? sm.l[jj] : l, nH, nL, mi, a, jx, jy, jz);
                }
            }
#pragma unroll
            for (int p = 0; p < 2; p++)
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    ds_add(acc_h[p][c].x, acc_l[p][c].x, a[p][c].x);
                    ds_add(acc_h[p][c].y, acc_l[p][c].y, a[p][c].y);
                }
        }
        if (sym) {
            __syncthreads();
            const int j = sub * kTile + t;
            if (j < P.n) {
                float2* o = P.rec + 3 * ((size_t)job.block * P.n + j);
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    float2 d = sm.j[0][c][t];
#pragma unroll
                    for (int k = 1; k < kTile / 32; k++) ds_merge(d.x, d.y, sm.j[k][c][t].x, sm.j[k][c][t].y);
                    d = dsn_norm(-d.x, -d.y);
                    o[c] = d;
                }
            }
        }
    }
#pragma unroll
    for (int p = 0; p < 2; p++)
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int i = i0 + 32 * (2 * p + q) + lane;
            if (i >= P.n) continue;
            float2* o = P.rec + 3 * ((size_t)job.slot * P.n + i);
#pragma unroll
            for (int c = 0; c < 3; c++)
                o[c] = q == 0 ? dsn_norm(acc_h[p][c].x, acc_l[p][c].x) : dsn_norm(acc_h[p][c].y, acc_l[p][c].y);
        }
}

void launch_pairs(const PairParams& P, int n_jobs, int mode, cudaStream_t s)
{
    if (mode == MODE_MIXED) launch_k(k_pairs<MODE_MIXED>, (unsigned)n_jobs, (unsigned)kTile, s, P);
    else launch_k(k_pairs<MODE_FP32>, (unsigned)n_jobs, (unsigned)kTile, s, P);
}

}  // namespace redgb
