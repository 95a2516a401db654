// pairs.cu -- k_pairs: gravity with each pair formed once (pairs.cuh).
#include "common.cuh"
#include "pairs.cuh"

namespace redgb {

namespace {

__device__ __forceinline__ float2 dup(float a) { return make_float2(a, a); }

// x added to the double-single sums (h, l), two of them side by side in packed FP32:
// Knuth's TwoSum as ds_add has it, differences as a - b = fma(b, -1, a).
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, dup(-1.f), a); }
__device__ __forceinline__ void ds_add2(float2& h, float2& l, float2 x)
{
    const float2 s = __fadd2_rn(h, x);
    const float2 t = sub2(s, h);
    l = __fadd2_rn(l, __fadd2_rn(sub2(h, sub2(s, t)), sub2(x, t)));
    h = s;
}

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
    // MIXED sums the four terms on the body before the running sum takes them
    constexpr bool kApart = MODE == MODE_MIXED;
    float2 sx = make_float2(kApart ? 0.f : jx, 0.f), sy = make_float2(kApart ? 0.f : jy, 0.f),
           sz = make_float2(kApart ? 0.f : jz, 0.f);
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
        jx = kApart ? jx + (sx.x + sx.y) : sx.x + sx.y;
        jy = kApart ? jy + (sy.x + sy.y) : sy.x + sy.y;
        jz = kApart ? jz + (sz.x + sz.y) : sz.x + sz.y;
    }
}

struct PairSmem {
    float4 h[kTile], l[kTile];                // the sub-block's bodies
    float2 j[kTile / 32][3][kTile];           // per warp: their sums over the warp's sinks
};

}  // namespace

// Lane l of a warp takes body (l + s) mod 32 of a group of 32 in step s, so the
// 32 bodies are read without bank conflicts and each meets every sink of the warp
// once; the running sum of a body moves one lane down per step.  Runs of FP32 sums go
// into double-single ones: a body's every kRunJ steps (of four sinks), a sink's every kRun
// (kRunOwn against its own block; with eight there the whole takes 1 % longer).
//
// The runs of MIXED are as short as its accuracy needs: median relative error of the
// accelerations of a field of protoplanets 1.3 % below the one-sided tiles' (16 terms to a
// sum, in two halves), of a cube the same; with 32 terms to both sums, as FP32 mode
// has them, 10 and 7 % above.  That costs 10 % (16384 bodies, four tries: 6.82 -> 7.49 ms).
// In FP32 mode the rounding of the coordinates hides the sums': errors within 0.2 % of
// the one-sided tiles' (rms) with the long runs, which are 10 % faster than runs of 16.
//
// Bound by the FP32 pipe (76 % busy with long runs): 22 operations a pair in MIXED and 16 in
// FP32 mode, where one-sided terms take 36 and 24; the other per-step work (two loads,
// three shuffles, three adds, the packed copies of the body) issues beside it.
// 16384 bodies, adaptive RKF7(8) in MIXED: 2.74 -> 1.87 ms per try against the
// one-sided tiles; 65536 bodies, RK4 in FP32: 8.17 -> 5.52 ms.
template <int MODE>
__global__ void __launch_bounds__(kTile, 4) k_pairs(const PairParams P)
{
    __shared__ PairSmem sm;
    constexpr int kRun = MODE == MODE_MIXED ? 8 : 32, kRunJ = 8;   // steps of a run: a sink's, a body's
    constexpr int kRunOwn = MODE == MODE_MIXED ? 4 : 32;           // a sink's within its own block
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
            auto clear = [&]() {
#pragma unroll
                for (int p = 0; p < 2; p++)
#pragma unroll
                    for (int c = 0; c < 3; c++) a[p][c] = make_float2(0.f, 0.f);
            };
            auto fold = [&]() {
#pragma unroll
                for (int p = 0; p < 2; p++)
#pragma unroll
                    for (int c = 0; c < 3; c++) ds_add2(acc_h[p][c], acc_l[p][c], a[p][c]);
            };
            if (sym) {
#pragma unroll 1
                for (int s0 = 0; s0 < 32; s0 += kRunJ) {
                    float jx = 0.f, jy = 0.f, jz = 0.f;
                    if (s0 % kRun == 0) clear();
#pragma unroll
                    for (int s = 0; s < kRunJ; s++) {
                        if (s > 0) {
                            const int from = (lane + 1) & 31;
                            jx = __shfl_sync(0xffffffffu, jx, from);
                            jy = __shfl_sync(0xffffffffu, jy, from);
                            jz = __shfl_sync(0xffffffffu, jz, from);
                        }
                        const int jj = g + ((lane + s0 + s) & 31);
                        pair_step<MODE, true>(sm.h[jj], MODE == MODE_MIXED ? sm.l[jj] : l, nH, nL, mi, a, jx, jy, jz);
                    }
                    if ((s0 + kRunJ) % kRun == 0) fold();
                    const int jj = g + ((lane + s0 + kRunJ - 1) & 31);
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
#pragma unroll 1
                for (int s0 = 0; s0 < 32; s0 += kRunOwn) {
                    clear();
#pragma unroll 4
                    for (int s = 0; s < kRunOwn; s++) {
                        const int jj = g + ((lane + s0 + s) & 31);
                        pair_step<MODE, false>(sm.h[jj], MODE == MODE_MIXED ? sm.l[jj] : l, nH, nL, mi, a, jx, jy, jz);
                    }
                    fold();
                }
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
