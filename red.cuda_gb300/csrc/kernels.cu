// kernels.cu -- the sm_103a kernels of libredgb.
//
//   (k_stage, one Runge-Kutta stage, is in stage.cuh / stage_*.cu)
//   k_prep      positions of stage 0 from y (FP32 double-single copies)
//   k_control   per-system error -> accept / reject -> new step size
//   k_finish    y_{n+1} for accepted systems, positions of the next stage 0,
//               the small bodies into the collision check's spatial hash
//   k_collide   the collision check after a try: tile pairs of the large
//               bodies (FP32 prefilter + red's FP64 test) and hash queries
//   k_collision, k_grid_insert, k_grid_query   the same, for the explicit check
//   k_ejhc      ejection / hit-centrum test
//   k_potential potential sums for the integrals
#include <algorithm>
#include <cfloat>
#include <cstdio>

#include "common.cuh"
#include "control.cuh"
#include "try.cuh"

namespace redgb {

namespace {
thread_local bool t_pdl = false;
}
void set_pdl(bool on) { t_pdl = on; }
bool pdl_on() { return t_pdl; }

// ---------------------------------------------------------------------------
// per-body kernels
// ---------------------------------------------------------------------------
// FP32 copies of y_r for stage 0 (buffer 0), and the mass / radius words of
// both stage buffers: the stage kernels write only x, y, z, so the .w words
// set here hold until the next host update of the bodies.
__global__ void __launch_bounds__(kSegment) k_prep(const Segment* segs, const SysInfo* sinfo, const DevSys* sys,
                                                   const double* y_r, const double* mass, const double* radius,
                                                   const int* id, float4* hi, float4* lo, float4* hi1, float4* lo1,
                                                   int all)
{
    const Segment sg = segs[blockIdx.x];
    if (!all && !runnable(sys[sg.sys])) return;
    const int i = sg.b0 + threadIdx.x;
    if (i >= sg.b1) return;
    const double m_eff = id[i] >= 0 ? mass[i] : 0.0;
    write_pos(hi, lo, i, y_r[3 * i], y_r[3 * i + 1], y_r[3 * i + 2], m_eff, radius[i]);
    reinterpret_cast<float*>(hi1 + i)[3] = __double2float_rn(m_eff);
    reinterpret_cast<float*>(lo1 + i)[3] = __double2float_rn(radius[i]);
}

// One thread per system: the step control after a try (control.cuh).
__global__ void k_control(const ControlParams P)
{
    pdl_wait();
    pdl_trigger();
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= P.n_sys) return;
    DevSys& S = P.sys[s];
    S.accepted = 0;
    if (!runnable(S)) return;
    const unsigned long long err = S.err_bits;
    if (P.adaptive) S.err_bits = 0ull;
    control_system(P, S, err);
}

// Spatial-hash broad phase for the small bodies.
__device__ __forceinline__ int4 cell_of(double x, double y, double z, double inv_h)
{
    return make_int4(cell_coord(x, inv_h), cell_coord(y, inv_h), cell_coord(z, inv_h), 0);
}

// Inserts small body i at position (x, y, z) into its system's hash table.
__device__ __forceinline__ void grid_insert_one(const GridInfo& g, int4* cell, int* next, int* head, int i, double x,
                                                double y, double z)
{
    const int4 c = cell_of(x, y, z, g.inv_h);
    cell[i] = c;
    next[i] = atomicExch(&head[g.toff + bucket_of(c.x, c.y, c.z, g.mask)], i);
}

// y_{n+1} of the accepted systems and the positions of the next stage 0.  One
// thread per component: element e of a segment of kFinishBodies bodies is
// component e % 3 of body e / 3, contiguous in memory, so every FP64 warp
// instruction runs on full warps (the FP64 pipe charges a warp instruction the
// same for any number of active lanes).  The threads then form the hash-cell
// coordinate of their component, and one thread per small body inserts it
// into the collision check's spatial hash.
template <bool EXACT>
__global__ void __launch_bounds__(3 * kFinishBodies) k_finish(const FinishParams P)
{
    pdl_wait();
    pdl_trigger();
    __shared__ int cellc[3 * kFinishBodies];
    const Segment sg = P.segs[blockIdx.x];
    DevSys* S = P.sys + sg.sys;
    if (S->halted) return;
    const bool acc = S->accepted;
    if (!acc && !runnable(*S)) return;   // uniform over the CTA
    const int e = threadIdx.x;
    const int nb = sg.b1 - sg.b0;
    const bool live = e < 3 * nb;
    const int i = sg.b0 + e / 3;
    const int c = e % 3;
    const int x = 3 * sg.b0 + e;
    double r = 0.0;
    if (live) {
        if (acc) {
            const double dt = S->dt_did;
            double v;
            if (P.scheme == SCHEME_RKF78) {
                r = rk8_ynp1<EXACT>(P.y_r[x], dt, P.Kr, x);
                v = rk8_ynp1<EXACT>(P.y_v[x], dt, P.Kv, x);
            } else if (P.scheme == SCHEME_EULER) {
                // euler::calc_y_np1 -> sum_vector, int_euler.cu:19-31, 54-71: y + dt f0
                r = madd<EXACT>(P.y_r[x], dt, P.Kr[0][x]);
                v = madd<EXACT>(P.y_v[x], dt, P.Kv[0][x]);
            } else if (P.scheme == SCHEME_RK2) {
                // rungekutta2::calc_y_np1, int_rungekutta2.cu:66-83: y + (b_1 dt) f2
                const double bf = mul<EXACT>(c_tb.b2[1], dt);
                r = madd<EXACT>(P.y_r[x], bf, P.Kr[1][x]);
                v = madd<EXACT>(P.y_v[x], bf, P.Kv[1][x]);
            } else if (P.commit_from_stage4) {
                r = P.t_r0[x];
                v = P.Kr[4][x];
            } else {
                const double b0 = mul<EXACT>(c_tb.b4[0], dt), b1 = mul<EXACT>(c_tb.b4[1], dt);
                r = rk4_ynp1<EXACT>(P.y_r[x], b0, b1, P.Kr[0][x], P.Kr[1][x], P.Kr[2][x], P.Kr[3][x]);
                v = rk4_ynp1<EXACT>(P.y_v[x], b0, b1, P.Kv[0][x], P.Kv[1][x], P.Kv[2][x], P.Kv[3][x]);
            }
            P.y_r[x] = r;
            P.y_v[x] = v;
            // finiteness from the exponent bits (integer pipe, not the FP64 pipe)
            const long long br = __double_as_longlong(r), bv = __double_as_longlong(v);
            if (((br >> 52) & 0x7ff) == 0x7ff || ((bv >> 52) & 0x7ff) == 0x7ff) S->status = 5;   // RED_ERR_NONFINITE
        } else {
            r = P.y_r[x];
        }
        // x, y, z of the FP32 copies; k_prep holds the .w words (mass, radius)
        write_pos_c(P.pos_hi0, P.pos_lo0, i, c, r);
    }
    if (P.head && acc) {   // uniform over the CTA
        const GridInfo g = P.grid[sg.sys];
        if (!g.enabled) return;
        if (live) cellc[e] = cell_coord(r, g.inv_h);
        __syncthreads();
        const int small0 = P.sinfo[sg.sys].off + P.sinfo[sg.sys].n_SI;
        if (e < nb && sg.b0 + e >= small0) {
            const int b = sg.b0 + e;
            const int4 cl = make_int4(cellc[3 * e], cellc[3 * e + 1], cellc[3 * e + 2], 0);
            P.cell[b] = cl;
            P.next[b] = atomicExch(&P.head[g.toff + bucket_of(cl.x, cl.y, cl.z, g.mask)], b);
        }
    }
}

// ---------------------------------------------------------------------------
// collision detection: kernel_pp_disk::check_for_collision (pp_disk.cu:320-371)
// over tile pairs; an FP32 filter with a safety margin picks the candidates, red's
// FP64 test (no FMA) decides.
// ---------------------------------------------------------------------------
// After a try the check runs for the systems that just accepted one (a halted
// system makes no tries, so it never has `accepted` set); the explicit check
// runs for every system.  `halted` is not consulted: the first kernel of the
// check may set it.
__device__ __forceinline__ bool coll_runs(const CollParams& P, const DevSys& S)
{
    return !P.only_accepted || S.accepted;
}

// red's test for one pair i < j, bit for bit (pp_disk.cu:336-357), and the event.
__device__ __forceinline__ void collide_exact(const CollParams& P, DevSys* S, int sys, int i, int jx, double f)
{
    if (!(0 < P.id[i]) || 0 > P.id[jx]) return;
    const double ddx = __dsub_rn(P.y_r[3 * jx], P.y_r[3 * i]);
    const double ddy = __dsub_rn(P.y_r[3 * jx + 1], P.y_r[3 * i + 1]);
    const double ddz = __dsub_rn(P.y_r[3 * jx + 2], P.y_r[3 * i + 2]);
    const double w = __dadd_rn(__dadd_rn(__dmul_rn(ddx, ddx), __dmul_rn(ddy, ddy)), __dmul_rn(ddz, ddz));
    const double rs = __dadd_rn(P.radius[i], P.radius[jx]);
    if (!(w < __dmul_rn(f, __dmul_rn(rs, rs)))) return;
    int surv = i, merg = jx;
    if (P.mass[merg] > P.mass[surv]) {
        surv = jx;
        merg = i;
    }
    const unsigned kk = atomicAdd(P.n_events, 1u);
    if (kk < P.capacity) {
        DevEvent ev;
        ev.sys = sys;
        ev.name = 3;   // RED_EVENT_COLLISION
        ev.i = i;
        ev.j = jx;
        ev.surv = surv;
        ev.merg = merg;
        ev.d = __dsqrt_rn(w);
        P.events[kk] = ev;
    }
    if (P.mark) {
        atomicAdd(&S->n_coll, 1);
        S->halted = 1;
    }
}

// Brute-force tile pairs: the large bodies (SI class) against every later body.
// A thread takes four later bodies, as two pairs of packed FP32; the i tile (the SI
// bodies) sits in shared memory, every value twice.
//
// The filter sees the FP32 copies of the positions alone: two bodies closer than
// T = factor (R_i + R_j) are there closer than A_i + A_j, A = factor R + 2^-23 M, M the
// largest |coordinate|.  A copy is its coordinate truncated, off by up to 2^-23 |x| towards
// zero.  Coordinates of one sign: the errors' difference is at most the larger one, over
// three of them sqrt(3) 2^-23 max(M_i, M_j), which is below 2^-23 (M_i + M_j) where T <
// 0.26 max(M_i, M_j), since the M differ by at most T, and below 8e-7 T elsewhere.
// Coordinates of opposite signs: at most 2^-23 of their distance.  The factor 1.0001 covers
// the shares of T and the filter's own rounding, 1e-15 what FP32 flushes.  The few that
// pass, and whatever compares with NaN or infinity, take red's FP64 test.
//
// Bound by instruction issue: ~6 a pair, where double-single differences of one pair
// at a time took ~24.  16384 bodies, all pairs: 158 -> 57 us. The
// rare pairs go through one copy of the FP64 test: eight inlined ones cost a
// 261-body step 5 us of instruction fetches.
__device__ __forceinline__ float2 coll_reach(const float4 (&H)[2], const float (&R)[2], float fac)
{
    float a[2];
#pragma unroll
    for (int q = 0; q < 2; q++)
        a[q] = fmaf(fmaf(fac, fabsf(R[q]), 0x1p-23f * fmaxf(fmaxf(fabsf(H[q].x), fabsf(H[q].y)), fabsf(H[q].z))),
                    1.0001f, 1.0e-15f);
    return make_float2(a[0], a[1]);
}
__device__ __forceinline__ void coll_pairs(const CollParams& P, int item)
{
    __shared__ float4 sxy[kTile], sza[kTile];   // x, x, y, y; z, z, reach, reach
    const PairItem it = P.items[item];
    DevSys* S = P.sys + it.sys;
    if (!coll_runs(P, *S)) return;
    const SysInfo si = P.sinfo[it.sys];
    const int end = si.off + si.n;
    const int ni = min(kTile, it.i1 - it.i0);
    const int t = threadIdx.x;
    const float fac = fabsf((float)P.factor);
    if (t < ni) {
        const float4 H[2] = {P.pos_hi[it.i0 + t], make_float4(0.f, 0.f, 0.f, 0.f)};
        const float R[2] = {P.pos_lo[it.i0 + t].w, 0.f};
        const float2 A = coll_reach(H, R, fac);
        sxy[t] = make_float4(H[0].x, H[0].x, H[0].y, H[0].y);
        sza[t] = make_float4(H[0].z, H[0].z, A.x, A.x);
    }
    constexpr int N = kCollBodies / 2;
    float2 nx[N], ny[N], nz[N], A[N];
#pragma unroll
    for (int p = 0; p < N; p++) {
        float4 H[2];
        float R[2];
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int j = it.j0 + (2 * p + q) * kTile + t;
            H[q] = j < end ? P.pos_hi[j] : make_float4(0.f, 0.f, 0.f, 0.f);
            R[q] = j < end ? P.pos_lo[j].w : 0.f;
        }
        nx[p] = make_float2(-H[0].x, -H[1].x);
        ny[p] = make_float2(-H[0].y, -H[1].y);
        nz[p] = make_float2(-H[0].z, -H[1].z);
        A[p] = coll_reach(H, R, fac);
    }
    __syncthreads();
    if (it.j0 + t >= end) return;
    const double f = P.factor * P.factor;
#pragma unroll 2
    for (int ii = 0; ii < ni; ii++) {
        const float4 u = sxy[ii], v = sza[ii];
        bool near[2 * N];
        bool any = false;
#pragma unroll
        for (int p = 0; p < N; p++) {
            const float2 dx = __fadd2_rn(make_float2(u.x, u.y), nx[p]), dy = __fadd2_rn(make_float2(u.z, u.w), ny[p]);
            const float2 dz = __fadd2_rn(make_float2(v.x, v.y), nz[p]), a = __fadd2_rn(make_float2(v.z, v.w), A[p]);
            const float2 d2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx))), a2 = __fmul2_rn(a, a);
            near[2 * p] = !(d2.x > a2.x);
            near[2 * p + 1] = !(d2.y > a2.y);
            any = any || near[2 * p] || near[2 * p + 1];
        }
        if (!any) continue;
        const int i = it.i0 + ii;
        unsigned m = 0;
#pragma unroll
        for (int q = 0; q < 2 * N; q++) {
            const int j = it.j0 + q * kTile + t;
            m |= near[q] && i < j && j < end ? 1u << q : 0u;   // a body is near itself
        }
#pragma unroll 1
        for (; m; m &= m - 1) collide_exact(P, S, it.sys, i, it.j0 + (__ffs((int)m) - 1) * kTile + t, f);
    }
}

__global__ void __launch_bounds__(kTile) k_collision(const CollParams P)
{
    pdl_wait();
    pdl_trigger();
    coll_pairs(P, blockIdx.x);
}



__global__ void __launch_bounds__(kSegment) k_grid_insert(const CollParams P)
{
    pdl_wait();
    pdl_trigger();
    const Segment sg = P.segs[blockIdx.x];
    const DevSys& S = P.sys[sg.sys];
    const GridInfo g = P.grid[sg.sys];
    if (!g.enabled || !coll_runs(P, S)) return;
    const SysInfo si = P.sinfo[sg.sys];
    const int i = sg.b0 + threadIdx.x;
    if (i >= sg.b1 || i < si.off + si.n_SI) return;
    grid_insert_one(g, P.cell, P.next, P.head, i, P.y_r[3 * i], P.y_r[3 * i + 1], P.y_r[3 * i + 2]);
}

// Half of the neighbourhood: the own cell (pairs with j > i) and the 13 cells
// of the forward half-space, so that every unordered pair of small bodies in
// neighbouring cells is seen once; the pair is tested as (min, max) like red's
// i < j loop.  The 14 bucket lists are walked side by side: each round loads
// the current element of every list at once, so a thread needs as many
// dependent memory round trips as its longest list, not their sum.
__device__ __forceinline__ void grid_query(const CollParams& P, int seg, int local)
{
    const Segment sg = P.segs[seg];
    DevSys* S = P.sys + sg.sys;
    const GridInfo g = P.grid[sg.sys];
    if (!g.enabled || !coll_runs(P, *S)) return;
    const SysInfo si = P.sinfo[sg.sys];
    const int i = sg.b0 + local;
    if (i >= sg.b1 || i < si.off + si.n_SI) return;
    const double f = P.factor * P.factor;
    const int4 c = P.cell[i];
    // A neighbouring cell is looked up if the body is within a collision distance of
    // it: with cells of four such distances 2.2 of the 14 lists on average (512 disks:
    // the check 123 -> ~50 us).  The body's place u in its cell, 0 .. 1, comes from the
    // FP32 copy, off by less than 2^-21 (|c| + 2) edges; a u far from there (edges or
    // positions out of FP32's range) tells nothing, and all neighbours are looked up.
    const float4 H = P.pos_hi[i];
    const float inv_h = (float)g.inv_h;
    bool lo[3], hi[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const int ck = k == 0 ? c.x : (k == 1 ? c.y : c.z);
        const float u = fmaf(k == 0 ? H.x : (k == 1 ? H.y : H.z), inv_h, -(float)ck);
        const float reach = g.reach + 0x1p-21f * (fabsf((float)ck) + 2.0f);
        const bool any = abs(ck) >= 1 << 18 || !(fabsf(u) < 2.0f);   // too far out for FP32
        lo[k] = any || !(u > reach);
        hi[k] = any || !(u < 1.0f - reach);
    }
    constexpr int kNb = 14;
    int cur[kNb];
    int4 nb[kNb];
    int q = 0;
#pragma unroll
    for (int dz = 0; dz <= 1; dz++)
#pragma unroll
        for (int dy = -1; dy <= 1; dy++)
#pragma unroll
            for (int dx = -1; dx <= 1; dx++) {
                const bool fwd = dz > 0 || (dz == 0 && (dy > 0 || (dy == 0 && dx >= 0)));
                if (!fwd) continue;
                nb[q] = make_int4(c.x + dx, c.y + dy, c.z + dz, 0);
                const bool near = (dx == 0 || (dx < 0 ? lo[0] : hi[0])) && (dy == 0 || (dy < 0 ? lo[1] : hi[1])) &&
                                  (dz == 0 || hi[2]);
                cur[q] = near ? __ldcg(P.head + g.toff + bucket_of(nb[q].x, nb[q].y, nb[q].z, g.mask)) : -1;
                q++;
            }
    // a list is at most as long as the system's small-body count: the bound ends every walk
    const int bound = si.n - si.n_SI;
    bool any = true;
    for (int round = 0; any && round <= bound; round++) {
        int4 cj[kNb];
        int nx[kNb];
#pragma unroll
        for (int b = 0; b < kNb; b++) {
            if (cur[b] >= 0) {
                cj[b] = P.cell[cur[b]];
                nx[b] = __ldcg(P.next + cur[b]);
            }
        }
        any = false;
#pragma unroll
        for (int b = 0; b < kNb; b++) {
            if (cur[b] >= 0) {
                const int j = cur[b];
                if (cj[b].x == nb[b].x && cj[b].y == nb[b].y && cj[b].z == nb[b].z && (b != 0 || j > i))
                    collide_exact(P, S, sg.sys, min(i, j), max(i, j), f);
                cur[b] = nx[b];
                any = any || nx[b] >= 0;
            }
        }
    }
}

__global__ void __launch_bounds__(kSegment) k_grid_query(const CollParams P)
{
    pdl_wait();
    pdl_trigger();
    grid_query(P, blockIdx.x, threadIdx.x);
}

// The collision check after a try in one launch: CTAs [0, n_pairs) test the
// tile pairs of the large bodies, the others run the hash-grid query for half
// a segment each (the bodies were inserted by k_finish).
static_assert(kSegment == 2 * kTile, "k_collide runs half a segment per CTA");
__global__ void __launch_bounds__(kTile) k_collide(const CollParams P, int n_pairs)
{
    pdl_wait();
    pdl_trigger();
    if ((int)blockIdx.x < n_pairs) {
        coll_pairs(P, blockIdx.x);
        return;
    }
    const int q = (int)blockIdx.x - n_pairs;
    grid_query(P, q / 2, (q % 2) * kTile + (int)threadIdx.x);
}

// kernel_pp_disk::check_for_ejection_hit_centrum (pp_disk.cu:283-318)
__global__ void __launch_bounds__(kSegment) k_ejhc(const EjhcParams P)
{
    pdl_wait();
    pdl_trigger();
    const Segment sg = P.segs[blockIdx.x];
    DevSys* S = P.sys + sg.sys;
    if (P.only_accepted && !S->accepted) return;
    if (S->halted && P.only_accepted) return;
    const int i = sg.b0 + threadIdx.x;
    if (i >= sg.b1) return;
    const double ed2 = 0.0 < P.ejection ? P.ejection * P.ejection : DBL_MAX;
    const double hcd2 = P.hit_centrum * P.hit_centrum;
    if (!(P.id[i] > 0 && P.btype[i] != 0)) return;
    const double x = P.y_r[3 * i], y = P.y_r[3 * i + 1], z = P.y_r[3 * i + 2];
    const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y)), __dmul_rn(z, z));
    const int star = P.sinfo[sg.sys].off;
    for (int which = 0; which < 2; which++) {
        const bool hit = which == 0 ? (ed2 < r2) : (hcd2 > r2);
        if (!hit) continue;
        const unsigned kk = atomicAdd(P.n_events, 1u);
        if (kk < P.capacity) {
            DevEvent ev;
            ev.sys = sg.sys;
            ev.name = which == 0 ? 2 : 1;   // RED_EVENT_EJECTION : RED_EVENT_HIT_CENTRUM
            ev.i = star;
            ev.j = i;
            ev.surv = star;
            ev.merg = i;
            ev.d = __dsqrt_rn(r2);
            P.events[kk] = ev;
        }
        if (P.mark) {
            atomicAdd(&S->n_ejhc, 1);
            S->halted = 1;
        }
    }
}

// Potential sums in FP64, each pair once: a CTA holds kTile bodies j (one per
// thread) against a range of bodies i, and writes sum m_i m_j / r_ij over its
// pairs with i < j, i < ni, j < nj (indices relative to the system; ids < 0 are
// skipped).  All pairs: ni = nj = n; the interacting ones: ni = n_SI, nj =
// n_massive.  CTA (x, y) of the grid: j from x kTile, i from y isub; one
// partial each, added by the host in order.  Bound by the FP64 pipe: 12
// instructions per pair.  With one thread per body i, over every j with a root
// and a division (one thread per large body for the interacting pairs), the
// two sums, the collision check and the state of the 16384-body disk took 44.1
// ms; with this kernel 4.6 ms.
__global__ void __launch_bounds__(kTile) k_potential(int off, int ni, int nj, int isub, const double* y_r,
                                                     const double* mass, const int* id, double* u)
{
    __shared__ D4 sh[kTile];
    __shared__ int on[kTile];
    __shared__ double part[kTile / 32];
    const int t = threadIdx.x;
    const int jt = blockIdx.x * kTile;
    const int i0 = blockIdx.y * isub, i1 = min(min(ni, i0 + isub), jt + kTile);
    const int j = jt + t;
    const bool live = j < nj && id[off + j] >= 0;
    double x = 0.0, y = 0.0, z = 0.0, acc = 0.0;
    if (live) {
        x = y_r[3 * (off + j)];
        y = y_r[3 * (off + j) + 1];
        z = y_r[3 * (off + j) + 2];
    }
    for (int b = i0; b < i1; b += kTile) {   // uniform over the CTA
        const int nb = min(kTile, i1 - b);
        __syncthreads();
        if (t < nb) {
            const int i = off + b + t;
            sh[t] = D4{y_r[3 * i], y_r[3 * i + 1], y_r[3 * i + 2], mass[i]};
            on[t] = id[i] >= 0;
        }
        __syncthreads();
        const int ne = live ? min(nb, j - b) : 0;   // i < j
#pragma unroll 4
        for (int k = 0; k < ne; k++) {
            const D4 q = sh[k];
            const double dx = q.x - x, dy = q.y - y, dz = q.z - z;
            const double ri = rsqrt_f64(fma(dz, dz, fma(dy, dy, dx * dx)));
            if (on[k]) acc = fma(q.w, ri, acc);
        }
    }
    acc = live ? acc * mass[off + j] : 0.0;
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((t & 31) == 0) part[t >> 5] = acc;
    __syncthreads();
    if (t == 0) {
        double a = part[0];
        for (int w = 1; w < kTile / 32; w++) a += part[w];
        u[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = a;
    }
}

// ---------------------------------------------------------------------------
// host transfers: one system's bodies between the device's structure of
// arrays and the caller's records (var4_t r, v; param_t p: 4n doubles each,
// one array per segment) and ib = [id, type] x n
// ---------------------------------------------------------------------------
__global__ void k_pack_state(int o, int n, const double* y_r, const double* y_v, const double* mass,
                             const double* radius, const double* density, const double* cd, const int* id,
                             const int* btype, StateSegs dst, int* ib)
{
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) {
        ib[2 * k] = id[o + k];
        ib[2 * k + 1] = btype[o + k];
    }
    if (k >= 12LL * n) return;
    const int seg = (int)(k / (4LL * n));
    double* out = dst.seg[seg];
    if (!out) return;
    const int w = (int)(k - seg * 4LL * n);
    const int i = o + w / 4, c = w % 4;
    double v;
    if (seg == 0) v = c < 3 ? y_r[3 * i + c] : 0.0;
    else if (seg == 1) v = c < 3 ? y_v[3 * i + c] : 0.0;
    else v = c == 0 ? mass[i] : (c == 1 ? radius[i] : (c == 2 ? density[i] : cd[i]));
    out[w] = v;
}

// Inverse of k_pack_state for the parts named in `what` (1 r, 2 v, 4 p, 8 id).
// New positions also go to the FP32 copies of stage 0 (x, y, z; the .w words
// follow mass and radius and are set by k_prep).
__global__ void k_unpack_state(int o, int n, int what, StateSegs src, const int* ib, double* y_r, double* y_v,
                               double* mass, double* radius, double* density, double* cd, int* id, float4* hi0,
                               float4* lo0)
{
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n && (what & 8)) id[o + k] = ib[2 * k];
    if (k >= 12LL * n) return;
    const int seg = (int)(k / (4LL * n));
    if (!(what & (1 << seg)) || !src.seg[seg]) return;
    const int w = (int)(k - seg * 4LL * n);
    const int i = o + w / 4, c = w % 4;
    const double v = src.seg[seg][w];
    if (seg == 0) {
        if (c < 3) y_r[3 * i + c] = v;
        write_pos_c(hi0, lo0, i, c, v);
    }
    else if (seg == 1) { if (c < 3) y_v[3 * i + c] = v; }
    else if (c == 0) mass[i] = v;
    else if (c == 1) radius[i] = v;
    else if (c == 2) density[i] = v;
    else cd[i] = v;
}

// Sets the try quota of every system (red_step: 1 accepted step, then -1 = none).
__global__ void k_set_quota(DevSys* sys, int n_sys, int q)
{
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < n_sys) sys[s].quota = q;
}

// Empties the partial-record slots of the stage kernel's chunk reduction.
__global__ void k_fill_records(unsigned long long* recs, size_t n)
{
    for (size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (size_t)gridDim.x * blockDim.x)
        recs[k] = kRecEmpty;
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
void launch_set_quota(DevSys* sys, int n_sys, int q, cudaStream_t s)
{
    if (n_sys > 0) k_set_quota<<<(unsigned)((n_sys + 127) / 128), 128, 0, s>>>(sys, n_sys, q);
}

void fill_records_empty(void* recs, size_t n, cudaStream_t s)
{
    if (n == 0) return;
    const unsigned blocks = (unsigned)std::min<size_t>((n + 255) / 256, 4 * 152);
    k_fill_records<<<blocks, 256, 0, s>>>(static_cast<unsigned long long*>(recs), n);
}

void set_tableau(const Tableau& tb, cudaStream_t s)
{
    cudaMemcpyToSymbolAsync(c_tb, &tb, sizeof(Tableau), 0, cudaMemcpyHostToDevice, s);
    set_tableau_mixed(tb, s);
    set_tableau_fp32(tb, s);
    set_tableau_fp64(tb, s);
    set_tableau_exact(tb, s);
    set_tableau_try(tb, s);
}

// Variant of k_stage: the shape of the combination its epilogue forms.
int stage_variant(const StageParams& P)
{
    if (P.standalone) return 0;
    if (P.err_after) return P.scheme == SCHEME_RKF78 ? 15 : 16;
    if (P.next < 0) return 0;
    if (P.scheme == SCHEME_RKF78) return P.next;   // next = stage + 1 in [1, 12]
    return P.ynp1_to_out ? 14 : 13;
}

void launch_stage(const StageParams& P, int n_items, int mode, cudaStream_t s)
{
    if (n_items <= 0) return;
    const int v = stage_variant(P);
    switch (mode) {
    case MODE_MIXED: launch_stage_mixed(P, n_items, v, s); break;
    case MODE_FP64: launch_stage_fp64(P, n_items, v, s); break;
    case MODE_FP64_EXACT: launch_stage_exact(P, n_items, v, s); break;
    default: launch_stage_fp32(P, n_items, v, s); break;
    }
}

int stage_active_clusters(int mode)
{
    if (mode == MODE_MIXED) return active_clusters_mixed();
    if (mode == MODE_FP32) return active_clusters_fp32();
    return 0;
}

void launch_prep(const Segment* segs, int n_segs, const SysInfo* sinfo, const DevSys* sys, const double* y_r,
                 const double* mass, const double* radius, const int* id, float4* hi, float4* lo, float4* hi1,
                 float4* lo1, int all, cudaStream_t s)
{
    if (n_segs > 0) k_prep<<<n_segs, kSegment, 0, s>>>(segs, sinfo, sys, y_r, mass, radius, id, hi, lo, hi1, lo1, all);
}

void launch_control(const ControlParams& P, cudaStream_t s)
{
    launch_k(k_control, (unsigned)((P.n_sys + 127) / 128), 128u, s, P);
}

void launch_finish(const FinishParams& P, int n_segs, cudaStream_t s)
{
    if (n_segs <= 0) return;
    if (P.stage_exact) launch_k(k_finish<true>, (unsigned)n_segs, 3u * kFinishBodies, s, P);
    else launch_k(k_finish<false>, (unsigned)n_segs, 3u * kFinishBodies, s, P);
}

// The explicit collision check (red_check_for_collision) on the current state.
void launch_collision(const CollParams& P, int n_items, int n_segs, bool use_grid, size_t table_size,
                      cudaStream_t s)
{
    if (n_items > 0) launch_k(k_collision, (unsigned)n_items, (unsigned)kTile, s, P);
    if (use_grid && n_segs > 0) {
        cudaMemsetAsync(P.head, 0xff, table_size * sizeof(int), s);
        launch_k(k_grid_insert, (unsigned)n_segs, (unsigned)kSegment, s, P);
        launch_k(k_grid_query, (unsigned)n_segs, (unsigned)kSegment, s, P);
    }
}

// The collision check after a try (k_collide): the bodies are in the hash
// already (k_finish), the pair tiles and the queries run in one launch.
void launch_collide(const CollParams& P, int n_items, int n_segs, bool use_grid, cudaStream_t s)
{
    const int nq = use_grid ? 2 * n_segs : 0;
    if (n_items + nq > 0) launch_k(k_collide, (unsigned)(n_items + nq), (unsigned)kTile, s, P, n_items);
}

void launch_pack_state(int o, int n, const double* y_r, const double* y_v, const double* mass, const double* radius,
                       const double* density, const double* cd, const int* id, const int* btype, StateSegs dst,
                       int* ib, cudaStream_t s)
{
    if (n <= 0) return;
    const long long tot = 12LL * n;
    k_pack_state<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(o, n, y_r, y_v, mass, radius, density, cd, id, btype,
                                                               dst, ib);
}

void launch_unpack_state(int o, int n, int what, StateSegs src, const int* ib, double* y_r, double* y_v,
                         double* mass, double* radius, double* density, double* cd, int* id, float4* hi0,
                         float4* lo0, cudaStream_t s)
{
    if (n <= 0) return;
    const long long tot = 12LL * n;
    k_unpack_state<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(o, n, what, src, ib, y_r, y_v, mass, radius,
                                                                 density, cd, id, hi0, lo0);
}

void launch_ejhc(const EjhcParams& P, int n_segs, cudaStream_t s)
{
    if (n_segs > 0) launch_k(k_ejhc, (unsigned)n_segs, (unsigned)kSegment, s, P);
}

int potential_partials(int ni, int nj, int* isub)
{
    const int tx = std::max(1, (nj + kTile - 1) / kTile);
    int ty = std::max(1, kPotentialCtas / tx);
    const int sub = std::max(32, ((ni + ty - 1) / ty + 31) / 32 * 32);
    ty = std::max(1, (ni + sub - 1) / sub);
    if (isub) *isub = sub;
    return tx * ty;
}

void launch_potential(int off, int ni, int nj, const double* y_r, const double* mass, const int* id, double* u,
                      cudaStream_t s)
{
    int isub = 0;
    const int parts = potential_partials(ni, nj, &isub);
    const int tx = std::max(1, (nj + kTile - 1) / kTile);
    k_potential<<<dim3((unsigned)tx, (unsigned)(parts / tx)), kTile, 0, s>>>(off, ni, nj, isub, y_r, mass, id, u);
}

}  // namespace redgb
