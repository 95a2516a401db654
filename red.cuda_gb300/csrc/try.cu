// try.cu -- k_try: a whole try of one sparse system; k_team: of an ensemble of them
// (try.cuh).
#include "records.cuh"
#include "try.cuh"

namespace redgb {

namespace {

// The acceleration m d / |d|^3 of a star of double-single mass m at (S, SL) on a
// body at (H, L), added to (ax, ay, az).
__device__ __forceinline__ void star_term(float4 S, float4 SL, float2 m, float4 H, float4 L, float2& ax, float2& ay,
                                          float2& az)
{
    const float2 dx = dsn_sub(dsn(S.x, SL.x), dsn(H.x, L.x));
    const float2 dy = dsn_sub(dsn(S.y, SL.y), dsn(H.y, L.y));
    const float2 dz = dsn_sub(dsn(S.z, SL.z), dsn(H.z, L.z));
    const float2 r2 = dsn_add(dsn_add(dsn_sqr(dx), dsn_sqr(dy)), dsn_sqr(dz));
    const float2 ri = dsn_rsqrt(r2);
    const float2 f = dsn_mul(m, dsn_mul(dsn_sqr(ri), ri));
    ax = dsn_add(ax, dsn_mul(f, dx));
    ay = dsn_add(ay, dsn_mul(f, dy));
    az = dsn_add(az, dsn_mul(f, dz));
}

// One FP32 pair term of the body at (H, L) from a source (h, l) of mass h.w,
// added to (x, y, z): the stage kernel's term (gravity_f32).
template <int MODE>
__device__ __forceinline__ void pair_term(float4 h, float4 l, float4 H, float4 L, float& x, float& y, float& z)
{
    float dx = h.x - H.x, dy = h.y - H.y, dz = h.z - H.z;
    if (MODE == MODE_MIXED) {
        dx += l.x - L.x;
        dy += l.y - L.y;
        dz += l.z - L.z;
    }
    const float ri = rsqrtf(fmaf(dz, dz, fmaf(dy, dy, fmaf(dx, dx, kEps2))));
    const float sc = h.w * ri * (ri * ri);
    x = fmaf(sc, dx, x);
    y = fmaf(sc, dy, y);
    z = fmaf(sc, dz, z);
}

// This CTA's copy of the large bodies' position records of stage s.
__device__ __forceinline__ const uint4* pos_records(const TryParams& P, int s)
{
    return P.pos + (size_t)((s & 3) * kTryCopies + blockIdx.x % kTryCopies) * P.n_large * 2;
}

struct Ds3 {   // a double-single vector
    float xh, xl, yh, yl, zh, zl;
};
__device__ __forceinline__ void fold(Ds3& a, float x, float y, float z)
{
    ds_add(a.xh, a.xl, x);
    ds_add(a.yh, a.yl, y);
    ds_add(a.zh, a.zl, z);
}
// The sum of a over `lanes` (4 .. 32) consecutive threads, a component to each:
// lane 0 returns x, lane 1 y, lane 2 z (of every group of 4).  The first two
// rounds halve the components a thread still carries.
__device__ __forceinline__ float2 reduce_scatter(const Ds3& a, int lane, int lanes)
{
    const bool odd = lane & 1;
    // round 1: even lanes keep (x, z), odd ones (y, -)
    const float sh = odd ? a.xh : a.yh, sl = odd ? a.xl : a.yl;
    float kh = odd ? a.yh : a.xh, kl = odd ? a.yl : a.xl, zh = a.zh, zl = a.zl;
    float rh = __shfl_xor_sync(0xffffffffu, sh, 1), rl = __shfl_xor_sync(0xffffffffu, sl, 1);
    ds_merge(kh, kl, rh, rl);
    rh = __shfl_xor_sync(0xffffffffu, zh, 1);
    rl = __shfl_xor_sync(0xffffffffu, zl, 1);
    ds_merge(zh, zl, rh, rl);
    // round 2: lanes 0, 1 keep x, y; lanes 2, 3 the z of their pair (the same in both)
    const bool up = lane & 2;
    rh = __shfl_xor_sync(0xffffffffu, up ? kh : zh, 2);
    rl = __shfl_xor_sync(0xffffffffu, up ? kl : zl, 2);
    kh = up ? zh : kh;
    kl = up ? zl : kl;
    ds_merge(kh, kl, rh, rl);
    for (int m = 4; m < lanes; m <<= 1) {
        rh = __shfl_xor_sync(0xffffffffu, kh, m);
        rl = __shfl_xor_sync(0xffffffffu, kl, m);
        ds_merge(kh, kl, rh, rl);
    }
    return dsn_norm(kh, kl);
}

__device__ __forceinline__ void put_comp(float4* hi, float4* lo, int b, int c, double x)
{
    float h, l;
    split_ds(x, h, l);
    reinterpret_cast<float*>(hi + b)[c] = h;
    reinterpret_cast<float*>(lo + b)[c] = l;
}

// Gas drag of a body at (H, L) with velocity v, added to its acceleration a: the
// stage kernel's, in FP64 but for the drag factor (drag_factor_fast).
// With the gas velocity in double-single a massless first body, whose gas is at rest,
// gave NaN, and its rounding grows where v_gas - v cancels.
__device__ __forceinline__ void gas_drag(const GasDev& G, double decr, double mstar, float4 H, float4 L,
                                         const double (&v)[3], double cd, double radius, double density,
                                         double (&a)[3])
{
    double f, gx, gy;
    drag_factor_fast(G, decr, mstar, dsn_to_double(dsn(H.x, L.x)), dsn_to_double(dsn(H.y, L.y)),
                     dsn_to_double(dsn(H.z, L.z)), v[0], v[1], v[2], cd, radius, density, f, gx, gy);
    a[0] = fma(f, gx - v[0], a[0]);
    a[1] = fma(f, gy - v[1], a[1]);
    a[2] = fma(f, -v[2], a[2]);
}

// row_sum of N components, each a chain of its own.
template <int N>
__device__ __forceinline__ void stage_sums(const NyTableau& T, int row, const double* k, int st, double (&out)[N])
{
#pragma unroll
    for (int c = 0; c < N; c++) out[c] = 0.0;
    const int u1 = T.beg[row + 1];
#pragma unroll 2
    for (int u = T.beg[row]; u < u1; u++) {
        const double a = T.term[u].a;
        const double* x = k + T.term[u].q * st;
#pragma unroll
        for (int c = 0; c < N; c++) out[c] = fma(a, x[c], out[c]);
    }
}

struct OwnerSmem {   // of the CTA that owns a large body
    float4 hi[kTryMaxLarge], lo[kTryMaxLarge];
    float2 red[2][kTryMaxOwners / 32 - 1][3];
    double k[kMaxStages][3];
    unsigned long long err;
    DevSys sys;   // CTA 0's copy of the system record
};

// The group of threads that owns large body k: per stage the sum of the
// CTAs' partials, the pairs of the large bodies and the stars' terms, then the
// body's position two stages on for everyone; at the end its solution.  CTA 0's
// group decides over the try.  All warps but the last gather the partials; the
// last one meanwhile forms what does not need them, and then the position.
template <int MODE>
__device__ __forceinline__ void run_owner(const TryParams& P, OwnerSmem& sm, const NyTableau& T, volatile int* dead,
                                          unsigned tag0, double dt, const double* ly, const double* lv, int o)
{
    const int k = blockIdx.x, nl = P.n_large;
    const int lane = o & 31, w = o >> 5, W = P.owners, GW = W / 32 - 1;   // warps that gather
    DevSys* S = P.sys;
    if (w < GW) {
        for (int s = 0; s < P.n_stage; s++) {
            Ds3 a{0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            for (int j = o; j < P.n_cta; j += 32 * GW) {
                const uint4* rec = P.part + ((size_t)((s & 1) * nl + k) * P.n_cta + j) * 2;
                const uint4 p = poll16(rec, tag0 + 1 + s, S, dead), q = poll16(rec + 1, tag0 + 1 + s, S, dead);
                ds_merge(a.xh, a.xl, __uint_as_float(p.x), __uint_as_float(p.y));
                ds_merge(a.yh, a.yl, __uint_as_float(p.z), __uint_as_float(q.x));
                ds_merge(a.zh, a.zl, __uint_as_float(q.y), __uint_as_float(q.z));
            }
            const float2 part = reduce_scatter(a, lane, 32);
            if (lane < 3) sm.red[s & 1][w][lane] = part;
            if (k == 0 && (s == 2 || s == 3) && P.head_n > 0) __threadfence();
            group_sync(2, W);   // two sets of `red`: the last warp reads one while the next is formed
        }
    }
    const int body = P.off + k;
    const int comp = min(lane, 2);
    const double y = ly[3 * k + comp], v = lv[3 * k + comp];
    if (w == GW) {
        const bool live = P.id[body] > 0;
        float mj[2];   // the masses of large bodies lane and lane + 32
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int j = lane + 32 * u;
            mj[u] = j < nl && P.id[P.off + j] >= 0 ? __double2float_rn(P.mass[P.off + j]) : 0.f;
        }
        float2 ms = make_float2(0.f, 0.f);
        if (lane < P.n_star) {
            const double m = P.id[P.off + lane] < 0 ? 0.0 : P.mass[P.off + lane];
            ms.x = __double2float_rn(m);
            ms.y = __double2float_rn(m - (double)ms.x);
        }
        if (lane == 0) sm.err = 0ull;
        for (int s = 0; s < P.n_stage; s++) {
            if (s < 2) {
                for (int e = lane; e < 3 * nl; e += 32)
                    put_comp(sm.hi, sm.lo, e / 3, e % 3, s == 0 ? ly[e] : fma(T.c[1] * dt, lv[e], ly[e]));
            } else {
                for (int e = lane; e < 2 * nl; e += 32) {
                    const uint4 q = poll16(pos_records(P, s) + e, tag0 + 1 + s, S, dead);
                    float* f = reinterpret_cast<float*>((e & 1 ? sm.lo : sm.hi) + (e >> 1));
                    f[0] = __uint_as_float(q.x);
                    f[1] = __uint_as_float(q.y);
                    f[2] = __uint_as_float(q.z);
                }
            }
            __syncwarp();
            const float4 H = sm.hi[k], L = sm.lo[k];
            Ds3 a{0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const int j = lane + 32 * u;
                if (j >= P.n_star && j < nl && j != k) {
                    float4 h = sm.hi[j];
                    h.w = mj[u];
                    float px = 0.f, py = 0.f, pz = 0.f;
                    pair_term<MODE>(h, sm.lo[j], H, L, px, py, pz);
                    fold(a, px, py, pz);
                }
            }
            if (lane < P.n_star && lane != k) {
                float2 ax = make_float2(0.f, 0.f), ay = ax, az = ax;
                star_term(sm.hi[lane], sm.lo[lane], ms, H, L, ax, ay, az);
                ds_merge(a.xh, a.xl, ax.x, ax.y);
                ds_merge(a.yh, a.yl, ay.x, ay.y);
                ds_merge(a.zh, a.zl, az.x, az.y);
            }
            float2 g0 = reduce_scatter(a, lane, 32);
            g0 = make_float2(__shfl_sync(0xffffffffu, g0.x, comp), __shfl_sync(0xffffffffu, g0.y, comp));
            // the position of stage s + 2 but for the term of K_s, its row's last one if present
            const bool more = s + 2 < P.n_stage;
            double base = 0.0, coef = 0.0;
            if (more) {
                const int u0 = T.beg[s + 2];
                int u1 = T.beg[s + 3];
                if (u1 > u0 && T.term[u1 - 1].q == s) coef = dt * dt * T.term[--u1].a;
                base = fma(dt * dt, row_sum(T, u0, u1, &sm.k[0][comp], 3), fma(T.c[s + 2] * dt, v, y));
            }
            group_sync(2, W);
            const float2(*red)[3] = sm.red[s & 1];
            float2 g = dsn_add(red[0][comp], g0);
            if (GW > 2) g = dsn_add(g, dsn_add(red[1][comp], red[2][comp]));
            else if (GW > 1) g = dsn_add(g, red[1][comp]);
            if (GW > 4) g = dsn_add(g, dsn_add(red[3][comp], red[4][comp]));
            else if (GW > 3) g = dsn_add(g, red[3][comp]);
            const double a_k = live ? dsn_to_double(g) : 0.0;
            if (more) {
                float2 x;
                split_ds(fma(coef, a_k, base), x.x, x.y);
                const float h1 = __shfl_sync(0xffffffffu, x.x, 1), h2 = __shfl_sync(0xffffffffu, x.x, 2);
                const float l0 = __shfl_sync(0xffffffffu, x.y, 0), l2 = __shfl_sync(0xffffffffu, x.y, 2);
                const float h0 = __shfl_sync(0xffffffffu, x.x, 0), l1 = __shfl_sync(0xffffffffu, x.y, 1);
                if (lane < 2 * kTryCopies) {   // lanes 2 c, 2 c + 1: the two words of copy c
                    uint4* rec = P.pos + ((size_t)(((s + 2) & 3) * kTryCopies + (lane >> 1)) * nl + k) * 2 + (lane & 1);
                    st_rec16(rec, __float_as_uint(lane & 1 ? l0 : h0), __float_as_uint(lane & 1 ? l1 : h1),
                             __float_as_uint(lane & 1 ? l2 : h2), tag_of(tag0 + 3 + s, dead));
                }
            }
            if (lane < 3) sm.k[s][lane] = a_k;
            __syncwarp();
        }
    }
    // the solution, the error, the decision: the last warp; CTA 0's others gather the errors
    if (w == GW) {
        unsigned long long eb = 0ull;
        if (P.adaptive) {
            eb = component_error(T, P.scheme, dt, &sm.k[0][comp], 3);
            const unsigned long long e1 = __shfl_sync(0xffffffffu, eb, 1), e2 = __shfl_sync(0xffffffffu, eb, 2);
            eb = max(eb, max(e1, e2));
        }
        if (lane == 0) st_pair(P.err + P.n_cta + k, (unsigned)eb, (unsigned)(eb >> 32), tag_of(tag0 + 14, dead));
    }
    if (k == 0) {
        if (w < GW) {
            // in fixed steps the owners' records alone: the last partial sums told of the CTAs
            unsigned long long m = 0ull;
            for (int j = (P.adaptive ? 0 : P.n_cta) + o; j < P.n_cta + nl; j += 32 * GW) {
                const uint2 q = poll_pair(P.err + j, tag0 + 14, S, dead);
                m = max(m, ((unsigned long long)q.y << 32) | q.x);
            }
            atomicMax(&sm.err, m);
        }
        group_sync(2, W);
        if (w == 0 && lane == 0) {
            // accepted or not: control_system's test, before the rest of the step control
            const double max_err = fabs(P.ctl.lambda * dt * __longlong_as_double((long long)sm.err));
            const bool heard = !*dead;
            const bool take = heard && (!P.adaptive || max_err <= P.ctl.tolerance);
            st_pair(P.decision, take ? 1u : 0u, 0u, tag_of(tag0 + 15, dead));
            if (heard) {
                control_of(P.ctl, sm.sys, P.adaptive ? sm.err : 0ull);
                store_control(S, sm.sys);
            } else {
                S->accepted = 0;
            }
            *P.epoch = tag0 / 16 + 1;
        }
    }
    if (w != GW) return;
    double rn = y, vn = v;
    solution(T, dt, &sm.k[0][comp], 3, rn, vn);
    unsigned take = 0u;
    if (lane == 0) take = poll_pair(P.decision, tag0 + 15, S, dead).x;
    take = __shfl_sync(0xffffffffu, take, 0);
    if (lane < 3 && take == 1u) {
        P.y_r[3 * body + lane] = rn;
        P.y_v[3 * body + lane] = vn;
        if (not_finite(rn) || not_finite(vn)) set_status(S, 5);   // RED_ERR_NONFINITE
        write_pos_c(P.pos_hi, P.pos_lo, body, lane, rn);
    }
}

}  // namespace

// The pull of the small bodies bhi / blo [0, pad) on large body k: the sum over
// the 1 << lg threads of a group.  pull_large: a record of this CTA's sums at
// stage s for each large body, by the threads t.  The exchange waits for these
// records.
template <int MODE>
__device__ __forceinline__ float2 large_sum(int lane, int lg, int k, int pad, const float4* bhi, const float4* blo,
                                            const float4* si_hi, const float4* si_lo)
{
    const int LS = 1 << lg;
    const float4 H = si_hi[k], L = si_lo[k];
    Ds3 a{0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int j0 = lane; j0 < pad; j0 += 16 << lg) {
        float x = 0.f, y = 0.f, z = 0.f;
        const int j1 = min(pad, j0 + (16 << lg));
#pragma unroll 4
        for (int j = j0; j < j1; j += LS) pair_term<MODE>(bhi[j], blo[j], H, L, x, y, z);
        fold(a, x, y, z);
    }
    return reduce_scatter(a, lane, LS);   // x, y, z in lanes 0, 1, 2
}
template <int MODE>
__device__ __forceinline__ void pull_large(const TryParams& P, int s, int t, int pad, const float4* bhi,
                                           const float4* blo, const float4* si_hi, const float4* si_lo, unsigned tag)
{
    const int nl = P.n_large, lg = P.lanes_log2;
    if ((t & ~31) >> lg >= nl) return;   // uniform over the warp
    const int lane = t & ((1 << lg) - 1), g = t >> lg, k = min(g, nl - 1);
    const float2 part = large_sum<MODE>(lane, lg, k, pad, bhi, blo, si_hi, si_lo);
    const int l0 = (t & 31) - lane;
    const float yh = __shfl_sync(0xffffffffu, part.x, l0 + 1), yl = __shfl_sync(0xffffffffu, part.y, l0 + 1);
    const float zh = __shfl_sync(0xffffffffu, part.x, l0 + 2), zl = __shfl_sync(0xffffffffu, part.y, l0 + 2);
    if (lane < 2 && g < nl) {
        uint4* rec = P.part + (((size_t)(s & 1) * nl + k) * P.n_cta + blockIdx.x) * 2;
        if (lane == 0) st_rec16(rec, __float_as_uint(part.x), __float_as_uint(part.y), __float_as_uint(yh), tag);
        else st_rec16(rec + 1, __float_as_uint(yl), __float_as_uint(zh), __float_as_uint(zl), tag);
    }
}

// The accelerations of small bodies b, ... by the large ones, share p of them:
// part 0 the stars, the others (or part 0 too, if it is alone) a share of the
// protoplanets each.  FP32 sums of two terms go into double-single ones, as long as
// the stage kernel's for 16 protoplanets: with eight terms the median error of the
// accelerations was 5 % (16 protoplanets) and 10 % (eight, k_team) above the stage
// kernel's, with two it is 0 to 7 % below, for 1 % of the ensemble's time.
constexpr int kSmallRun = 2;
template <int MODE>
__device__ __forceinline__ void pull_small(int nl, int n_star, int step0, int p, int b, int cnt, int pad, int np,
                                           const float4* bhi, const float4* blo, const float4* si_hi,
                                           const float4* si_lo, const float2* star_m, float2* parts)
{
    if (p >= np) return;
    for (; b < cnt; b += np > 1 ? pad : step0) {
        const float4 H = bhi[b], L = blo[b];
        float2 ax = make_float2(0.f, 0.f), ay = ax, az = ax;
        if (p > 0 || np == 1) {
            const int step = np > 1 ? np - 1 : 1;
            Ds3 a{0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            for (int k0 = n_star + (np > 1 ? p - 1 : 0); k0 < nl; k0 += kSmallRun * step) {
                float x = 0.f, y = 0.f, z = 0.f;
                const int k1 = min(nl, k0 + kSmallRun * step);
#pragma unroll
                for (int k = k0; k < k1; k += step) pair_term<MODE>(si_hi[k], si_lo[k], H, L, x, y, z);
                fold(a, x, y, z);
            }
            ax = dsn_norm(a.xh, a.xl);
            ay = dsn_norm(a.yh, a.yl);
            az = dsn_norm(a.zh, a.zl);
        }
        if (p == 0)
            for (int k = 0; k < n_star; k++) star_term(si_hi[k], si_lo[k], star_m[k], H, L, ax, ay, az);
        float2* o = parts + 3 * (p * pad + b);
        o[0] = ax;
        o[1] = ay;
        o[2] = az;
    }
}

template <int MODE, bool DRAG>
__global__ void __launch_bounds__(try_max_threads(DRAG)) k_try(const __grid_constant__ TryParams P)
{
    __shared__ float4 si_hi[2][kTryMaxLarge], si_lo[2][kTryMaxLarge];
    __shared__ float2 star_m[kTryMaxStars];
    __shared__ double ly[3 * kTryMaxLarge], lv[3 * kTryMaxLarge];   // the large bodies' state at the start of the try
    __shared__ NyTableau T;
    __shared__ OwnerSmem own;
    __shared__ unsigned long long err_sm;
    __shared__ int dead, take;
    __shared__ struct { double dt, t; unsigned tag; int runs; } start;
    extern __shared__ __align__(16) unsigned char dyn[];

    const int t = threadIdx.x;
    const int nl = P.n_large, ns = P.n_stage, nb = P.nb;
    const int main = P.pull + P.bodies;
    DevSys* S = P.sys;
    const int b0 = nl + blockIdx.x * nb;
    const int cnt = max(0, min(P.n - b0, nb));
    const int first = P.off + b0;
    const int pad = try_pad(nb), np = try_parts(nb, P.pull);
    // 16-byte records first: the doubles' count may be odd
    float4* bhi = reinterpret_cast<float4*>(dyn);            // [2][pad], by stage parity
    float4* blo = bhi + 2 * pad;
    float2* parts = reinterpret_cast<float2*>(blo + 2 * pad);   // [2][np][pad][3]
    const int n3 = 3 * nb;
    double* ks = reinterpret_cast<double*>(parts + (size_t)2 * np * 3 * pad);   // accelerations, [stage][nb][3]
    double* yr = ks + (size_t)ns * n3;                          // [nb][3]
    double* yv = yr + n3;

    // ---- everything the try starts from, read before this CTA's first record, so
    // before any CTA writes the solution ----
    if (t >= P.pull && t < main) {
        for (int b = t - P.pull; b < pad; b += P.bodies) {   // a thread per body here
            float4 H = make_float4(1.0e9f, 0.f, 0.f, 0.f), L = make_float4(0.f, 0.f, 0.f, 0.f);   // no body: no mass
            if (b < cnt) {
                const int i = first + b;
                const int id = P.id[i];
                const double m = P.mass[i];
                double y[3], v[3];
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    y[c] = P.y_r[3 * i + c];
                    v[c] = P.y_v[3 * i + c];
                }
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    yr[3 * b + c] = y[c];
                    yv[3 * b + c] = v[c];
                }
                split_ds(y[0], H.x, L.x);
                split_ds(y[1], H.y, L.y);
                split_ds(y[2], H.z, L.z);
                H.w = id >= 0 ? __double2float_rn(m) : 0.f;
                L.w = id > 0 ? 1.f : 0.f;   // an inactive sink's gravity is zero
            }
            bhi[b] = H;
            blo[b] = L;
            bhi[pad + b] = H;
            blo[pad + b] = L;
        }
    } else if (t < 3 * nl) {   // 3 n_large <= pull
        const double y = P.y_r[3 * P.off + t], v = P.y_v[3 * P.off + t];
        const int id = P.id[P.off + t / 3];
        const double m = P.mass[P.off + t / 3];
        ly[t] = y;
        lv[t] = v;
        float h, l;
        split_ds(y, h, l);
        reinterpret_cast<float*>(&si_hi[0][t / 3])[t % 3] = h;
        reinterpret_cast<float*>(&si_lo[0][t / 3])[t % 3] = l;
        if (t % 3 == 0) {
            const double me = id >= 0 ? m : 0.0;
            const float mh = __double2float_rn(me);
            si_hi[0][t / 3].w = si_hi[1][t / 3].w = mh;
            if (t / 3 < P.n_star) star_m[t / 3] = make_float2(mh, __double2float_rn(me - (double)mh));
        }
    } else if (t >= main) {
        const int o = t - main;
        const uint4* src = reinterpret_cast<const uint4*>(P.tab);
        for (int k = o; k < (int)(sizeof(NyTableau) / 16); k += P.owners) reinterpret_cast<uint4*>(&T)[k] = src[k];
        if (blockIdx.x == 0)
            for (int k = o; k < (int)(sizeof(DevSys) / 4); k += P.owners)
                reinterpret_cast<unsigned*>(&own.sys)[k] = reinterpret_cast<const volatile unsigned*>(S)[k];
        if (o == 0) {   // one thread of a CTA: every thread's reads would queue up on these sectors for ~4 us
            const volatile DevSys* V = S;
            const double dt = V->dt_try, ts = V->t;
            const unsigned ep = *(volatile unsigned*)P.epoch;
            start.runs = V->active && !V->halted && V->quota != 0;
            start.dt = dt;
            start.t = ts;
            start.tag = try_tag(ep);
            dead = 0;
            err_sm = 0ull;
        }
    }
    __syncthreads();
    if (!start.runs) {   // uniform over the grid
        if (blockIdx.x == 0 && t == 0) S->accepted = 0;
        return;
    }
    const double dt = start.dt, tsys = start.t;
    const unsigned tag0 = start.tag;
    if (t < P.pull)   // the pull group fences this before its second record
        for (long long k = (long long)blockIdx.x * P.pull + t; k < P.head_n; k += (long long)gridDim.x * P.pull)
            P.head[k] = -1;
    if (t >= main) {
        if ((int)blockIdx.x < nl) run_owner<MODE>(P, own, T, &dead, tag0, dt, ly, lv, t - main);
        return;
    }
    if (t < P.pull) {
        const int share = np > 1 ? t / pad : 0, body = np > 1 ? t % pad : t;
        for (int s = 0; s < ns; s++) {
            const int q = s & 1;
            pull_large<MODE>(P, s, t, pad, bhi + q * pad, blo + q * pad, si_hi[q], si_lo[q],
                             tag_of(tag0 + 1 + s, &dead));
            pull_small<MODE>(nl, P.n_star, P.pull, share, body, cnt, pad, np, bhi + q * pad, blo + q * pad, si_hi[q], si_lo[q], star_m,
                             parts + (size_t)q * np * 3 * pad);
            if (s == 1 && P.head_n > 0) __threadfence();   // the cleared hash before the later records
            group_sync(1, main);
        }
        return;
    }

    // ---- the body group: K of the previous stage, positions of the next ----
    constexpr int N = DRAG ? 3 : 1;   // components of a thread; its item x: component x % 3 of body x / 3, or body x
    const int tb = t - P.pull, items = DRAG ? cnt : 3 * cnt;
    GridInfo grid{};
    if (P.head) grid = *P.grid;
    const double mstar = DRAG ? P.mass[P.off] : 0.0;
    for (int s = 0; s <= ns; s++) {
        if (DRAG && s < ns)
            pull_large<MODE>(P, s, t, pad, bhi + (s & 1) * pad, blo + (s & 1) * pad, si_hi[s & 1], si_lo[s & 1],
                             tag_of(tag0 + 1 + s, &dead));
        double decr = 0.0;
        if (DRAG && s > 0) decr = gas_reduction_factor<false>(P.gas, tsys + stage_c(P.scheme, s - 1) * dt);
        for (int x = tb; x < items; x += P.bodies) {
            const int b = DRAG ? x : x / 3, e = N * x;
            double* k = ks + e;
            if (s > 0) {
                const int q = (s - 1) & 1;
                const float2* pt = parts + (size_t)q * np * 3 * pad + e;
                const bool live = blo[b].w != 0.f;
                double g[N];
#pragma unroll
                for (int c = 0; c < N; c++) {
                    float2 a = pt[c];
                    for (int u = 1; u < np; u++) a = dsn_add(a, pt[3 * u * pad + c]);
                    g[c] = live ? dsn_to_double(a) : 0.0;
                }
                if constexpr (DRAG) {
                    if (!(1.0e-6 > decr)) {
                        double v[3];
                        stage_sums(T, kTryRowV + s - 1, k, n3, v);
#pragma unroll
                        for (int c = 0; c < 3; c++) v[c] = fma(dt, v[c], yv[e + c]);
                        const int i = first + b;
                        gas_drag(P.gas, decr, mstar, bhi[q * pad + b], blo[q * pad + b], v, P.cd[i], P.radius[i],
                                 P.density[i], g);
                    }
                }
#pragma unroll
                for (int c = 0; c < N; c++) k[(size_t)(s - 1) * n3 + c] = g[c];
            }
            if (s + 1 < ns) {
                const int q = (s + 1) & 1;
                double r[N];
                stage_sums(T, s + 1, k, n3, r);
                const double cdt = T.c[s + 1] * dt, dt2 = dt * dt;
#pragma unroll
                for (int c = 0; c < N; c++)
                    put_comp(bhi + q * pad, blo + q * pad, b, DRAG ? c : x % 3,
                             fma(dt2, r[c], fma(cdt, yv[e + c], yr[e + c])));
            }
        }
        if (s == ns) break;
        if (s == 0) {   // the large bodies' positions of stage 1
            if (ns > 1)
                for (int e = tb; e < 3 * nl; e += P.bodies)
                    put_comp(si_hi[1], si_lo[1], e / 3, e % 3, fma(T.c[1] * dt, lv[e], ly[e]));
        } else if (s + 1 < ns) {
            const int q = (s + 1) & 1;
            for (int e = tb; e < 2 * nl; e += P.bodies) {
                const uint4 v = poll16(pos_records(P, s + 1) + e, tag0 + 2 + s, S, &dead);
                float* f = reinterpret_cast<float*>((e & 1 ? si_lo[q] : si_hi[q]) + (e >> 1));
                f[0] = __uint_as_float(v.x);
                f[1] = __uint_as_float(v.y);
                f[2] = __uint_as_float(v.z);
            }
        }
        if (DRAG && s == 1 && P.head_n > 0) __threadfence();   // these threads write partial sums too
        group_sync(1, main);
    }

    // ---- the error, the solution (formed while the decision is on its way) ----
    if (P.adaptive) {
        unsigned long long eb = 0ull;
        for (int x = tb; x < items; x += P.bodies)   // the threads that formed the accelerations
#pragma unroll
            for (int c = 0; c < N; c++) eb = max(eb, component_error(T, P.scheme, dt, ks + N * x + c, n3));
        for (int m = 16; m > 0; m >>= 1) eb = max(eb, __shfl_xor_sync(0xffffffffu, eb, m));
        if ((tb & 31) == 0) atomicMax(&err_sm, eb);
        group_sync(3, P.bodies);
        if (tb == 0)
            st_pair(P.err + blockIdx.x, (unsigned)err_sm, (unsigned)(err_sm >> 32), tag_of(tag0 + 14, &dead));
    }
    for (int x = tb; x < items; x += P.bodies)
#pragma unroll
        for (int c = 0; c < N; c++) solution(T, dt, ks + N * x + c, n3, yr[N * x + c], yv[N * x + c]);
    if (tb == 0) {
        take = poll_pair(P.decision, tag0 + 15, S, &dead).x == 1u;
        if (P.head_n > 0) __threadfence();
    }
    group_sync(3, P.bodies);
    if (!take) return;
    int* cell = reinterpret_cast<int*>(parts);   // the pull group has left it
    bool bad = false;
    for (int e = tb; e < 3 * cnt; e += P.bodies) {
        const double r = yr[e], v = yv[e];
        P.y_r[3 * first + e] = r;
        P.y_v[3 * first + e] = v;
        bad = bad || not_finite(r) || not_finite(v);
        write_pos_c(P.pos_hi, P.pos_lo, first + e / 3, e % 3, r);
        if (grid.enabled) cell[e] = cell_coord(r, grid.inv_h);
    }
    if (bad) set_status(S, 5);   // RED_ERR_NONFINITE
    if (!grid.enabled) return;   // uniform
    group_sync(3, P.bodies);
    for (int b = tb; b < cnt; b += P.bodies) {
        const int4 cl = make_int4(cell[3 * b], cell[3 * b + 1], cell[3 * b + 2], 0);
        P.cell[first + b] = cl;
        P.next[first + b] = atomicExch(&P.head[grid.toff + bucket_of(cl.x, cl.y, cl.z, grid.mask)], first + b);
    }
}

// ---------------------------------------------------------------------------
// k_team
// ---------------------------------------------------------------------------
namespace {

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;\n" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;\n" ::: "memory"); }
__device__ __forceinline__ void cluster_sync()
{
    cluster_arrive();
    cluster_wait();
}
// Another CTA's copy of a shared-memory word.
__device__ __forceinline__ unsigned peer(const void* local, int rank)
{
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n"
                 : "=r"(r)
                 : "r"((unsigned)__cvta_generic_to_shared(local)), "r"(rank));
    return r;
}
__device__ __forceinline__ void st_peer(unsigned a, float2 v)
{
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};\n" ::"r"(a), "f"(v.x), "f"(v.y) : "memory");
}
__device__ __forceinline__ void st_peer(unsigned a, float v)
{
    asm volatile("st.shared::cluster.f32 [%0], %1;\n" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void st_peer(unsigned a, unsigned long long v)
{
    asm volatile("st.shared::cluster.b64 [%0], %1;\n" ::"r"(a), "l"(v) : "memory");
}

// row_sum and component_error of a pair of components.
__device__ __forceinline__ double2 pair_sums(const NyTableau& T, int row, const double2* k, int st)
{
    double2 r = make_double2(0.0, 0.0);
    const int u1 = T.beg[row + 1];
#pragma unroll 4
    for (int u = T.beg[row]; u < u1; u++) {
        const double a = T.term[u].a;
        const double2 x = k[T.term[u].q * st];
        r.x = fma(a, x.x, r.x);
        r.y = fma(a, x.y, r.y);
    }
    return r;
}
__device__ __forceinline__ unsigned long long pair_error(const NyTableau& T, int scheme, double dt, const double2* k,
                                                         int st, bool both)
{
    const double2 r = pair_sums(T, kTryRowER, k, st);
    double2 d;
    if (scheme == SCHEME_RKF78) {
        const double2 a = k[0], b = k[10 * st], c = k[11 * st], e = k[12 * st];
        d = make_double2(((a.x + b.x) - c.x) - e.x, ((a.y + b.y) - c.y) - e.y);
    } else {
        const double2 a = k[3 * st], b = k[4 * st];
        d = make_double2(a.x - b.x, a.y - b.y);
    }
    const unsigned long long m = error_bits(dt * r.x, d.x);
    return both ? max(m, error_bits(dt * r.y, d.y)) : m;
}

struct TeamSmem {
    float4 si_hi[3][kTeamLarge], si_lo[3][kTeamLarge];   // the large bodies, by stage mod 3
    float2 star_m[kTryMaxStars];
    float mass[kTeamLarge];
    double ly[3 * kTeamLarge], lv[3 * kTeamLarge];
    NyTableau T;
    float2 part[2][2 * (kTeamLarge + kTeamSize)][3];   // partials of the bodies owned here: stage parity; slot, rank, half
    double k[kTeamLarge][kMaxStages][3];         // their accelerations
    unsigned long long err, all, errs[kTeamSize];     // this CTA's error; the team's; its CTAs', in the first of them
    DevSys sys;
    int live[kTeamLarge];
    double dt;
    int runs;
};

}  // namespace

template <int MODE>
__global__ void __launch_bounds__(kTeamPull + kTeamBody + kTeamOwners, 1) k_team(const __grid_constant__ TeamParams P)
{
    __shared__ TeamSmem sm;
    extern __shared__ __align__(16) unsigned char dyn[];
    const int t = threadIdx.x;
    const TeamItem it = P.items[blockIdx.x];
    const int ns = P.n_stage;
    pdl_wait();
    pdl_trigger();
    if (t == 0) {
        int runs = 0;
        double dt = 0.0;
        if (it.sys >= 0) {
            const volatile DevSys* V = P.sys + it.sys;
            dt = V->dt_try;
            runs = V->active && !V->halted && V->quota != 0;
        }
        sm.dt = dt;
        sm.runs = runs;
        sm.err = 0ull;
    }
    __syncthreads();
    if (!sm.runs) {   // uniform over the team; the cluster's barriers still count this CTA
        if (it.sys >= 0 && it.rank == 0 && t == 0) P.sys[it.sys].accepted = 0;
        for (int k = 0; k < ns + 3; k++) cluster_sync();
        return;
    }
    const double dt = sm.dt;
    DevSys* S = P.sys + it.sys;
    const SysInfo si = P.sinfo[it.sys];
    const int nl = si.n_SI, n_star = si.n_star, small = si.n - nl;
    const int nb = team_bodies(small, it.size);
    const int b0 = nl + it.rank * nb;
    const int cnt = max(0, min(si.n - b0, nb));
    const int first = si.off + b0;
    const int pad = try_pad(nb), np = 3 * nb / 2;   // components in pairs: nb is even
    float4* bhi = reinterpret_cast<float4*>(dyn);               // [2][pad], by stage parity
    float4* blo = bhi + 2 * pad;
    float2* parts = reinterpret_cast<float2*>(blo + 2 * pad);   // [2][pad][3]
    double2* ks = reinterpret_cast<double2*>(parts + (size_t)2 * 3 * pad);   // [stage][pair]

    // ---- load ----
    for (int b = t; b < pad; b += blockDim.x) {
        float4 H = make_float4(1.0e9f, 0.f, 0.f, 0.f), L = make_float4(0.f, 0.f, 0.f, 0.f);   // no body: no mass
        if (b < cnt) {
            const int i = first + b;
            const int id = P.id[i];
            const double m = P.mass[i];
            split_ds(P.y_r[3 * i], H.x, L.x);
            split_ds(P.y_r[3 * i + 1], H.y, L.y);
            split_ds(P.y_r[3 * i + 2], H.z, L.z);
            H.w = id >= 0 ? __double2float_rn(m) : 0.f;
            L.w = id > 0 ? 1.f : 0.f;   // an inactive sink's gravity is zero
        }
        bhi[b] = H;
        blo[b] = L;
        bhi[pad + b] = H;
        blo[pad + b] = L;
    }
    for (int k = t; k < (int)(sizeof(NyTableau) / 16); k += blockDim.x)
        reinterpret_cast<uint4*>(&sm.T)[k] = reinterpret_cast<const uint4*>(P.tab)[k];
    if (t < 3 * nl) {
        sm.ly[t] = P.y_r[3 * si.off + t];
        sm.lv[t] = P.y_v[3 * si.off + t];
        put_comp(sm.si_hi[0], sm.si_lo[0], t / 3, t % 3, sm.ly[t]);
    }
    if (t < nl) {
        const int id = P.id[si.off + t];
        const double m = id >= 0 ? P.mass[si.off + t] : 0.0;
        const float mh = __double2float_rn(m);
        sm.mass[t] = mh;
        sm.live[t] = id > 0;
        for (int q = 0; q < 3; q++) sm.si_hi[q][t].w = mh;
        if (t < n_star) sm.star_m[t] = make_float2(mh, __double2float_rn(m - (double)mh));
    }
    if (it.rank == 0)
        for (int k = t; k < (int)(sizeof(DevSys) / 4); k += blockDim.x)
            reinterpret_cast<unsigned*>(&sm.sys)[k] = reinterpret_cast<const volatile unsigned*>(S)[k];
    GridInfo grid{};
    if (P.head) {
        grid = P.grid[it.sys];
        if (grid.enabled)   // this team's bodies alone go there; inserted after the barriers below
            for (int k = it.rank * (int)blockDim.x + t; k <= grid.mask; k += it.size * (int)blockDim.x)
                P.head[grid.toff + k] = -1;
    }
    const NyTableau& T = sm.T;
    const double dt2 = dt * dt;
    cluster_sync();

    const bool puller = t < kTeamPull, owner = t >= kTeamPull + kTeamBody;
    const int tb = t - kTeamPull;
    const int lane = t & 31, ow = (t - kTeamPull - kTeamBody) >> 5;
    const int comp = min(lane, 2);
    const int mid = pad / 64 * 32;   // large_sum's halves

    // pairs of components of the body group; the error and the solution follow the same split
    const int pairs = (3 * cnt + 1) / 2;
    const int share = min(pairs, kTeamRounds * kTeamBody);
    const int x0 = puller ? share + t : tb, x1 = puller ? pairs : share, xs = puller ? kTeamPull : kTeamBody;
    // phase s: pair terms of stage s, K of stage s - 1, positions of stage s + 1
    for (int s = 0; s <= ns; s++) {
        const int q = s & 1, c3 = s % 3;
        if (s < ns && !owner) {
            // a warp per large body and half of the small ones
            for (int g = t >> 5; g < 2 * nl; g += (kTeamPull + kTeamBody) / 32) {
                const int k = g >> 1, half = g & 1, j0 = half ? mid : 0, j1 = half ? pad : mid;
                const float2 v = large_sum<MODE>(lane, 5, k, j1 - j0, bhi + q * pad + j0, blo + q * pad + j0,
                                                 sm.si_hi[c3], sm.si_lo[c3]);
                if (lane < 3)
                    st_peer(peer(&sm.part[q][((k / it.size) * it.size + it.rank) * 2 + half][lane],
                                 it.base + k % it.size), v);
            }
        }
        if (s < ns && puller)
            pull_small<MODE>(nl, n_star, kTeamPull, 0, t, cnt, pad, 1, bhi + q * pad, blo + q * pad, sm.si_hi[c3],
                             sm.si_lo[c3], sm.star_m, parts + (size_t)q * 3 * pad);
        if (!owner) {
            // the body group's pairs first, the pull group takes the rest when it is done
            for (int x = x0; x < x1; x += xs) {
                const int e = 2 * x, b = e / 3, c = e - 3 * b;   // component c of body b, and the next one
                const int b2 = c == 2 ? b + 1 : b, d = c == 2 ? 0 : c + 1;
                const bool both = e + 1 < 3 * cnt;
                double2* k = ks + x;
                if (s > 0) {
                    const float4 g = *reinterpret_cast<const float4*>(parts + (size_t)(q ^ 1) * 3 * pad + e);
                    const float m0 = blo[b].w, m1 = blo[b2].w;   // 1, or 0 for an inactive body
                    k[(size_t)(s - 1) * np] = make_double2(m0 != 0.f ? dsn_to_double(make_float2(g.x, g.y)) : 0.0,
                                                           m1 != 0.f ? dsn_to_double(make_float2(g.z, g.w)) : 0.0);
                }
                if (s + 1 < ns) {
                    const double cdt = T.c[s + 1] * dt;
                    const size_t i = 3 * (size_t)first + e, j = both ? i + 1 : i;
                    const double2 r = pair_sums(T, s + 1, k, np);
                    put_comp(bhi + (q ^ 1) * pad, blo + (q ^ 1) * pad, b, c,
                             fma(dt2, r.x, fma(cdt, P.y_v[i], P.y_r[i])));
                    if (both)
                        put_comp(bhi + (q ^ 1) * pad, blo + (q ^ 1) * pad, b2, d,
                                 fma(dt2, r.y, fma(cdt, P.y_v[j], P.y_r[j])));
                }
            }
            if (s == 0 && ns > 1 && tb >= 0 && tb < 3 * nl)
                put_comp(sm.si_hi[1], sm.si_lo[1], tb / 3, tb % 3, fma(T.c[1] * dt, sm.lv[tb], sm.ly[tb]));
        } else if (s > 0) {
            // a warp per large body owned here: slot u is body u size + rank
            const int p3 = (s - 1) % 3;
            for (int u = ow; u * it.size + it.rank < nl; u += kTeamOwners / 32) {
                const int k = u * it.size + it.rank;
                const float4 H = sm.si_hi[p3][k], L = sm.si_lo[p3][k];
                Ds3 a{0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                if (lane >= n_star && lane < nl && lane != k) {
                    float px = 0.f, py = 0.f, pz = 0.f;
                    pair_term<MODE>(sm.si_hi[p3][lane], sm.si_lo[p3][lane], H, L, px, py, pz);
                    fold(a, px, py, pz);
                }
                if (lane < n_star && lane != k) {
                    float2 ax = make_float2(0.f, 0.f), ay = ax, az = ax;
                    star_term(sm.si_hi[p3][lane], sm.si_lo[p3][lane], sm.star_m[lane], H, L, ax, ay, az);
                    ds_merge(a.xh, a.xl, ax.x, ax.y);
                    ds_merge(a.yh, a.yl, ay.x, ay.y);
                    ds_merge(a.zh, a.zl, az.x, az.y);
                }
                if (lane < 2 * it.size) {
                    const float2* pt = sm.part[q ^ 1][2 * u * it.size + lane];
                    ds_merge(a.xh, a.xl, pt[0].x, pt[0].y);
                    ds_merge(a.yh, a.yl, pt[1].x, pt[1].y);
                    ds_merge(a.zh, a.zl, pt[2].x, pt[2].y);
                }
                const float2 g = reduce_scatter(a, lane, 32);
                if (lane < 3) sm.k[u][s - 1][lane] = sm.live[k] ? dsn_to_double(g) : 0.0;
                __syncwarp();
                if (s + 1 < ns) {
                    float2 x;
                    split_ds(fma(dt2, row_sum(T, s + 1, &sm.k[u][0][comp], 3),
                                 fma(T.c[s + 1] * dt, sm.lv[3 * k + comp], sm.ly[3 * k + comp])),
                             x.x, x.y);
                    if (lane < 3) {
                        const int n3s = (s + 1) % 3;
                        float* h = reinterpret_cast<float*>(&sm.si_hi[n3s][k]) + lane;
                        float* l = reinterpret_cast<float*>(&sm.si_lo[n3s][k]) + lane;
                        for (int c = 0; c < it.size; c++) {
                            st_peer(peer(h, it.base + c), x.x);
                            st_peer(peer(l, it.base + c), x.y);
                        }
                    }
                }
            }
        }
        if (s < ns) cluster_sync();
    }

    // ---- the error of the team, in its first CTA ----
    const int own_n = it.rank < nl ? (nl - it.rank + it.size - 1) / it.size : 0;
    if (P.adaptive) {
        unsigned long long eb = 0ull;
        if (!owner) {
            for (int x = x0; x < x1; x += xs)
                eb = max(eb, pair_error(T, P.scheme, dt, ks + x, np, 2 * x + 1 < 3 * cnt));
        } else if (lane < 3) {
            for (int u = ow; u < own_n; u += kTeamOwners / 32)
                eb = max(eb, component_error(T, P.scheme, dt, &sm.k[u][0][lane], 3));
        }
        for (int m = 16; m > 0; m >>= 1) eb = max(eb, __shfl_xor_sync(0xffffffffu, eb, m));
        if (lane == 0) atomicMax(&sm.err, eb);
    }
    __syncthreads();
    if (t == 0) st_peer(peer(&sm.errs[it.rank], it.base), sm.err);
    cluster_arrive();
    // the solution meanwhile, a pair's positions and velocities, where the stage positions were
    double* sol = reinterpret_cast<double*>(dyn);   // [4][np]
    if (!owner) {
        const double cdt = T.cb * dt;
        for (int x = x0; x < x1; x += xs) {
            const double2 r = pair_sums(T, kTryRowRB, ks + x, np), w = pair_sums(T, kTryRowVB, ks + x, np);
            const size_t i = 3 * (size_t)first + 2 * x, j = 2 * x + 1 < 3 * cnt ? i + 1 : i;
            const double v0 = P.y_v[i], v1 = P.y_v[j];
            double* o = sol + x;
            o[0] = fma(dt2, r.x, fma(cdt, v0, P.y_r[i]));
            o[np] = fma(dt2, r.y, fma(cdt, v1, P.y_r[j]));
            o[2 * np] = fma(dt, w.x, v0);
            o[3 * np] = fma(dt, w.y, v1);
        }
    }
    cluster_wait();
    if (t < 32) {
        unsigned long long e = 0ull;
        if (t < it.size)
            asm volatile("ld.shared::cluster.b64 %0, [%1];\n" : "=l"(e) : "r"(peer(&sm.errs[t], it.base)) : "memory");
        for (int m = kTeamSize / 2; m > 0; m >>= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, m));
        if (t == 0) sm.all = e;
    }
    cluster_sync();   // the errors are read: CTAs may leave from here on
    // control_system's test, the same in every CTA of the team
    const unsigned long long err = sm.all;
    const double max_err = fabs(P.ctl.lambda * dt * __longlong_as_double((long long)err));
    const bool accepted = !P.adaptive || max_err <= P.ctl.tolerance;
    if (it.rank == 0 && t == kTeamPull - 1) {
        control_of(P.ctl, sm.sys, P.adaptive ? err : 0ull);
        store_control(S, sm.sys);
    }
    if (!accepted) return;
    bool bad = false;
    if (!owner) {
        for (int x = x0; x < x1; x += xs) {
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int e = 2 * x + h;
                if (e >= 3 * cnt) break;
                const double y = sol[h * np + x], v = sol[(2 + h) * np + x];
                P.y_r[3 * first + e] = y;
                P.y_v[3 * first + e] = v;
                bad = bad || not_finite(y) || not_finite(v);
                write_pos_c(P.pos_hi, P.pos_lo, first + e / 3, e % 3, y);
                if (grid.enabled) reinterpret_cast<int*>(parts)[e] = cell_coord(y, grid.inv_h);
            }
        }
    } else if (lane < 3) {
        for (int u = ow; u < own_n; u += kTeamOwners / 32) {
            const int k = u * it.size + it.rank, x = 3 * (si.off + k) + lane;
            double y = sm.ly[3 * k + lane], v = sm.lv[3 * k + lane];
            solution(T, dt, &sm.k[u][0][lane], 3, y, v);
            P.y_r[x] = y;
            P.y_v[x] = v;
            bad = bad || not_finite(y) || not_finite(v);
            write_pos_c(P.pos_hi, P.pos_lo, si.off + k, lane, y);
        }
    }
    if (bad) set_status(S, 5);   // RED_ERR_NONFINITE
    if (!grid.enabled) return;   // uniform
    __syncthreads();
    const int* cell = reinterpret_cast<const int*>(parts);
    for (int b = t; b < cnt; b += blockDim.x) {
        const int4 cl = make_int4(cell[3 * b], cell[3 * b + 1], cell[3 * b + 2], 0);
        P.cell[first + b] = cl;
        P.next[first + b] = atomicExch(&P.head[grid.toff + bucket_of(cl.x, cl.y, cl.z, grid.mask)], first + b);
    }
}

namespace {
typedef void (*TryKernel)(const TryParams);
TryKernel try_kernel(int mode, bool drag)
{
    if (mode == MODE_MIXED) return drag ? k_try<MODE_MIXED, true> : k_try<MODE_MIXED, false>;
    if (mode == MODE_FP32) return drag ? k_try<MODE_FP32, true> : k_try<MODE_FP32, false>;
    return nullptr;
}
}  // namespace

int try_ctas_per_sm(int mode, bool drag, int threads, size_t smem)
{
    TryKernel k = try_kernel(mode, drag);
    int dev = 0, most = 0, n = 0;
    if (!k || cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
        return 0;
    cudaFuncAttributes a;
    if (cudaFuncGetAttributes(&a, k) != cudaSuccess || smem + a.sharedSizeBytes > (size_t)most ||
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)a.sharedSizeBytes) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, threads, smem) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

void launch_try(const TryParams& P, int mode, cudaStream_t s)
{
    const bool drag = P.gas.enabled != 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)P.n_cta);
    cfg.blockDim = dim3((unsigned)(P.pull + P.bodies + P.owners));
    cfg.dynamicSmemBytes = try_smem(P.nb, P.n_stage, P.pull);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, try_kernel(mode, drag), P);
}

namespace {
typedef void (*TeamKernel)(const TeamParams);
TeamKernel team_kernel(int mode)
{
    return mode == MODE_MIXED ? k_team<MODE_MIXED> : mode == MODE_FP32 ? k_team<MODE_FP32> : nullptr;
}
}  // namespace

int team_clusters(int mode, int cluster, size_t smem)
{
    TeamKernel k = team_kernel(mode);
    int dev = 0, most = 0, n = 0;
    if (!k || cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
        return 0;
    cudaFuncAttributes a;
    if (cudaFuncGetAttributes(&a, k) != cudaSuccess || smem + a.sharedSizeBytes > (size_t)most ||
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)a.sharedSizeBytes) !=
            cudaSuccess ||
        cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)cluster);
    cfg.blockDim = dim3(kTeamPull + kTeamBody + kTeamOwners);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)cluster;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, k, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

void launch_team(const TeamParams& P, int n_ctas, int mode, cudaStream_t s)
{
    launch_kx(team_kernel(mode), (unsigned)n_ctas, (unsigned)(kTeamPull + kTeamBody + kTeamOwners),
              (unsigned)P.cluster, team_smem(P.cap, P.n_stage), s, P);
}

void set_tableau_try(const Tableau& tb, cudaStream_t s)
{
    cudaMemcpyToSymbolAsync(c_tb, &tb, sizeof(Tableau), 0, cudaMemcpyHostToDevice, s);
}

}  // namespace redgb
