// try64.cu -- k_try64: a whole try of one sparse system in FP64 (try.cuh).
#include "records.cuh"
#include "try.cuh"

namespace redgb {

namespace {

// A barrier of some warps whose lanes need not come together.  (With bar.sync, the
// aligned form, this kernel did not finish; a warp's lanes do come apart here.)
__device__ __forceinline__ void lanes_sync(int id, int threads)
{
    asm volatile("barrier.cta.sync %0, %1;\n" ::"r"(id), "r"(threads) : "memory");
}

__device__ __forceinline__ void st_rec(uint4* p, double v, unsigned tag)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    st_pair(p, (unsigned)b, (unsigned)(b >> 32), tag);
}
__device__ __forceinline__ double poll_rec(const uint4* p, unsigned tag, DevSys* S, volatile int* dead)
{
    const uint2 v = poll_pair(p, tag, S, dead);
    return __longlong_as_double((long long)(((unsigned long long)v.y << 32) | v.x));
}

// 1 / |d|^3 for |d|^2 = x, nothing for coincident bodies: with the FP32 estimate y of
// 1 / sqrt(x) (of the truncated x) and e = 1 - x y^2, |e| < 2^-21, it is y^3 (1 - e)^(-3/2)
// = y^3 (1 + 3/2 e + 15/8 e^2) to 2^-61; y^2 is exact.  Six FP64 instructions, two
// of them rounding at full size.
__device__ __noinline__ double inverse_cube_far(double x)   // x outside FP32's normal range
{
    double ri = rsqrt(x);
    ri = x > 0.0 ? ri : 0.0;
    return ri * ri * ri;
}
__device__ __forceinline__ double inverse_cube(double dx, double dy, double dz)
{
    const double x = fma(dz, dz, fma(dy, dy, dx * dx));
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const int ex = (int)(b >> 52);   // negative x and NaN are above the range
    if (!(ex > 1023 - 126 && ex < 1023 + 127)) return inverse_cube_far(x);
    const float xf = __uint_as_float(((unsigned)(ex - 1023 + 127) << 23) | (unsigned)((b >> 29) & 0x7FFFFFu));
    const double y = f2d_bits(rsqrtf(xf));
    const double w = y * y, e = fma(-x, w, 1.0), y3 = y * w;
    return fma(y3 * e, fma(e, 1.875, 1.5), y3);
}

// The sums of v over the half-warp, of the twelve values four large bodies'
// components: lane l ends with component (l & 2 ? 2 : l & 1) of body
// 2 (l >> 3 & 1) + (l >> 2 & 1).  Every round halves the values a lane carries:
// 12 additions instead of 48.
__device__ __forceinline__ double half_sum12(const double (&v)[12], int lane)
{
    double a[6], b[3];
    const bool h8 = lane & 8, h4 = lane & 4, h2 = lane & 2, h1 = lane & 1;
#pragma unroll
    for (int i = 0; i < 6; i++) a[i] = (h8 ? v[6 + i] : v[i]) + __shfl_xor_sync(0xffffffffu, h8 ? v[i] : v[6 + i], 8);
#pragma unroll
    for (int i = 0; i < 3; i++) b[i] = (h4 ? a[3 + i] : a[i]) + __shfl_xor_sync(0xffffffffu, h4 ? a[i] : a[3 + i], 4);
    // x and y in the lanes without bit 1, z in the others
    const double c0 = (h2 ? b[2] : b[0]) + __shfl_xor_sync(0xffffffffu, h2 ? b[0] : b[2], 2);
    const double c1 = b[1] + __shfl_xor_sync(0xffffffffu, b[1], 2);
    const bool up = h1 && !h2;
    return (up ? c1 : c0) + __shfl_xor_sync(0xffffffffu, h2 || h1 ? c0 : c1, 1);
}
// The same of one body's components, in lanes 0 .. 2 (and again in the lanes from 4, 8, 12).
__device__ __forceinline__ double half_sum3(double x, double y, double z, int lane)
{
    const bool h2 = lane & 2, h1 = lane & 1;
    const double c0 = (h2 ? z : x) + __shfl_xor_sync(0xffffffffu, h2 ? x : z, 2);
    const double c1 = y + __shfl_xor_sync(0xffffffffu, y, 2);
    double r = (h1 && !h2 ? c1 : c0) + __shfl_xor_sync(0xffffffffu, h2 || h1 ? c0 : c1, 1);
    r += __shfl_xor_sync(0xffffffffu, r, 4);
    return r + __shfl_xor_sync(0xffffffffu, r, 8);
}
// The sums of (x, y, z) over the warp in lanes 0, 1, 2.
__device__ __forceinline__ double warp_sum3(double x, double y, double z, int lane)
{
    const bool odd = lane & 1, up = lane & 2;
    double k = (odd ? y : x) + __shfl_xor_sync(0xffffffffu, odd ? x : y, 1);
    z += __shfl_xor_sync(0xffffffffu, z, 1);
    k = (up ? z : k) + __shfl_xor_sync(0xffffffffu, up ? k : z, 2);
#pragma unroll
    for (int m = 4; m < 32; m <<= 1) k += __shfl_xor_sync(0xffffffffu, k, m);
    return k;
}

struct Owner64 {
    double pos[3 * kTryMaxLarge];
    double red[2][kTryMaxOwners / 32 - 1][3];
    double k[kMaxStages][3];
    unsigned long long err;
    DevSys sys;
};

__device__ __forceinline__ const uint4* pos_records64(const TryParams& P, int s)
{
    return P.pos + (size_t)((s & 3) * kTryCopies + blockIdx.x % kTryCopies) * P.n_large * 3;
}

// run_owner (try.cu) in FP64.
__device__ __forceinline__ void run_owner64(const TryParams& P, Owner64& sm, const NyTableau& T, volatile int* dead,
                                            unsigned tag0, double dt, const double* ly, const double* lv, int o)
{
    const int k = blockIdx.x, nl = P.n_large;
    const int lane = o & 31, w = o >> 5, W = P.owners, GW = W / 32 - 1;
    DevSys* S = P.sys;
    if (w < GW) {
        for (int s = 0; s < P.n_stage; s++) {
            double x = 0.0, y = 0.0, z = 0.0;
            for (int j = o; j < P.n_cta; j += 32 * GW) {
                const uint4* rec = P.part + ((size_t)((s & 1) * nl + k) * P.n_cta + j) * 3;
                x += poll_rec(rec, tag0 + 1 + s, S, dead);
                y += poll_rec(rec + 1, tag0 + 1 + s, S, dead);
                z += poll_rec(rec + 2, tag0 + 1 + s, S, dead);
            }
            const double part = warp_sum3(x, y, z, lane);
            if (lane < 3) sm.red[s & 1][w][lane] = part;
            if (k == 0 && (s == 2 || s == 3) && P.head_n > 0) __threadfence();
            lanes_sync(2, W);   // two sets of `red`: the last warp reads one while the next is formed
        }
    }
    const int body = P.off + k;
    const int comp = min(lane, 2);
    const double y = ly[3 * k + comp], v = lv[3 * k + comp];
    if (w == GW) {
        const bool live = P.id[body] > 0;
        double mj[2];
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const int j = lane + 32 * u;
            mj[u] = j < nl && P.id[P.off + j] >= 0 ? P.mass[P.off + j] : 0.0;
        }
        if (lane == 0) sm.err = 0ull;
        for (int s = 0; s < P.n_stage; s++) {
            for (int e = lane; e < 3 * nl; e += 32)
                sm.pos[e] = s == 0 ? ly[e]
                                   : (s == 1 ? fma(T.c[1] * dt, lv[e], ly[e])
                                             : poll_rec(pos_records64(P, s) + e, tag0 + 1 + s, S, dead));
            __syncwarp();
            double ax = 0.0, ay = 0.0, az = 0.0;
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const int j = lane + 32 * u;
                if (j < nl && j != k) {
                    const double dx = sm.pos[3 * j] - sm.pos[3 * k], dy = sm.pos[3 * j + 1] - sm.pos[3 * k + 1],
                                 dz = sm.pos[3 * j + 2] - sm.pos[3 * k + 2];
                    const double f = mj[u] * inverse_cube(dx, dy, dz);
                    ax = fma(f, dx, ax);
                    ay = fma(f, dy, ay);
                    az = fma(f, dz, az);
                }
            }
            double g = __shfl_sync(0xffffffffu, warp_sum3(ax, ay, az, lane), comp);
            // the position of stage s + 2 but for the term of K_s, its row's last one if present
            const bool more = s + 2 < P.n_stage;
            double base = 0.0, sum = 0.0, coef = 0.0;
            if (more) {
                const int u0 = T.beg[s + 2];
                int u1 = T.beg[s + 3];
                if (u1 > u0 && T.term[u1 - 1].q == s) coef = T.term[--u1].a;
                sum = row_sum(T, u0, u1, &sm.k[0][comp], 3);
                base = fma(T.c[s + 2] * dt, v, y);
            }
            __syncwarp();
            lanes_sync(2, W);
            for (int u = 0; u < GW; u++) g += sm.red[s & 1][u][comp];
            if (!live) g = 0.0;
            if (more) {
                const double x = fma(dt * dt, fma(coef, g, sum), base);
                const double px = __shfl_sync(0xffffffffu, x, lane % 3);
                if (lane < 3 * kTryCopies)   // lanes 3 c .. 3 c + 2: copy c
                    st_rec(P.pos + ((size_t)(((s + 2) & 3) * kTryCopies + lane / 3) * nl + k) * 3 + lane % 3, px,
                           tag_of(tag0 + 3 + s, dead));
            }
            if (lane < 3) sm.k[s][lane] = g;
            __syncwarp();
        }
    }
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
        lanes_sync(2, W);
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

__global__ void __launch_bounds__(kTry64Threads, 1) k_try64(const __grid_constant__ TryParams P)
{
    __shared__ double si[2][3 * kTryMaxLarge], si_m[kTryMaxLarge];
    __shared__ double ly[3 * kTryMaxLarge], lv[3 * kTryMaxLarge];   // the large bodies' state at the start of the try
    __shared__ NyTableau T;
    __shared__ Owner64 own;
    __shared__ unsigned long long err_sm;
    __shared__ int dead, take;
    __shared__ struct { double dt; unsigned tag; int runs; } start;
    extern __shared__ __align__(16) unsigned char dyn[];

    const int t = threadIdx.x;
    const int nl = P.n_large, ns = P.n_stage, nb = P.nb;
    const int main = P.pull + P.bodies;
    DevSys* S = P.sys;
    const int b0 = nl + blockIdx.x * nb;
    const int cnt = max(0, min(P.n - b0, nb));
    const int first = P.off + b0;
    const int pad = try64_pad(nb), np = try64_parts(nb), n3 = 3 * nb, bw = pad / 16;
    double* pos = reinterpret_cast<double*>(dyn);       // [2][pad][3], by stage parity
    double* mass = pos + 6 * pad;                       // [pad]: 0 for an inactive source
    double* parts = mass + pad;                         // [2][np][pad][3]
    double* ks = parts + (size_t)6 * np * pad;          // [stage][nb][3]
    double* yr = ks + (size_t)ns * n3;
    double* yv = yr + n3;
    double* wp = yv + n3;                               // [large body][16 small bodies][3]

    if (t >= P.pull && t < main) {
        for (int e = t - P.pull; e < 3 * pad; e += P.bodies) {
            const int b = e / 3;
            double y = e % 3 == 0 ? 1.0e9 : 0.0;        // no body: no mass, far from everything
            if (b < cnt) {
                y = P.y_r[3 * first + e];
                yr[e] = y;
                yv[e] = P.y_v[3 * first + e];
            }
            pos[e] = y;
            pos[3 * pad + e] = y;
            if (e % 3 == 0) mass[b] = b < cnt && P.id[first + b] >= 0 ? P.mass[first + b] : 0.0;
        }
    } else if (t < 3 * nl) {   // 3 n_large <= pull
        ly[t] = P.y_r[3 * P.off + t];
        lv[t] = P.y_v[3 * P.off + t];
        si[0][t] = ly[t];
        if (t % 3 == 0) si_m[t / 3] = P.id[P.off + t / 3] >= 0 ? P.mass[P.off + t / 3] : 0.0;
        if (t < 3 && nl % 2) {   // an odd one's partner: no mass, far from everything
            si[0][3 * nl + t] = si[1][3 * nl + t] = 2.0e9;
            si_m[nl] = 0.0;
        }
    } else if (t >= main) {
        const int o = t - main;
        for (int k = o; k < (int)(sizeof(NyTableau) / 16); k += P.owners)
            reinterpret_cast<uint4*>(&T)[k] = reinterpret_cast<const uint4*>(P.tab)[k];
        if (blockIdx.x == 0)
            for (int k = o; k < (int)(sizeof(DevSys) / 4); k += P.owners)
                reinterpret_cast<unsigned*>(&own.sys)[k] = reinterpret_cast<const volatile unsigned*>(S)[k];
        if (o == 0) {
            const volatile DevSys* V = S;
            const double dt = V->dt_try;
            const unsigned ep = *(volatile unsigned*)P.epoch;
            start.runs = V->active && !V->halted && V->quota != 0;
            start.dt = dt;
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
    const double dt = start.dt;
    const unsigned tag0 = start.tag;
    if (t < P.pull)   // the pull group fences this before its second record
        for (long long k = (long long)blockIdx.x * P.pull + t; k < P.head_n; k += (long long)gridDim.x * P.pull)
            P.head[k] = -1;
    if (t >= main) {
        if ((int)blockIdx.x < nl) run_owner64(P, own, T, &dead, tag0, dt, ly, lv, t - main);
        return;
    }
    const int lane = t & 31;
    if (t < P.pull) {
        // a warp takes 16 small bodies and share p of the pairs of large ones, a half-warp one
        // of the two; four pairs of them at a time
        const int half = lane >> 4, nk = (nl + 1) / 2;
        for (int s = 0; s < ns; s++) {
            const int q = s & 1;
            for (int job = t / 32; job < np * bw; job += kTry64Pull / 32) {
                const int bg = job % bw, p = job / bw, b = 16 * bg + (lane & 15);
                const double x = pos[3 * (q * pad + b)], y = pos[3 * (q * pad + b) + 1], z = pos[3 * (q * pad + b) + 2];
                const double m = mass[b];
                double ax = 0.0, ay = 0.0, az = 0.0;
                for (int i0 = p; i0 < nk; i0 += 4 * np) {
                    double v[12];
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        const int i = i0 + u * np, k = 2 * i + half;
                        v[3 * u] = v[3 * u + 1] = v[3 * u + 2] = 0.0;
                        if (i < nk) {   // uniform
                            const double dx = x - si[q][3 * k], dy = y - si[q][3 * k + 1], dz = z - si[q][3 * k + 2];
                            const double c = inverse_cube(dx, dy, dz);
                            const double f = m * c, g = -(si_m[k] * c);
                            v[3 * u] = f * dx;
                            v[3 * u + 1] = f * dy;
                            v[3 * u + 2] = f * dz;
                            ax = fma(g, dx, ax);
                            ay = fma(g, dy, ay);
                            az = fma(g, dz, az);
                        }
                    }
                    double r;
                    int u = 0;
                    if (i0 + np < nk) {   // uniform
                        r = half_sum12(v, lane);
                        u = 2 * ((lane >> 3) & 1) + ((lane >> 2) & 1);
                    } else {
                        r = half_sum3(v[0], v[1], v[2], lane);
                        if (lane & 12) u = nk;   // one copy of it
                    }
                    const int k = 2 * (i0 + u * np) + half;
                    if (k < nl && (lane & 3) < 3) wp[(k * bw + bg) * 3 + (lane & 3)] = r;
                }
                ax += __shfl_xor_sync(0xffffffffu, ax, 16);
                ay += __shfl_xor_sync(0xffffffffu, ay, 16);
                az += __shfl_xor_sync(0xffffffffu, az, 16);
                if (half == 0) {
                    double* o = parts + 3 * ((size_t)(q * np + p) * pad + b);
                    o[0] = ax;
                    o[1] = ay;
                    o[2] = az;
                }
            }
            lanes_sync(4, P.pull);
            const unsigned tag = tag_of(tag0 + 1 + s, &dead);
            for (int e = t; e < 3 * nl; e += P.pull) {
                const double* o = wp + e / 3 * bw * 3 + e % 3;
                double a0 = 0.0, a1 = 0.0;
                for (int u = 0; u < bw; u += 2) {
                    a0 += o[3 * u];
                    if (u + 1 < bw) a1 += o[3 * u + 3];
                }
                st_rec(P.part + ((size_t)(q * nl + e / 3) * P.n_cta + blockIdx.x) * 3 + e % 3, a0 + a1, tag);
            }
            if (s == 1 && P.head_n > 0) __threadfence();   // the cleared hash before the later records
            lanes_sync(1, main);   // also before wp is written again
        }
        return;
    }

    // ---- the body group: K of the previous stage, positions of the next ----
    const int tb = t - P.pull, items = 3 * cnt;
    GridInfo grid{};
    if (P.head) grid = *P.grid;
    for (int s = 0; s <= ns; s++) {
        for (int e = tb; e < items; e += P.bodies) {
            if (s > 0) {
                const double* pt = parts + (size_t)((s - 1) & 1) * np * 3 * pad + e;
                double g = pt[0];
                for (int u = 1; u < np; u++) g += pt[(size_t)3 * u * pad];
                ks[(size_t)(s - 1) * n3 + e] = P.id[first + e / 3] > 0 ? g : 0.0;
            }
            if (s + 1 < ns)
                pos[((s + 1) & 1) * 3 * pad + e] =
                    fma(dt * dt, row_sum(T, s + 1, ks + e, n3), fma(T.c[s + 1] * dt, yv[e], yr[e]));
        }
        if (s == ns) break;
        if (s + 1 < ns)
            for (int e = tb; e < 3 * nl; e += P.bodies)
                si[(s + 1) & 1][e] = s == 0 ? fma(T.c[1] * dt, lv[e], ly[e])
                                            : poll_rec(pos_records64(P, s + 1) + e, tag0 + 2 + s, S, &dead);
        lanes_sync(1, main);
    }
    if (P.adaptive) {
        unsigned long long eb = 0ull;
        for (int e = tb; e < items; e += P.bodies) eb = max(eb, component_error(T, P.scheme, dt, ks + e, n3));
        for (int m = 16; m > 0; m >>= 1) eb = max(eb, __shfl_xor_sync(0xffffffffu, eb, m));
        if ((tb & 31) == 0) atomicMax(&err_sm, eb);
        lanes_sync(3, P.bodies);
        if (tb == 0)
            st_pair(P.err + blockIdx.x, (unsigned)err_sm, (unsigned)(err_sm >> 32), tag_of(tag0 + 14, &dead));
    }
    for (int e = tb; e < items; e += P.bodies) solution(T, dt, ks + e, n3, yr[e], yv[e]);
    if (tb == 0) {
        take = poll_pair(P.decision, tag0 + 15, S, &dead).x == 1u;
        if (P.head_n > 0) __threadfence();
    }
    lanes_sync(3, P.bodies);
    if (!take) return;
    int* cell = reinterpret_cast<int*>(parts);   // the pull group has left it
    bool bad = false;
    for (int e = tb; e < items; e += P.bodies) {
        const double r = yr[e], v = yv[e];
        P.y_r[3 * first + e] = r;
        P.y_v[3 * first + e] = v;
        bad = bad || not_finite(r) || not_finite(v);
        write_pos_c(P.pos_hi, P.pos_lo, first + e / 3, e % 3, r);
        if (grid.enabled) cell[e] = cell_coord(r, grid.inv_h);
    }
    if (bad) set_status(S, 5);   // RED_ERR_NONFINITE
    if (!grid.enabled) return;   // uniform
    lanes_sync(3, P.bodies);
    for (int b = tb; b < cnt; b += P.bodies) {
        const int4 cl = make_int4(cell[3 * b], cell[3 * b + 1], cell[3 * b + 2], 0);
        P.cell[first + b] = cl;
        P.next[first + b] = atomicExch(&P.head[grid.toff + bucket_of(cl.x, cl.y, cl.z, grid.mask)], first + b);
    }
}

int try64_ctas_per_sm(int threads, size_t smem)
{
    int dev = 0, most = 0, n = 0;
    cudaFuncAttributes a;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
        cudaFuncGetAttributes(&a, k_try64) != cudaSuccess || smem + a.sharedSizeBytes > (size_t)most ||
        cudaFuncSetAttribute(k_try64, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)a.sharedSizeBytes) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_try64, threads, smem) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

void launch_try64(const TryParams& P, cudaStream_t s)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)P.n_cta);
    cfg.blockDim = dim3((unsigned)(P.pull + P.bodies + P.owners));
    cfg.dynamicSmemBytes = try64_smem(P.nb, P.n_stage, P.n_large);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k_try64, P);
}

}  // namespace redgb
