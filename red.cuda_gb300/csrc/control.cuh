// control.cuh -- the step control of one system after a try, shared by k_control
// and by the kernel that makes a whole try (try.cu).
#pragma once
#include "common.cuh"

namespace redgb {

// x^(-1/n) for 1e-30 < x < 1e30, n <= 7: the FP32 power, then one third-order
// step z (1 + t/n + (n+1) t^2 / (2 n^2)) with t = 1 - x z^n.  t ~ 1e-6, so the
// result is good to an ulp (largest error found: 0.76 ulp, where pow(1 / x, 1.0 / n) is off by
// up to 5.6, for the rounded exponent); ten dependent FP64 operations of 64 cycles
// each, where pow() takes ~60.
__device__ __forceinline__ double inverse_root(double x, int n)
{
    const float rn = 1.0f / (float)n;
    const double z = (double)powf((float)x, -rn);
    const double z2 = z * z, z4 = z2 * z2;
    const double zn = n == 7 ? z4 * (z2 * z) : (n == 4 ? z4 : (n == 2 ? z2 : z));
    const double t = fma(-x, zn, 1.0);
    const double r = 1.0 / (double)n;
    return fma(z * t, fma(t, 0.5 * r * (1.0 + r), r), z);
}

// integrator::step's accept / reject logic (int_rungekutta8.cu:690-716,
// int_rungekutta4.cu:226-248), the counters (integrator.cu:270-275) and
// run_simulation's dt_next clamp and loop bound (main.cu:471, 535-538), for a
// runnable system whose try ended with the largest error of bits err_bits.
__device__ __forceinline__ void control_system(const ControlParams& P, DevSys& S, unsigned long long err_bits)
{
    S.accepted = 0;
    const double dt = S.dt_try;
    double dt_new = dt;
    S.iter++;
    if (P.adaptive) {
        const double err = __longlong_as_double((long long)err_bits);
        const double max_err = fabs(P.lambda * dt * err);
        S.err_last = max_err;
        if (max_err != max_err) {
            S.status = 5;   // RED_ERR_NONFINITE
            S.halted = 1;
            S.active = 0;
            return;
        }
        // the red-exact mode takes the nearest double of the power, as the C
        // library's pow of red's host controller does (crmath.cuh)
        if (0.0 < max_err) {
            const double x = max_err / P.tolerance;
            double f;
            if (P.exact) f = crmath::cr_pow(P.tolerance / max_err, 1.0 / (double)P.order);
            else if (x > 1.0e-30 && x < 1.0e30) f = inverse_root(x, P.order);
            else f = pow(P.tolerance / max_err, 1.0 / (double)P.order);
            dt_new = dt * (0.9 * f);
        } else {
            dt_new = dt * 2.0;
        }
        if (max_err > P.tolerance) {
            S.dt_try = dt_new;
            S.dt_next = dt_new;
            return;
        }
    }
    S.dt_did = dt;
    S.dt_next = dt_new;
    S.t += dt;
    S.n_tried += (unsigned long long)S.iter;
    S.n_failed += (unsigned long long)(S.iter - 1);
    S.n_passed += 1ull;
    S.iter = 0;
    S.accepted = 1;
    if (S.quota > 0) S.quota--;
    if (P.output_interval != 0.0 && fabs(P.output_interval) < fabs(S.dt_next))
        S.dt_next = 0.0 < dt ? P.output_interval : -P.output_interval;
    // euler::step / rungekutta2::step take dt_try, never dt_next (int_euler.cu:73-105)
    if (!P.keep_dt) S.dt_try = S.dt_next;
    if (P.length != 0.0 && fabs(S.t - S.t_start) > fabs(P.length)) S.active = 0;
}

// Cell coordinates of the collision check's spatial hash, clamped so that
// far-away bodies share border cells (tested exactly, never missed), and the
// bucket of a cell.
__device__ __forceinline__ int cell_coord(double x, double inv_h)
{
    const double lim = 1.0e9;
    return (int)floor(fmin(fmax(x * inv_h, -lim), lim));
}
__device__ __forceinline__ int bucket_of(int cx, int cy, int cz, int mask)
{
    const unsigned h = ((unsigned)cx * 73856093u) ^ ((unsigned)cy * 19349663u) ^ ((unsigned)cz * 83492791u);
    return (int)(h & (unsigned)mask);
}

}  // namespace redgb
