// records.cuh -- what the whole-try kernels (try.cu, try64.cu) share: the tagged
// exchange records, the barriers of a group of warps, the step control at the end.
#pragma once
#include "common.cuh"
#include "control.cuh"
#include "try.cuh"

namespace redgb {

namespace {

// 16-byte records: three words and a tag, one 128-bit access each way.  The compiler
// keeps the load whole only if all four words are used: with x and the tag alone it made
// two 32-bit loads of it, and a reader met the new tag beside the old x (one read in
// 70 while the record changed).  So a record of three words is read for all three, and one of
// two words or less goes through st_pair and poll_pair.
__device__ __forceinline__ void st_rec16(uint4* p, unsigned x, unsigned y, unsigned z, unsigned tag)
{
    asm volatile("{\n\t.reg .b128 q;\n\t.reg .b64 a, b;\n\tmov.b64 a, {%1, %2};\n\tmov.b64 b, {%3, %4};\n\t"
                 "mov.b128 q, {a, b};\n\tst.relaxed.gpu.global.b128 [%0], q;\n\t}\n" ::"l"(p), "r"(x), "r"(y), "r"(z),
                 "r"(tag)
                 : "memory");
}
__device__ __forceinline__ uint4 ld_rec16(const uint4* p)
{
    uint4 v;
    asm volatile("{\n\t.reg .b128 q;\n\t.reg .b64 a, b;\n\tld.relaxed.gpu.global.b128 q, [%4];\n\t"
                 "mov.b128 {a, b}, q;\n\tmov.b64 {%0, %1}, a;\n\tmov.b64 {%2, %3}, b;\n\t}\n"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p)
                 : "memory");
    return v;
}

// A status that no earlier one is overwritten by.
__device__ __forceinline__ void set_status(DevSys* S, int status) { atomicCAS(&S->status, 0, status); }

// Waits for the record with this tag.  A missing one, or one whose writer has given
// the try up, stops the system; *dead (shared memory) then ends the CTA's other waits
// and marks its records (tag_of).
__device__ __noinline__ uint4 missing_record(DevSys* S, volatile int* dead)
{
    *dead = 1;
    set_status(S, 4);   // RED_ERR_TIMEOUT
    S->halted = 1;
    return make_uint4(0x7fc00000u, 0x7fc00000u, 0x7fc00000u, 0u);
}
// A record of the try of this tag whose writer has given it up, at whatever stage.
__device__ __forceinline__ bool given_up(unsigned got, unsigned tag) { return ((got ^ tag) & ~15u) == kTryAbort; }
__device__ __forceinline__ uint4 poll16(const uint4* p, unsigned tag, DevSys* S, volatile int* dead)
{
    for (int k = 0; k < kTryPollLimit; k++) {
        const uint4 v = ld_rec16(p);
        if (v.w == tag) return v;
        if (given_up(v.w, tag)) break;
        if ((k & 63) == 63 && *dead) break;
    }
    return missing_record(S, dead);
}

// A record of two words.  The third one is their sum modulo 2 with the tag, so that all
// four are needed and words of two records do not pass for one.
__device__ __forceinline__ void st_pair(uint4* p, unsigned lo, unsigned hi, unsigned tag)
{
    st_rec16(p, lo, hi, lo ^ hi ^ tag, tag);
}
__device__ __forceinline__ uint2 poll_pair(const uint4* p, unsigned tag, DevSys* S, volatile int* dead)
{
    for (int k = 0; k < kTryPollLimit; k++) {
        const uint4 v = ld_rec16(p);
        if (v.w == tag && (v.x ^ v.y ^ v.z) == tag) return make_uint2(v.x, v.y);
        if (given_up(v.w, tag)) break;
        if ((k & 63) == 63 && *dead) break;
    }
    const uint4 v = missing_record(S, dead);
    return make_uint2(v.x, v.y);
}

__device__ __forceinline__ unsigned tag_of(unsigned tag, const volatile int* dead)
{
    return *dead ? tag ^ kTryAbort : tag;
}

// A barrier of some warps.  bar.sync is the aligned form: all lanes of a warp must
// come together, which nothing promises after a loop or branch that only some
// took, so __syncwarp() brings them together first.
__device__ __forceinline__ void group_sync(int id, int threads)
{
    __syncwarp();
    asm volatile("bar.sync %0, %1;\n" ::"r"(id), "r"(threads) : "memory");
}

__device__ __forceinline__ bool not_finite(double x)
{
    return ((__double_as_longlong(x) >> 52) & 0x7ff) == 0x7ff;
}

// sum a_q K_q over the terms [u0, u1) of the tableau, or over a row, K_q at k[q st].
// In FP64, as every stage sum, error and solution of the whole-try kernels.
__device__ __forceinline__ double row_sum(const NyTableau& T, int u0, int u1, const double* k, int st)
{
    double a = 0.0;
#pragma unroll 4
    for (int u = u0; u < u1; u++) a = fma(T.term[u].a, k[T.term[u].q * st], a);
    return a;
}
__device__ __forceinline__ double row_sum(const NyTableau& T, int row, const double* k, int st)
{
    return row_sum(T, T.beg[row], T.beg[row + 1], k, st);
}
// The larger of a component's position error er and velocity error ev, as bits (NaN above all).
__device__ __forceinline__ unsigned long long error_bits(double er, double ev)
{
    double e = fmax(fabs(er), fabs(ev));
    if (er != er || ev != ev) e = __longlong_as_double(0x7ff8000000000000ll);
    return (unsigned long long)__double_as_longlong(e);
}
__device__ __forceinline__ unsigned long long component_error(const NyTableau& T, int scheme, double dt,
                                                              const double* k, int st)
{
    return error_bits(dt * row_sum(T, kTryRowER, k, st),
                      scheme == SCHEME_RKF78 ? ((k[0] + k[10 * st]) - k[11 * st]) - k[12 * st]
                                             : k[3 * st] - k[4 * st]);
}
// The solution of a component from (y, v): y + dt (cb v + dt sum), v + dt sum.
__device__ __forceinline__ void solution(const NyTableau& T, double dt, const double* k, int st, double& y, double& v)
{
    y = fma(dt, fma(dt, row_sum(T, kTryRowRB, k, st), T.cb * v), y);
    v = fma(dt, row_sum(T, kTryRowVB, k, st), v);
}

// The step control on a copy of the system record; the fields it sets go back.
__device__ __noinline__ void control_of(const ControlParams& P, DevSys& C, unsigned long long err)
{
    control_system(P, C, err);
}
__device__ __forceinline__ void store_control(DevSys* S, const DevSys& C)
{
    S->t = C.t;
    S->dt_try = C.dt_try;
    S->dt_did = C.dt_did;
    S->dt_next = C.dt_next;
    S->n_tried = C.n_tried;
    S->n_passed = C.n_passed;
    S->n_failed = C.n_failed;
    S->iter = C.iter;
    S->accepted = C.accepted;
    S->active = C.active;
    S->quota = C.quota;
    S->err_last = C.err_last;
    if (C.status) set_status(S, C.status);   // other CTAs may set these
    if (C.halted) S->halted = C.halted;
}

}  // namespace

}  // namespace redgb
