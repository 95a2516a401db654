// records.cuh -- what the whole-try kernels (try.cu, try64.cu) share: the tagged
// exchange records, the barriers of a group of warps, the step control at the end.
#pragma once
#include "common.cuh"
#include "control.cuh"
#include "try.cuh"

namespace redgb {

namespace {

// 16-byte records: three words and a tag, one 128-bit access each way.
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

// Waits for the record with this tag.  A missing one stops the system; *dead
// (shared memory) then ends the CTA's other waits.
__device__ __noinline__ uint4 missing_record(DevSys* S, volatile int* dead)
{
    *dead = 1;
    S->status = 4;   // RED_ERR_TIMEOUT
    S->halted = 1;
    return make_uint4(0x7fc00000u, 0x7fc00000u, 0x7fc00000u, 0u);
}
__device__ __forceinline__ uint4 poll16(const uint4* p, unsigned tag, DevSys* S, volatile int* dead)
{
    for (int k = 0; k < kTryPollLimit; k++) {
        const uint4 v = ld_rec16(p);
        if (v.w == tag) return v;
        if ((k & 63) == 63 && *dead) break;
    }
    return missing_record(S, dead);
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
    if (C.status) S->status = C.status;   // else as it is: other CTAs may set these
    if (C.halted) S->halted = C.halted;
}

}  // namespace

}  // namespace redgb
