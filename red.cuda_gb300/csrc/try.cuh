// try.cuh -- a whole try of one sparse system in one cooperative launch.
//
// A planetesimal disk has a handful of large bodies (stars and protoplanets, the
// SI class) that everything feels, and many small bodies (the NSI class) that
// only the large ones feel.  A small body's equations then need nothing but the
// large bodies' positions, and the large bodies need one sum over the small
// ones per stage.  k_try gives every CTA a range of small bodies for the whole
// try: their state, their accelerations of all stages and the large bodies'
// positions stay in shared memory; per stage the CTAs exchange only the partial
// sums on the large bodies and the new positions of these.
//
// The stages run on accelerations alone.  With the stage velocity v_s = y_v + dt
// sum_q a_sq K_q put into the stage position (Nystroem's form of the same
// method),
//   r_s = y_r + dt (c_s y_v + dt sum_q A_sq K_q),   A = a a,
// and A_sq = 0 for q >= s - 1: the positions of stage s do not wait for the
// accelerations of stage s - 1.  An exchange (partial sums to the CTA that owns a
// large body, its new position back to all) therefore has the time of a whole
// stage to complete, and stage velocities are formed only for gas drag.
//
// The pair and star sums leave the accelerations as double-single numbers (the star
// term is good to ~7e-14); everything formed from them is FP64, as in the stage
// kernel: the stage sums, positions and velocities, the drag, the error, the solution.
// GB300 issues an FP64 warp instruction every 19 cycles and SM and a dependent one
// takes 64, so a component's sum is one thread's chain, off the exchange's path but for
// the last term.  (Double-single sums, ~12 FP32 instructions a term, took 56 instead of
// 59 us per try of the 16384-body disk.  They round at 2^-47, and the modes promise
// FP64.)
//
// Bound: latency -- of the exchange, two trips through L2 per two stages, and of
// the instruction chains of a phase (~2.7 us per phase on the 16384-body disk, 1.3
// of them the pull on the large bodies, whose records the exchange waits for).
// Measured against one launch per stage, per try: 16384-body disk, adaptive
// RKF7(8), 115 -> 58 us; 65536-body gas-drag disk 418 -> 259 us (FP64 pipe: the rows of
// velocities and the drag); 2053-body disk, RK4, 33.2 -> 21.3 us.  What that took besides the layout: the system record is
// read by one thread of a CTA and the position records are written in kTryCopies
// copies, because thousands of readers of one sector queue up for microseconds.
//
// Records: 16 bytes with a 32-bit tag of the try and stage, written and read as
// one 128-bit access, so a record is complete when its tag is right and needs no
// fence or reset.  Two sets of partial sums alternate by stage: a CTA writes a slot
// again two stages later, when it has positions that the slot's reader formed
// from it.  The positions take four sets: the group that sums body j's partials
// can be three stages ahead of the group of body k, but not four, since the
// partials of a stage wait for k's positions.
//
// The cleared hash of the collision check precedes every insertion by a chain of fences
// and records: a CTA's clearing, its barrier, a fence in each thread that writes its partial
// sums (stage 1), the sums of stage 2; in the first CTA a fence after reading them, its
// barrier, a fence in the thread that decides (stage 3), the decision; a fence after reading
// that, a barrier, the insertions.  Schemes of one or two stages have the hash cleared before.
//
// Every wait is bounded.  After kTryPollLimit reads a record counts as missing: the
// system's status becomes RED_ERR_TIMEOUT and it halts, the CTA's other waits end at
// once, and its own records carry kTryAbort, which ends the waits for them too.  No CTA
// writes its solution before the first one, which hears of every CTA's and every owner's
// try, has decided (in fixed steps too), and it takes no step then: state, time and
// counters stay as they were.  (In fixed steps the decision costs 1.6 us of a try, 2053 bodies.)  The launch is
// cooperative: all its CTAs are resident together.
#pragma once
#include "common.cuh"
#include "control.cuh"

namespace redgb {

constexpr int kTryMaxOwners = 192;     // threads of the owner group, at most
constexpr int kTryMaxLarge = 64;       // large bodies of a system on this path
constexpr int kTryMaxStars = 4;
constexpr int kTryCopies = 8;          // of the position records: 1/8 of the CTAs wait on each
#ifndef REDGB_TRY_POLL_LIMIT
#define REDGB_TRY_POLL_LIMIT (1 << 20)     // about a second
#endif
constexpr int kTryPollLimit = REDGB_TRY_POLL_LIMIT;
constexpr unsigned kTryAbort = 0x80000000u;   // in a record's tag: its writer has given the try up
// The tags of a try follow this one; below kTryAbort.
__host__ __device__ constexpr unsigned try_tag(unsigned epoch) { return (epoch & 0x07ffffffu) * 16u; }

// Nystroem form of a scheme: its rows over the accelerations, nonzero terms only,
// ascending stages.  Row s: the positions of stage s (dt^2 sum a K); kTryRowV + s:
// the velocities (dt sum a K); kTryRowRB and kTryRowVB: the solution's positions
// (dt^2) and velocities (dt); kTryRowER: the position error (dt).
constexpr int kTryRowV = kMaxStages, kTryRowRB = 2 * kMaxStages, kTryRowVB = kTryRowRB + 1, kTryRowER = kTryRowVB + 1;
constexpr int kTryRows = kTryRowER + 1;
struct NyTerm {
    double a;                // the coefficient
    int q, pad;              // the stage
};
struct alignas(16) NyTableau {
    NyTerm term[176];
    double c[kMaxStages];    // sum of row s of a: the factor of dt y_v in stage s
    double cb;               // sum of b
    int beg[kTryRows + 1];   // row k: terms [beg[k], beg[k + 1])
    int pad[2];
};
static_assert(sizeof(NyTableau) % 16 == 0, "copied by 16 bytes");

struct TryParams {
    int scheme, n_stage, adaptive;
    int n_cta, nb;           // CTAs, small bodies of each (the last may have fewer)
    int pull, bodies, owners;   // threads of the three groups
    int lanes_log2;          // threads per large body in the partial sums (4 .. 32)
    int off, n, n_large, n_star;
    DevSys* sys;
    double* y_r;
    double* y_v;
    const double* mass;
    const double* radius;
    const double* density;
    const double* cd;
    const int* id;
    float4* pos_hi;          // stage-0 copies
    float4* pos_lo;
    const NyTableau* tab;
    uint4* part;             // [2][n_large][n_cta][2], in FP64 [..][3]
    uint4* pos;              // [4][kTryCopies][n_large][2], in FP64 [..][3]
    uint4* err;              // [n_cta + n_large]
    uint4* decision;         // [1]
    unsigned* epoch;         // tries made by this kernel
    GasDev gas;
    ControlParams ctl;
    int* head;               // the collision check's hash (null: none)
    long long head_n;
    int* next;
    int4* cell;
    const GridInfo* grid;
};

// Bytes of dynamic shared memory of a CTA with nb small bodies.
__host__ __device__ constexpr int try_pad(int nb) { return (nb + 31) / 32 * 32; }
// shares of the pair terms on a small body, one thread each
__host__ __device__ constexpr int try_parts(int nb, int pull)
{
    return pull / try_pad(nb) < 1 ? 1 : (pull / try_pad(nb) > 4 ? 4 : pull / try_pad(nb));
}
__host__ __device__ constexpr size_t try_smem(int nb, int n_stage, int pull)
{
    return (size_t)try_pad(nb) * 2 * (2 * sizeof(float4) + (size_t)try_parts(nb, pull) * 3 * sizeof(float2)) +
           (size_t)nb * 3 * sizeof(double) * (n_stage + 2);
}
// Threads of a CTA at most.
__host__ __device__ constexpr int try_max_threads(bool drag) { return drag ? 1024 : 928; }

// ---------------------------------------------------------------------------
// k_team: the same for an ensemble of sparse systems.  A system's small bodies
// are shared by a team of up to kTeamSize CTAs of one thread-block cluster, the
// teams of a cluster side by side; the exchange goes through the CTAs' shared
// memory, ordered by one cluster barrier per phase (the cluster's CTAs run the
// same phases).  A large body's sum and its next position are formed by a warp
// of the team in the phase after the partials, as long as that phase lasts.  512
// disks (1.1 M bodies), adaptive RKF7(8), four tries with the states in and out, against
// one launch per stage: 11.35 -> 8.46 ms (7.04 with double-single stage sums and longer
// FP32 runs).  FP64 pipe 46 % busy, 46 % of the stall at the barriers.
// ---------------------------------------------------------------------------
constexpr int kTeamCtas = 10;          // largest cluster; a team is at most 8 of its CTAs
constexpr int kTeamSize = 8;
constexpr int kTeamLarge = 16;         // large bodies of a system on this path
constexpr int kTeamBodies = 512;       // small bodies of a CTA at most
constexpr int kTeamPull = 512, kTeamBody = 256, kTeamOwners = 256;   // threads of the groups
constexpr int kTeamRounds = 2;         // pairs of components of a body-group thread before the pull group takes its share
__host__ __device__ constexpr int team_bodies(int small, int size) { return ((small + size - 1) / size + 1) / 2 * 2; }   // per CTA: even

struct TeamItem {
    int sys;                 // -1: an idle CTA
    int rank, size;          // of the CTA in its team
    int base;                // cluster rank of the team's first CTA
};

struct TeamParams {
    int scheme, n_stage, adaptive;
    int cluster;             // CTAs of a cluster
    int cap;                 // small bodies a CTA's shared memory is laid out for
    const TeamItem* items;
    const SysInfo* sinfo;
    DevSys* sys;
    double* y_r;
    double* y_v;
    const double* mass;
    const int* id;
    float4* pos_hi;
    float4* pos_lo;
    const NyTableau* tab;
    ControlParams ctl;
    int* head;               // the collision check's hash (null: none)
    int* next;
    int4* cell;
    const GridInfo* grid;
};

__host__ __device__ constexpr size_t team_smem(int cap, int n_stage)
{
    return (size_t)try_pad(cap) * 2 * (2 * sizeof(float4) + 3 * sizeof(float2)) +
           (size_t)cap * 3 * sizeof(double) * n_stage;
}
// Clusters resident at once (0: none, or the query failed), and the launch.
int team_clusters(int mode, int cluster, size_t smem);
void launch_team(const TeamParams& P, int n_ctas, int mode, cudaStream_t s);

// ---------------------------------------------------------------------------
// k_try64: k_try in FP64 (try64.cu), without gas drag.  A pair of a small and a
// large body is formed once, for both.  A warp takes 16 small bodies and, a
// half-warp each, two large ones at a time: a CTA's ~108 bodies of the 16384-body
// disk fill 7 x 16 lanes, but only 3.4 x 32.  A lane adds the large bodies' pull on
// its small body in registers; the pull on the large ones is summed over the
// half-warp, four of them at a time.  Records hold one double each, three per body.
//
// Bound by the FP64 pipe: ~24 warp instructions per 32 pairs, one in ~19 cycles and
// SM, are ~17 of the 18.7 us of a stage of the 16384-body disk with 17 large bodies.
// The stage kernel forms a pair twice, with 16 instructions and the library's root
// each.  That disk, adaptive RKF7(8): 535 us per try with one launch per stage, 243
// here; RKF7(8) with fixed steps, collisions on: 261 bodies 301 -> 56 us, 65000 small
// and 34 large ones 2190 -> 1143 us.
// ---------------------------------------------------------------------------
constexpr int kTry64Pull = 512, kTry64Bodies = 224, kTry64Owners = 160;   // threads of the groups (the latter two: at most)
constexpr int kTry64Threads = kTry64Pull + kTry64Bodies + kTry64Owners;
__host__ __device__ constexpr int try64_pad(int nb) { return (nb + 15) / 16 * 16; }
// shares of the pairs of 16 small bodies, a warp each
__host__ __device__ constexpr int try64_parts(int nb)
{
    return 256 / try64_pad(nb) < 1 ? 1 : (256 / try64_pad(nb) > 4 ? 4 : 256 / try64_pad(nb));
}
__host__ __device__ constexpr size_t try64_smem(int nb, int n_stage, int nl)
{
    return sizeof(double) * ((size_t)try64_pad(nb) * (2 * 3 + 1 + 2 * 3 * try64_parts(nb)) +
                             (size_t)nb * 3 * (n_stage + 2) + (size_t)nl * 3 * (try64_pad(nb) / 16));
}
int try64_ctas_per_sm(int threads, size_t smem);
void launch_try64(const TryParams& P, cudaStream_t s);

// CTAs of the cooperative launch that are resident at once per SM with this much
// shared memory (0: none, or the query failed), and the launch.
int try_ctas_per_sm(int mode, bool drag, int threads, size_t smem);
void launch_try(const TryParams& P, int mode, cudaStream_t s);
void set_tableau_try(const Tableau& tb, cudaStream_t s);

}  // namespace redgb
