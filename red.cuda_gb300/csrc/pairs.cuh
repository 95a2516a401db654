// pairs.cuh -- gravity of a class in which every body pulls every other: each
// pair once (pairs.cu).
//
// The large bodies [b0, b0 + n) of one system lie in blocks of kPairBlock.  A CTA
// (PairJob) takes a block I of sinks against some sub-blocks of kTile bodies at or
// after it and forms each pair's separation and inverse cube once, for both
// bodies.  It leaves two kinds of partial sums, as records of three double-single
// values per body, [slot][body]: its block's sums over the job's bodies, in the
// slot kPairBlock-block index + chunk of the job, and for every body of a later
// block the sum over block I, in slot I.  The stage kernel adds a tile's slots and
// goes on as usual (GravItem::n_rec).
#pragma once
#include "redgb_dev.cuh"

namespace redgb {

constexpr int kPairSinks = 4;                      // sinks per thread
constexpr int kPairBlock = kPairSinks * kTile;     // 512

struct PairJob {
    int block;        // I: sinks [I kPairBlock, ..), relative to b0
    int sub0, sub1;   // sub-blocks of kTile bodies, [4 I, ..)
    int slot;         // of the sinks' sums
};

struct PairParams {
    const PairJob* jobs;
    const DevSys* sys;
    int b0, n;
    const float4* pos_hi;
    const float4* pos_lo;
    float2* rec;      // [slot][n][3]
};

void launch_pairs(const PairParams& P, int n_jobs, int mode, cudaStream_t s);

}  // namespace redgb
