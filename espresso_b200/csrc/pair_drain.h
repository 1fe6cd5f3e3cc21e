// How a pair of SMs leaves the product on pairs (pair_gemm.cuh) after a wait gave up: what the first CTA does to its `full`
// barriers so that they complete exactly when every copy that either CTA has issued has landed.  Plain C++, so that it can be
// checked on the host.
//
// A fill is one K block: `bytes` copied by the first CTA and `bytes` by its peer, all counted on the first CTA's barrier of stage
// fill % stages, which also waits for one arrival (the first CTA's, with the bytes of both).  The CTAs stop after
// n_first and n_peer fills, which may differ.
#pragma once

#ifndef __CUDACC__
#define __host__
#define __device__
#define __forceinline__ inline
#endif

namespace esp {

struct PgDrainStep {
    int stage;
    unsigned parity;  // phase of the stage's barrier to wait for
    int expect;       // bytes to arrive with (the first CTA had not reached this fill), or 0
    int complete;     // bytes to count as landed (announced for a peer that never issued them), or 0
};

__host__ __device__ __forceinline__ int pg_drain_end(int n_first, int n_peer) { return n_first > n_peer ? n_first : n_peer; }
// Fills before the last `stages` ones have been consumed: their stage was filled again.
__host__ __device__ __forceinline__ int pg_drain_begin(int n_first, int n_peer, int stages) {
    const int n = pg_drain_end(n_first, n_peer) - stages;
    return n > 0 ? n : 0;
}
__host__ __device__ __forceinline__ PgDrainStep pg_drain_step(int fill, int n_first, int n_peer, int stages, int bytes) {
    PgDrainStep d;
    d.stage = fill % stages;
    d.parity = (unsigned)(fill / stages) & 1u;
    d.expect = fill >= n_first ? bytes : 0;
    d.complete = fill >= n_peer ? bytes : 0;
    return d;
}

}  // namespace esp
