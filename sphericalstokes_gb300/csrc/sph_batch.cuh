// Batched correction sweeps over many grids of uneven size in one launch.
//
// A batch of mixed-precision solves advances in lockstep: every solve whose
// correction problem is being iterated runs the same number of FP32 sweeps per
// round.  One sweep of all of them is one launch of k_sweep_batch per
// geometry over a work list of (solve, tile x, tile y, x3 chunk) items — the
// blocks each solve's own k_sweep launch would have; the sweeps handle the
// boundary velocities themselves (SweepOut::gmask, smask), and a round of sweeps
// is replayed from one CUDA graph.  The kernels run the single-grid bodies
// (sweep_body, velocity_norm_body), so each solve computes exactly what it
// computes alone.
//
// Per-solve data live in device memory (BatchSweep), read by the kernels at
// run time, so the captured graph stays valid while solves enter and leave the
// correction phase: the host rewrites a solve's entry and its active flag,
// and blocks of inactive solves return at once.
#pragma once
#include "sph_pt.cuh"
#include "sph_sweep.cuh"

namespace sph {

struct BatchSweep {
    KP<float> p[2];                // correction problem in both ping-pong arrangements (a: the sweep reads p[a])
    SweepOut<float> o[2];          // outputs of a sweep reading arrangement a (the other buffer set)
    const CUtensorMap* maps[2];    // TMA maps of the arrangement a sweep reads
    int* err;                      // the solve's bounded-wait error word
    int kchunk;                    // x3 planes per block
};

// one correction sweep of every active solve of geometry G (items: x = solve, y, z, w = tile x, y, chunk)
template <int G>
__global__ void __launch_bounds__(SW_NT, 2) k_sweep_batch(const BatchSweep* __restrict__ b, const int4* __restrict__ items,
                                                             const int* __restrict__ active, int a) {
    pdl_wait();  // as k_sweep: no early release of the next grid
    const int4 it = items[blockIdx.x];
    if (!active[it.x]) return;  // whole block: no barrier is reached
    // the solve's scalars and pointers in shared memory: the march reads them plane by plane
    __shared__ KP<float> p;
    __shared__ SweepOut<float> o;
    const BatchSweep& s = b[it.x];
    auto copy = [](void* dst, const void* src, int bytes) {
        for (int i = threadIdx.x; i < bytes / 4; i += SW_NT) static_cast<int*>(dst)[i] = static_cast<const int*>(src)[i];
    };
    copy(&p, &s.p[a], sizeof(p));
    copy(&o, &s.o[a], sizeof(o));
    __syncthreads();
    sweep_body<G, 1>(p, o, s.kchunk, s.maps[a], s.err, it.y, it.z, it.w);
}

// inner stopping test of every active solve of geometry G: max |dV + rV| of arrangement 0 into
// red[solve]; items: x = solve, y, z, w = velocity-node block; 32 x 8 threads
template <int G>
__global__ void __launch_bounds__(256) k_velocity_norm_batch(const BatchSweep* __restrict__ b, const int4* __restrict__ items,
                                                             const int* __restrict__ active, unsigned long long* __restrict__ red) {
    const int4 it = items[blockIdx.x];
    if (!active[it.x]) return;
    velocity_norm_body<float, G>(b[it.x].p[0], it.y, it.z, it.w, red + it.x);
}

}  // namespace sph
