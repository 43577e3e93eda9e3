// Batched correction sweeps over many grids of uneven size in one launch.
//
// A batch of mixed-precision solves advances in lockstep: every solve whose
// correction problem is being iterated runs the same number of FP32 sweeps per
// round.  One sweep of all of them is one launch of k_sweep_batch over a work
// list of (solve, tile x, tile y, x3 chunk) items; the sweeps handle the boundary
// velocities themselves (SweepOut::gmask, smask), and a round of sweeps
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
    SweepMaps maps[2];             // TMA maps of the arrangement a sweep reads
    int* err;                      // the solve's bounded-wait error word
    int geom;
};

// one correction sweep of every active solve (items: x = solve, y, z, w = tile x, y, chunk; kchunk: planes per
// block of each solve).  All geometries in one launch: a block runs the body of its own, and the
// blocks of a small batch fill the SMs together (12 grids of 31 .. 47 cells a side, 600 sweeps with the
// FP64 steps and copies: 50.8 ms with a launch per geometry and each solve's own chunk, 39.2 ms so, 26.6 ms with
// the sweep of now and blocks of one geometry on an SM).
// LIFT: if any solve has small viscosities (the others' results do not change).
template <bool LIFT>
__global__ void __launch_bounds__(SW_NT, 2) k_sweep_batch(const BatchSweep* __restrict__ b, const int4* __restrict__ items,
                                                          const int* __restrict__ active, const int* __restrict__ kchunk, int a) {
    // (items, flags and entries change between launches of the whole round only)
    const int4 it = items[blockIdx.x];
    if (!active[it.x]) {  // whole block: no barrier is reached
        pdl_wait();
        return;
    }
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
    // maps in global memory are copied there between launches: the copy unit may hold older ones of this address
    if (threadIdx.x == SW_NT - 32)
        for (int i = 0; i < SM_COUNT; ++i)
            asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;\n" ::"l"(s.maps[a].m + i) : "memory");
    const int kc = kchunk[it.x];
    if (s.geom == SPH) sweep_body<SPH, 1, LIFT>(p, o, kc, s.maps[a].m, s.err, it.y, it.z, it.w);
    else if (s.geom == CYL) sweep_body<CYL, 1, LIFT>(p, o, kc, s.maps[a].m, s.err, it.y, it.z, it.w);
    else sweep_body<CART, 1, LIFT>(p, o, kc, s.maps[a].m, s.err, it.y, it.z, it.w);
}

// inner stopping test of every active solve: max |dV + rV| of arrangement 0 into red[solve];
// items: x = solve, y, z, w = velocity-node block; 32 x 8 threads
__global__ void __launch_bounds__(256) k_velocity_norm_batch(const BatchSweep* __restrict__ b, const int4* __restrict__ items,
                                                             const int* __restrict__ active, unsigned long long* __restrict__ red) {
    const int4 it = items[blockIdx.x];
    if (!active[it.x]) return;
    const BatchSweep& s = b[it.x];
    if (s.geom == SPH) velocity_norm_body<float, SPH>(s.p[0], it.y, it.z, it.w, red + it.x);
    else if (s.geom == CYL) velocity_norm_body<float, CYL>(s.p[0], it.y, it.z, it.w, red + it.x);
    else velocity_norm_body<float, CART>(s.p[0], it.y, it.z, it.w, red + it.x);
}

}  // namespace sph
