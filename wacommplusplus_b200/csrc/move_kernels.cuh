// Move kernels: one thread per particle, the whole interval (or one chunk of it) in registers.
#pragma once

#include "engine.h"
#include "launch_rules.h"
#include "step.cuh"
#include "step_fast.cuh"

namespace wb {

// Structure-of-arrays particle state resident in the engine.
struct ParticleSoA {
    uint64_t *id;
    double *k, *j, *i, *health, *age, *time;
    uint16_t *type;
    int8_t *side;
    double *elapsed;  // resume point between chunks
};

inline PackedView packed_view(const PackedArgs &A) {
    PackedView V;
    V.g = GridShape{A.eta, A.xi, A.sW, A.sRho};
    V.nodes = A.nodes;
    V.surf = A.surf;
    V.env = A.env;
    V.hasWindU = A.hasWindU;
    V.hasWindV = A.hasWindV;
    V.hasStokes = A.hasStokes;
    V.lonRad = A.lonRad;
    V.latRad = A.latRad;
    V.depthIntervals = A.depthIntervals;
    V.metric = A.metric;
    return V;
}

struct MoveLaunch {
    int count;                    // work items
    const uint32_t *order;        // work item -> particle slot (cell-sorted), or null
    uint32_t *conc;               // uint32 concentration grid, or null
    int concTimeIndex, concTimes;
    unsigned long long *steps;    // particle-step counter, or null
    int *err;
    // When set, the work items are the first min(count, *countDevice): a list whose length a
    // kernel earlier on the stream wrote (the launch covers `count`, blocks past the list exit).
    const uint32_t *countDevice = nullptr;
    // FP32 step: work items per thread; the grid is that many times smaller and each block
    // strides over it (results do not depend on it).
    int perThread = 1;
    // Work items per warp (1 to 32): a small launch leaves the other lanes of its warps idle and
    // spreads over the SMs instead (spread_launch; results do not depend on it).
    int lanes = 32;
    // FP32 step with the reference's random keys: the three normals of every substep of every slot,
    // drawn ahead ([drawSteps][drawStride], draw_normals; VAR_DRAWN), or null: drawn in the step.
    const float4 *draws = nullptr;
    unsigned drawSteps = 0, drawStride = 0;
};

// The work item of this thread in a block that starts at item `base`; `count` (none) on the lanes
// left idle.
__device__ __forceinline__ unsigned launch_item(const MoveLaunch &L, unsigned base, unsigned count) {
    if (L.lanes >= 32) return base + threadIdx.x;
    const unsigned lane = threadIdx.x & 31;
    return lane < (unsigned)L.lanes ? base + (threadIdx.x >> 5) * L.lanes + lane : count;
}

// Work items of a launch: count, or the device-side length of its list.
__device__ __forceinline__ int launch_count(const MoveLaunch &L) {
    if (!L.countDevice) return L.count;
    const uint32_t listed = *L.countDevice;
    return listed < (uint32_t)L.count ? (int)listed : L.count;
}

// Linear index of the concentration cell of an alive particle, or -1
// (Concentration.hpp:28-41: round-half-away indices, bounds 0<=j<eta, 0<=i<xi, -sRho<k<=0).
__device__ __forceinline__ long long concentration_cell(const ParticleState &p, int concTime,
                                                        int sRho, int eta, int xi) {
    if (!(p.health > 0)) return -1;
    double rk = round(p.k), rj = round(p.j), ri = round(p.i);
    if (!(rj >= 0.0 && rj < (double)eta && ri >= 0.0 && ri < (double)xi &&
          rk >= (double)(-sRho + 1) && rk <= 0.0))
        return -1;
    int k = (int)rk, j = (int)rj, i = (int)ri;
    return (((long long)concTime * sRho + (k + sRho - 1)) * eta + j) * (long long)xi + i;
}

// Warp-aggregated increment: lanes holding the same cell elect one lane that adds the count.
__device__ __forceinline__ void warp_count(uint32_t *grid, long long cell) {
    unsigned active = __activemask();
    unsigned peers = __match_any_sync(active, (unsigned long long)cell);
    int lane = threadIdx.x & 31;
    if (cell >= 0 && lane == __ffs(peers) - 1) atomicAdd(grid + cell, (uint32_t)__popc(peers));
}

__device__ __forceinline__ void warp_sum_steps(unsigned long long *counter, int steps) {
    unsigned active = __activemask();
    for (int off = 16; off > 0; off >>= 1) steps += __shfl_down_sync(active, steps, off);
    if ((threadIdx.x & 31) == 0 && counter && steps) atomicAdd(counter, (unsigned long long)steps);
}

// Reference arithmetic. The latency of FP64 chains and the conversions to float and back bound it;
// 128 registers allow 16 warps per SM. Where one or two warps per scheduler hold all records, or they are
// spread thinly over the grid (keeps_stencil), the registers go to the velocity stencil instead (KEEP), out
// of the substep's chain of loads. Move kernel on 128 x 128 x 10, KEEP / not: 16,384 records 0.366 / 0.449 ms, 65,536 0.751 / 0.802 ms, 131,072 1.37 / 1.36 ms,
// 500,009 4.73 / 3.71 ms (with the random walk 0.609 / 0.687, 1.28 / 1.15, 2.44 / 1.96, 8.14 / 6.30);
// 242 registers and float operands before: 500,009 with the random walk 10.2 ms, XU pipe 54 -> 22 %,
// FP64 24 -> 44 %, issue 36 -> 57 %. The drift form spills 622 bytes at 128 registers, which cost it what the
// warps brought in (whole interval, at 242 without spills / now): 500,009 records 13.3 / 12.8 ms, with the
// random walk 15.2 / 14.6 ms; 100,000, with the stencil kept, 3.35 / 2.78 ms (4.0 at 128 registers).
template <int SEM, bool DRIFT, bool KEEP>
__global__ void __launch_bounds__(256, KEEP ? 1 : 2) move_soa_kernel(const wacomm_b200_config cfg,
                                                          const IntervalParams P,
                                                          const PackedView V, ParticleSoA S,
                                                          const MoveLaunch L) {
    const unsigned t = launch_item(L, blockIdx.x * (blockDim.x >> 5) * L.lanes, L.count);
    long long cell = -1;
    int steps = 0;
    if (t < (unsigned)L.count) {
        uint32_t slot = L.order ? L.order[t] : (uint32_t)t;
        ParticleState p;
        p.id = S.id[slot];
        p.k = S.k[slot];
        p.j = S.j[slot];
        p.i = S.i[slot];
        p.health = S.health[slot];
        p.age = S.age[slot];
        p.time = S.time[slot];
        p.type = S.type[slot];
        p.side = S.side[slot];
        double elapsed = P.firstChunk ? P.elapsed0 : S.elapsed[slot];
        steps = move_particle<SEM, DRIFT, KEEP>(cfg, P, V, p, elapsed, L.err);
        S.k[slot] = p.k;
        S.j[slot] = p.j;
        S.i[slot] = p.i;
        S.health[slot] = p.health;
        S.age[slot] = p.age;
        S.side[slot] = (int8_t)p.side;
        if (!P.lastChunk) S.elapsed[slot] = elapsed;
        if (L.conc && P.lastChunk) cell = concentration_cell(p, L.concTimeIndex, V.g.sRho, V.g.eta, V.g.xi);
    }
    if (L.steps) warp_sum_steps(L.steps, steps);
    if (L.conc && P.lastChunk) warp_count(L.conc, cell);
}

// Launch shapes of the FP32 kernel: threads per block and the minimum resident blocks per SM the
// register allocation must allow (WACOMM_B200 launch_shape 0..3).
template <int SHAPE>
struct LaunchShape;
template <>
struct LaunchShape<0> {
    static constexpr int threads = 256, minBlocks = 1;
};
template <>
struct LaunchShape<1> {
    static constexpr int threads = 128, minBlocks = 3;
};
template <>
struct LaunchShape<2> {
    static constexpr int threads = 256, minBlocks = 2;
};
template <>
struct LaunchShape<3> {
    static constexpr int threads = 128, minBlocks = 5;
};

// FP32 step over the cell-column pair (step_fast.cuh); same state handling as move_soa_kernel.
template <int SEM, int STORE, int SHAPE, int VARIANT>
__global__ void __launch_bounds__(LaunchShape<SHAPE>::threads, LaunchShape<SHAPE>::minBlocks)
    move_fast_kernel(const wacomm_b200_config cfg,
                                                        const IntervalParams P,
                                                        const FastView<STORE> F, ParticleSoA S,
                                                        const MoveLaunch L) {
    const int count = launch_count(L);
    // block-uniform stride loop (blocks past a device-side list take no turn)
    const int items = (int)(blockDim.x >> 5) * L.lanes;
    for (long long base = (long long)blockIdx.x * items; base < count;
         base += (long long)gridDim.x * items) {
        const unsigned t = launch_item(L, (unsigned)base, (unsigned)count);
        long long cell = -1;
        int steps = 0;
        if (t < (unsigned)count) {
            uint32_t slot = L.order ? L.order[t] : (uint32_t)t;
            ParticleState p;
            p.id = S.id[slot];
            p.k = S.k[slot];
            p.j = S.j[slot];
            p.i = S.i[slot];
            p.health = S.health[slot];
            p.age = S.age[slot];
            p.time = S.time[slot];
            p.type = S.type[slot];
            p.side = S.side[slot];
            double elapsed = P.firstChunk ? P.elapsed0 : S.elapsed[slot];
            steps = move_particle_fast<SEM, STORE, VARIANT>(
                cfg, P, F, Draws{L.draws + slot, L.drawSteps, L.drawStride}, p,
                elapsed, L.err);
            S.k[slot] = p.k;
            S.j[slot] = p.j;
            S.i[slot] = p.i;
            S.health[slot] = p.health;
            S.age[slot] = p.age;
            S.side[slot] = (int8_t)p.side;
            if (!P.lastChunk) S.elapsed[slot] = elapsed;
            if (L.conc && P.lastChunk)
                cell = concentration_cell(p, L.concTimeIndex, F.V.g.sRho, F.V.g.eta, F.V.g.xi);
        }
        if (L.steps) warp_sum_steps(L.steps, steps);
        if (L.conc && P.lastChunk) warp_count(L.conc, cell);
    }
}

template <int SEM, int STORE, int SHAPE, int VARIANT>
cudaError_t launch_move_fast(const wacomm_b200_config &cfg, const IntervalParams &P,
                             const FastView<STORE> &F, const ParticleSoA &S, const MoveLaunch &L,
                             cudaStream_t stream) {
    if (L.count <= 0) return cudaSuccess;
    MoveLaunch M = L;
    int threads;
    spread_launch(L.count, LaunchShape<SHAPE>::threads, M.lanes, threads);
    const long long items = (long long)(threads / 32) * M.lanes * (L.perThread > 1 ? L.perThread : 1);
    const int blocks = launch_blocks(L.count, items);
    FastView<STORE> G = F;
    G.X.K = step_constants(cfg, P, F.V.g.eta, F.V.g.xi);
    move_fast_kernel<SEM, STORE, SHAPE, VARIANT><<<blocks, threads, 0, stream>>>(cfg, P, G, S, M);
    return cudaGetLastError();
}

// Host launchers (one per template instance, defined in the instantiation units).
template <int SEM>
cudaError_t launch_move_soa(const wacomm_b200_config &cfg, const IntervalParams &P,
                            const PackedView &V, const ParticleSoA &S, const MoveLaunch &L,
                            int blockSize, cudaStream_t stream) {
    if (L.count <= 0) return cudaSuccess;
    MoveLaunch M = L;
    int threads;
    spread_launch(L.count, blockSize, M.lanes, threads);
    const int items = threads / 32 * M.lanes;
    const int blocks = launch_blocks(L.count, items);
    const bool keep = keeps_stencil(L.count, V.g.eta, V.g.xi, V.g.sRho);
    if (cfg.driftModel == 1) {
        if (keep) move_soa_kernel<SEM, true, true><<<blocks, threads, 0, stream>>>(cfg, P, V, S, M);
        else move_soa_kernel<SEM, true, false><<<blocks, threads, 0, stream>>>(cfg, P, V, S, M);
    } else {
        if (keep) move_soa_kernel<SEM, false, true><<<blocks, threads, 0, stream>>>(cfg, P, V, S, M);
        else move_soa_kernel<SEM, false, false><<<blocks, threads, 0, stream>>>(cfg, P, V, S, M);
    }
    return cudaGetLastError();
}

}  // namespace wb
