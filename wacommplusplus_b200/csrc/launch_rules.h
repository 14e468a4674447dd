// Rules of the launches that follow from sizes and options alone: plain C++, for the host.
#pragma once

#include <cmath>
#include <cstddef>

#include "wacomm_b200.h"

namespace wb {

constexpr int B200_SMS = 148;

// Two full warps per scheduler: up to here the plain step's records are not sorted, and the reference
// arithmetic keeps its velocity stencil in registers (keeps_stencil).
constexpr int KEEP_RECORDS = 2 * 4 * B200_SMS * 32;
// All resident at once at launch shape 1 of the FP32 step (12 warps per SM).
constexpr int RESIDENT_RECORDS = 12 * B200_SMS * 32;

// Lanes per warp and threads per block (at most maxThreads) of a launch over `count` items: one warp
// per scheduler of the chip before a warp is filled, as blocks of one size on every SM. Such a launch
// is bound by the latency of its substep chain; fewer lanes per warp meet fewer cell changes and
// lines per load. 1,021 records (random walk) per host interval 0.473 -> 0.428 ms, 16,384 in
// reference arithmetic 0.640 -> 0.564 ms; two warps per scheduler: 0.459 and 0.628 ms. From 18,945
// items on the warps are full.
inline void spread_launch(int count, int maxThreads, int &lanes, int &threads) {
    constexpr long long SMS = B200_SMS, WARPS = 4 * SMS;
    const long long per = (count + WARPS - 1) / WARPS;
    lanes = (int)(per < 1 ? 1 : per > 32 ? 32 : per);
    const long long warps = ((long long)count + lanes - 1) / lanes, even = 32 * ((warps + SMS - 1) / SMS);
    threads = even < maxThreads ? (int)even : maxThreads;
}

// Bins of the counting sort by forcing cell: one per cell or, with levels > 1, per vertical level
// of a cell; each split by release time into `late` parts (the first: released by the interval's
// start, the others: equal parts of the interval), then one last bin for the records that take no
// step in the interval (off the grid, or released at or after its end).
struct SortBins {
    int eta, xi, levels, late;
    double start, end;  // of a forward interval; infinite: no release test
    size_t count() const { return (size_t)eta * xi * levels * late + 1; }
};

// The bins `count` records are sorted into on a grid of sRho levels for a launch of `substeps`;
// `forward`: records are released in the interval's direction.
//
// Levels are told apart from one record per bin on: the forcing records of a cell's levels lie apart
// in memory, so a warp of one cell on several levels reads several lines per load, and the FP32 step
// over FP32 storage is bound by its L1 wavefronts (83 % of the L1 throughput with four levels mixed).
// 16.8 M records on 128 x 128 x 10 with the upper four levels in use: 46.9 ms per host interval
// against 53.6 ms by cell alone; 1.05 M with the random walk: 10.0 against 11.1 ms. With fewer
// records than bins a warp meets as many lines either way and the larger scan costs: 2 M records on
// 640 x 768 x 24, 11.8 M bins: 0.6 % slower with levels.
//
// Records released during the interval take fewer substeps the later they come; the lanes of a warp run
// as long as its longest. Parts of the interval are told apart while the bins stay below four per
// record (their scan is cheap): 2 M records released in the first of two hours on 640 x 768 x 24, 8
// parts: 31.1 -> 27.4 ms; 400,000 drift records of 32 scenarios over six hours 11.6 -> 11.4 ms; no
// change where all are released.
//
// A launch of one to three substeps does not bring in the larger scan: 4 M records on 128 x 128 x 10, one
// substep 0.94 ms by cell and 1.03 split, four 1.28 and 1.24 ms.
inline SortBins sort_bins(int eta, int xi, int sRho, size_t count, bool forward, double substeps) {
    const size_t split = (size_t)eta * xi * sRho + 1;
    SortBins B{eta, xi, 1, 1, -INFINITY, INFINITY};
    if (substeps < 4) return B;
    if (split <= count && split < ((size_t)1 << 31)) B.levels = sRho;
    const size_t cells = (size_t)eta * xi * B.levels;
    while (forward && B.late < 16 && cells * 2 * B.late <= 4 * count &&
           cells * 2 * B.late < ((size_t)1 << 31))
        B.late *= 2;
    return B;
}

// Whether the reference arithmetic keeps the velocity stencil of `count` records in registers (8 warps per
// SM) instead of reading it twice per substep (16 warps per SM): where one or two warps per scheduler hold
// all records, and up to a record per cell and level. With fewer, the lanes of a warp share no lines, and
// the stencils of 512 threads (384 bytes of lines each) do not fit L1. Whole interval read / kept, 200 x
// 200 x 20: 100,000 records 1.98 / 1.24 ms, 500,000 5.55 / 5.09, 1.5 M 12.5 / 14.3; 300 x 300 x 20: 100,000
// 2.37 / 1.35, 1.5 M 15.6 / 14.5; 128 x 128 x 10: 100,000 1.30 / 1.17, 200,000 2.06 / 2.21 ms.
inline bool keeps_stencil(int count, int eta, int xi, int sRho) {
    return count <= KEEP_RECORDS || count <= (long long)eta * xi * sRho;
}

// Blocks of `items` work items each that cover `count` (1 to 2^31 - 1).
inline int launch_blocks(int count, long long items) {
    return (int)(((long long)count + items - 1) / items);
}

// Up to here the move with the draws ahead is the faster one (whole interval of 120 substeps, with /
// without): 1,021 records 0.26 / 0.43 ms, 20,011 0.40 / 0.51 ms, 30,000 0.45 / 0.52 ms, 45,000 0.54 /
// 0.56 ms, 59,000 0.59 / 0.56 ms: beyond, the chip is busy with substeps and the draws cost the same
// either way. The draws of 120 substeps stay in L2 (77 MB at the limit); longer intervals gain less
// (601 substeps: 20,000 records, 192 MB, 1.50 ms; 27,915 records, the largest buffer, 1.64 ms against
// 1.74 ms for one more drawn in the step).
constexpr size_t DRAW_AHEAD_RECORDS = 40000;
constexpr double DRAW_AHEAD_BYTES = 256.0 * (1 << 20);

// Substeps whose normals are drawn ahead (draw_normals) of an interval of `length` seconds over `count`
// records; 0: the step draws them itself. The form that reads them has one launch shape, so an explicit
// launch_shape keeps the draws in the step.
inline unsigned draw_steps(const wacomm_b200_options &opt, const wacomm_b200_config &cfg, double length,
                           size_t count) {
    const bool diffuse = cfg.random && (cfg.trackingDirection > 0 || cfg.backwardDiffusion);
    const bool plain = cfg.driftModel != 1 && !(cfg.leewayJibeProbabilityHourly > 0);
    if (!diffuse || !plain || opt.rng != WACOMM_B200_RNG_REFERENCE ||
        opt.arithmetic != WACOMM_B200_ARITH_FP32 || opt.launch_shape != WACOMM_B200_LAUNCH_SHAPE_AUTO)
        return 0;
    // floor(elapsed / dti) of a substep that starts before the end; the quotient may round up to the
    // next whole number there
    const double steps = std::ceil(length / cfg.dti) + 1;
    constexpr size_t DRAW_BYTES = 4 * sizeof(float);  // three normals and padding
    if (!(steps >= 2 && steps <= 1e6) || count > DRAW_AHEAD_RECORDS ||
        steps * count * DRAW_BYTES > DRAW_AHEAD_BYTES)
        return 0;
    return (unsigned)steps;
}

// Whether the drop-in launcher packs the forcing pair of `count` records into `bytes` of scratch from
// the caller's memory pool. Packing saves 10 ns and more per record and hour of 120 substeps (at least
// 0.4 ms per call) and costs 4 us per MB, and 9 us more per MB in a program that synchronizes after the
// call, when the pool gives its memory back and maps it anew. Up to 80 MiB it is worth it for any
// count: 1,000 records on 990,000 nodes 1.00 -> 0.84 ms per queued call, 1.45 -> 1.77 ms per
// synchronized one; on 840,000 nodes 0.99 -> 0.59 and 1.43 -> 1.31 ms (intervals of a few substeps pay the
// pack without the gain: four on 990,000 nodes 0.2 -> 0.4 and 0.6 -> 1.3 ms). Beyond, from a node record and
// its tables per record on, where synchronized calls of four substeps lose little, too (records, nodes,
// synchronized / queued read from the window -> packed): 4 M on 5.5 M 82 / 83 -> 48 / 44 ms, four substeps
// 4.4 / 3.6 -> 8.3 / 3.6; 200,000 on 1.94 M 5.0 / 4.6 -> 6.0 / 3.8 ms, four substeps 0.7 / 0.3 -> 2.4 /
// 0.7; 500,000 on 12.3 M 11.7 / 11.1 -> 18.5 / 10.8 ms, four substeps 1.0 / 0.6 -> 11 / 3.3. At most 1 GiB
// is asked for.
constexpr size_t PACK_BYTES = (size_t)80 << 20, PACK_BYTES_PER_RECORD = 96, PACK_BYTES_MOST = (size_t)1 << 30;

inline bool packs_pair(size_t bytes, size_t count) {
    return bytes <= PACK_BYTES || (bytes <= PACK_BYTES_MOST && bytes / PACK_BYTES_PER_RECORD <= count);
}

}  // namespace wb
