// FP32 move kernels (step_fast.cuh) for one rule set and one forcing storage: the instances of
// move_fast_kernel by launch shape and compiled form. Each move_f32_<rules>_<storage>.cu unit
// instantiates move_f32_unit for its pair, so the kernels build in parallel.
#pragma once

#include "engine.h"
#include "move_kernels.cuh"

namespace wb {

template <int STORE>
inline FastView<STORE> fast_view(const PackedArgs &A) {
    FastView<STORE> F;
    F.V = packed_view(A);
    F.X.invMetric = A.invMetric;
    F.X.depthIntervals = A.depthIntervalsF;
    F.X.cfgDevice = A.cfgDevice;
    F.C.eta = A.eta;
    F.C.xi = A.xi;
    F.C.sW = A.sW;
    F.C.columns = static_cast<const CellQuad<STORE> *>(A.cells);
    F.C.surface = static_cast<const CellSurface *>(A.cellSurface);
    return F;
}

// The compiled form a run needs (VAR_*).
inline int fast_variant(const wacomm_b200_config &cfg, int direction) {
    const bool diffuse = cfg.random && (direction > 0 || cfg.backwardDiffusion);
    const bool drift = cfg.driftModel == 1, jibe = cfg.leewayJibeProbabilityHourly > 0;
    const bool plainDrift = cfg.observationalCalibrationRegionCount == 0 &&
                            !(cfg.windErrorStdDev > 0) && !cfg.leewayCoefficientEnsemble;
    if (jibe || (drift && !plainDrift)) return VAR_FULL;
    if (drift) return VAR_DRIFT;
    return diffuse ? VAR_DIFFUSE : VAR_LEAN;
}

// Shapes 1, 2 and 3 carry every form; shape 0 the full one. A negative shape picks by form, the
// register needs deciding (move kernel, shapes 1 / 2 / 3): lean, 4.2 M records 9.81 / 9.91 / 9.80 ms
// (FP16 storage 10.46 / 10.62 / 10.29); random walk (Philox), 1.05 M 4.08 / 3.55 / 3.61 ms; leeway
// drift, 400,000 2.45 / 2.21 / 2.96 ms; full 5.14 / 5.74 / 6.90 ms (spills at shapes 2 and 3).
template <int SEM, int STORE>
cudaError_t move_f32_unit(int shape, const wacomm_b200_config &cfg, const IntervalParams &P,
                          const PackedArgs &A, const ParticleSoA &S, const MoveLaunch &L,
                          cudaStream_t stream) {
    FastView<STORE> F = fast_view<STORE>(A);
    const int variant = fast_variant(cfg, P.direction);
    // small launches under the automatic shape (draw_steps), bound by latency
    if (variant == VAR_DIFFUSE && L.draws)
        return launch_move_fast<SEM, STORE, 1, VAR_DRAWN>(cfg, P, F, S, L, stream);
    // records that are all resident at once at shape 1 (12 warps per SM): nothing is gained by more
    // warps, and its registers shorten the substep's chain: 600 records 0.130 ms (shape 3: 0.156),
    // 16,000 0.173 (0.196), 40,000 0.189 (0.212); random walk 0.263 (shape 2: 0.294)
    if (shape < 0 && !L.countDevice && L.count <= RESIDENT_RECORDS) shape = 1;
    if (shape < 0) shape = variant == VAR_LEAN ? 3 : variant == VAR_FULL ? 1 : 2;
    switch (shape) {
        case 0: return launch_move_fast<SEM, STORE, 0, VAR_FULL>(cfg, P, F, S, L, stream);
        case 3:
            switch (variant) {
                case VAR_LEAN: return launch_move_fast<SEM, STORE, 3, VAR_LEAN>(cfg, P, F, S, L, stream);
                case VAR_DIFFUSE: return launch_move_fast<SEM, STORE, 3, VAR_DIFFUSE>(cfg, P, F, S, L, stream);
                case VAR_DRIFT: return launch_move_fast<SEM, STORE, 3, VAR_DRIFT>(cfg, P, F, S, L, stream);
                default: return launch_move_fast<SEM, STORE, 3, VAR_FULL>(cfg, P, F, S, L, stream);
            }
        case 2:
            switch (variant) {
                case VAR_LEAN: return launch_move_fast<SEM, STORE, 2, VAR_LEAN>(cfg, P, F, S, L, stream);
                case VAR_DIFFUSE: return launch_move_fast<SEM, STORE, 2, VAR_DIFFUSE>(cfg, P, F, S, L, stream);
                case VAR_DRIFT: return launch_move_fast<SEM, STORE, 2, VAR_DRIFT>(cfg, P, F, S, L, stream);
                default: return launch_move_fast<SEM, STORE, 2, VAR_FULL>(cfg, P, F, S, L, stream);
            }
        default:
            switch (variant) {
                case VAR_LEAN: return launch_move_fast<SEM, STORE, 1, VAR_LEAN>(cfg, P, F, S, L, stream);
                case VAR_DIFFUSE: return launch_move_fast<SEM, STORE, 1, VAR_DIFFUSE>(cfg, P, F, S, L, stream);
                case VAR_DRIFT: return launch_move_fast<SEM, STORE, 1, VAR_DRIFT>(cfg, P, F, S, L, stream);
                default: return launch_move_fast<SEM, STORE, 1, VAR_FULL>(cfg, P, F, S, L, stream);
            }
    }
}

}  // namespace wb
