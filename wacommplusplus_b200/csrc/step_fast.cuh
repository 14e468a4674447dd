// The FP32 particle step: the same algorithm as step.cuh with FP32 interpolation and metric,
// FP64 kept for the position accumulation, the closures and the interval clock.
//
// Differences from the reference arithmetic (all below the reference's own CPU/GPU snapshot
// tolerance once forcing is FP32, and stated per configuration in the parity tests):
//   * corner weights, time blends and the velocity/diffusivity sums are FP32 with fused
//     multiply-adds;
//   * cell sizes come from a per-cell table of reciprocals, so index increments are products
//     (u dt / dx) instead of double divisions, and the midpoint stage is written directly in
//     index units (u* dt / dx*, algebraically the reference's s u* dt dx/dx* / dx);
//   * the time weight uses a multiply by 1/length.
// Host and device rules keep their differences in closures, level checks and metric formula.
#pragma once

#include "step.cuh"

namespace wb {

// Constants of a launch in the precision the step uses them in, computed on the host: read as constant
// operands, where a conversion of the FP64 parameter would cost a register over the substep loop or,
// repeated in it, a quarter-rate instruction (4.2 M records, lean: 9.96 -> 9.80 ms, FP16 storage 10.50 ->
// 10.29 ms).
struct StepConstants {
    double jEdge, iEdge;  // last node of each axis
    double invLength;     // 1 / length of the interval (0 for an empty one)
    double ageSafe;       // age below which the lazy survival tests cannot change their outcome
    float dti, sv, shore, direction, crid;
};

inline StepConstants step_constants(const wacomm_b200_config &cfg, const IntervalParams &P, int eta,
                                    int xi) {
    StepConstants K;
    K.jEdge = eta - 1;
    K.iEdge = xi - 1;
    K.invLength = P.length == 0 ? 0.0 : 1.0 / P.length;
    K.ageSafe = fmin(P.ageKillLo, P.ageUnder);
    K.dti = (float)cfg.dti;
    K.sv = (float)cfg.sv;
    K.shore = (float)cfg.shoreLimit;
    K.direction = (float)P.direction;
    K.crid = (float)cfg.crid;
    return K;
}

struct FastExtras {
    StepConstants K;
    const float2 *invMetric;     // [eta][xi] {1/xdist, 1/ydist}
    const float *depthIntervals; // [sW-1]
    const wacomm_b200_config *cfgDevice;  // device copy of the run parameters
};

template <int STORE>
struct FastView {
    PackedView V;          // grid, wind/Stokes pair, lon/lat (drift model)
    CellView<STORE> C;     // cell-column layout: velocity stencil and surface
    FastExtras X;
};

// Space-time weights of the 8 stencil values of one field: (1-a) w_c for record t0 and a w_c for
// record t1, corners (j,i), (j+1,i), (j+1,i+1), (j,i+1).
struct Weights8 {
    float p1, p2, p3, p4, q1, q2, q3, q4;
};

// The products run in pairs on the packed FP32x2 multiply of sm_100 (the same roundings).
__device__ __forceinline__ Weights8 weights8(float jF, float iF, float a) {
    const float oi = 1.f - iF, oj = 1.f - jF, b = 1.f - a;
    const float2 w12 = __fmul2_rn(make_float2(oi, oi), make_float2(oj, jF));
    const float2 w34 = __fmul2_rn(make_float2(iF, iF), make_float2(jF, oj));
    const float2 bb = make_float2(b, b), aa = make_float2(a, a);
    const float2 p12 = __fmul2_rn(bb, w12), p34 = __fmul2_rn(bb, w34);
    const float2 q12 = __fmul2_rn(aa, w12), q34 = __fmul2_rn(aa, w34);
    return Weights8{p12.x, p12.y, p34.x, p34.y, q12.x, q12.y, q34.x, q34.y};
}

// The 8 products summed as pairs of corners (c1, c2 | c3, c4) with the packed FP32x2 multiply
// and multiply-add of sm_100, record t0 and record t1 apart, then the four partial sums.
__device__ __forceinline__ float blend(const QuadPair &q, const Weights8 &w) {
    float2 x = __fmul2_rn(make_float2(q.t0.c1, q.t0.c2), make_float2(w.p1, w.p2));
    float2 y = __fmul2_rn(make_float2(q.t1.c1, q.t1.c2), make_float2(w.q1, w.q2));
    x = __ffma2_rn(make_float2(q.t0.c3, q.t0.c4), make_float2(w.p3, w.p4), x);
    y = __ffma2_rn(make_float2(q.t1.c3, q.t1.c4), make_float2(w.q3, w.q4), y);
    const float2 t = __fadd2_rn(x, y);
    return t.x + t.y;
}

// Bilinear h + zeta@t0 and zeta@t1 - zeta@t0 at a fractional position of a cell (FP32); the water
// column height at time weight a is s + a d.
struct SurfaceSums {
    float s, d;
    __device__ __forceinline__ float height(float a) const { return fmaf(a, d, s); }
};

// Corner weights in pairs {w1, w2}, {w3, w4} (packed FP32x2 multiplies).
__device__ __forceinline__ void corner_pairs(float jF, float iF, float2 &w12, float2 &w34) {
    const float oi = 1.f - iF, oj = 1.f - jF;
    w12 = __fmul2_rn(make_float2(oi, oi), make_float2(oj, jF));
    w34 = __fmul2_rn(make_float2(iF, iF), make_float2(jF, oj));
}

__device__ __forceinline__ SurfaceSums surface_from(const CellSurface &c, float jF, float iF) {
    float2 w12, w34;
    corner_pairs(jF, iF, w12, w34);
    float2 s = __fmul2_rn(make_float2(c.s0.x, c.s0.y), w12);
    float2 d = __fmul2_rn(make_float2(c.dz.x, c.dz.y), w12);
    s = __ffma2_rn(make_float2(c.s0.z, c.s0.w), w34, s);
    d = __ffma2_rn(make_float2(c.dz.z, c.dz.w), w34, d);
    return SurfaceSums{s.x + s.y, d.x + d.y};
}

// Current (u, v, w) at time weight a and a fractional position of the stencil's cell and level.
__device__ __forceinline__ void current_at(const Stencil &s, float a, float kF, float jF, float iF,
                                           float &uu, float &vv, float &ww) {
    const Weights8 w = weights8(jF, iF, a);
    uu = blend(s.u, w);
    vv = blend(s.v, w);
    const float up = blend(s.wUp, w), lo = blend(s.wLo, w);
    ww = fmaf(lo - up, kF, up);
}

// Bilinear value of t0 + a (t1 - t0) over the corners, two corners per packed FP32x2 operation.
__device__ __forceinline__ float changed(const QuadPair &q, float2 a2, float2 w12, float2 w34) {
    const float2 lo0 = make_float2(q.t0.c1, q.t0.c2), hi0 = make_float2(q.t0.c3, q.t0.c4);
    const float2 dLo = __fadd2_rn(make_float2(q.t1.c1, q.t1.c2), make_float2(-lo0.x, -lo0.y));
    const float2 dHi = __fadd2_rn(make_float2(q.t1.c3, q.t1.c4), make_float2(-hi0.x, -hi0.y));
    const float2 lo = __ffma2_rn(a2, dLo, lo0), hi = __ffma2_rn(a2, dHi, hi0);
    const float2 x = __ffma2_rn(hi, w34, __fmul2_rn(lo, w12));
    return x.x + x.y;
}

// current_at in the lean form's order of operations for a midpoint in its start column: the time
// blend first, then the corners.
__device__ __forceinline__ void current_changed(const Stencil &s, float a, float kF, float jF,
                                                float iF, float &uu, float &vv, float &ww) {
    float2 w12, w34;
    corner_pairs(jF, iF, w12, w34);
    const float2 a2 = make_float2(a, a);
    uu = changed(s.u, a2, w12, w34);
    vv = changed(s.v, a2, w12, w34);
    const float up = changed(s.wUp, a2, w12, w34), lo = changed(s.wLo, a2, w12, w34);
    ww = fmaf(lo - up, kF, up);
}

// AKT at time weight a and a fractional position of a cell and level (one stencil read).
template <int STORE>
__device__ __forceinline__ float akt_at_cell(const CellView<STORE> &C, uint32_t column, float a,
                                             float kF, float jF, float iF) {
    QuadPair up, lo;
    C.akt(column, up, lo);
    const Weights8 w = weights8(jF, iF, a);
    const float au = blend(up, w), al = blend(lo, w);
    return fmaf(al - au, kF, au);
}

// Whether a position lies in the interpolation cells of an axis whose last node is `edge`: the cell
// floor(x) has floor(x) >= 0 and floor(x) + 1 <= edge. Under the device rules a NaN counts as cell
// 0 (to_index).
template <int SEM>
__device__ __forceinline__ bool on_axis(double x, double edge) {
    return SEM == SEM_HOST ? (x >= 0.0 && x < edge) : !(x < 0.0) && !(x >= edge);
}

// Cell index and fraction of a position on the axis (on_axis).
template <int SEM>
__device__ __forceinline__ int split_axis(double x, float &fraction) {
    const double shifted = __dadd_rd(x, INTEGER_SHIFT);
    fraction = (float)(x - (shifted - INTEGER_SHIFT));
    const int index = __double2loint(shifted);
    return SEM == SEM_HOST || x == x ? index : 0;
}

// Level index ceil(k) and the fraction ceil(k) - k below it.
template <int SEM>
__device__ __forceinline__ int split_level(double k, float &fraction) {
    if (fabs(k) < 2147483648.0) {
        const double shifted = __dadd_ru(k, INTEGER_SHIFT);
        fraction = (float)((shifted - INTEGER_SHIFT) - k);
        return __double2loint(shifted);
    }
    const double up = ceil(k);
    fraction = (float)(up - k);
    return to_index<SEM>(up);
}

// Leeway and Stokes velocity of a drifting object (the drift branch of advective_velocity) in FP32:
// wind and Stokes interpolated from the environment pair, the leeway regression of the object's
// catalogue row (computeLeeway, DriftModel.hpp:204-219) on the interpolated 10-m wind. The
// position-dependent parts (calibration regions, wind-error fields) and the coefficient ensemble
// exist only in the FULL form, run in FP64 there and only when the run configures them.
template <bool FULL, class View>
__device__ __forceinline__ void drift_velocity(const wacomm_b200_config &cfg, const IntervalParams &P,
                                            const View &V, uint64_t id, int type, int side,
                                            int jI, float jF, int iI, float iF, float a,
                                            double elapsed, double physicalTime, double stepDt,
                                            float &du, float &dv) {
    float windU = (float)cfg.windU10, windV = (float)cfg.windV10;
    EnvPair e1{}, e2{}, e3{}, e4{};
    if (V.hasWindU || V.hasWindV || V.hasStokes) {
        e1 = V.environment(jI, iI);
        e2 = V.environment(jI + 1, iI);
        e3 = V.environment(jI + 1, iI + 1);
        e4 = V.environment(jI, iI + 1);
    }
    const float w1 = (1.f - iF) * (1.f - jF), w2 = (1.f - iF) * jF, w3 = iF * jF, w4 = iF * (1.f - jF);
    if (V.hasWindU)
        windU = at_f32(e1.wu0 * w1 + e2.wu0 * w2 + e3.wu0 * w3 + e4.wu0 * w4,
                       e1.wu1 * w1 + e2.wu1 * w2 + e3.wu1 * w3 + e4.wu1 * w4, a);
    if (V.hasWindV)
        windV = at_f32(e1.wv0 * w1 + e2.wv0 * w2 + e3.wv0 * w3 + e4.wv0 * w4,
                       e1.wv1 * w1 + e2.wv1 * w2 + e3.wv1 * w3 + e4.wv1 * w4, a);
    if (FULL && (cfg.observationalCalibrationRegionCount > 0 || cfg.windErrorStdDev > 0)) {
        const double jd = jF, id_ = iF;
        double longitude = V.lon(jI, iI) * (1.0 - id_) * (1.0 - jd) + V.lon(jI + 1, iI) * (1.0 - id_) * jd +
                           V.lon(jI + 1, iI + 1) * id_ * jd + V.lon(jI, iI + 1) * id_ * (1.0 - jd);
        double latitude = V.lat(jI, iI) * (1.0 - id_) * (1.0 - jd) + V.lat(jI + 1, iI) * (1.0 - id_) * jd +
                          V.lat(jI + 1, iI + 1) * id_ * jd + V.lat(jI, iI + 1) * id_ * (1.0 - jd);
        double stdDev = cfg.windErrorStdDev, corr = cfg.windErrorComponentCorrelation;
        double spatial = cfg.windErrorSpatialScale, temporal = cfg.windErrorTemporalScale;
        int region = calibration_region(cfg, longitude, latitude);
        if (region >= 0) {
            const wacomm_b200_calibration_region &g = cfg.observationalCalibrationRegions[region];
            stdDev = g.windErrorStdDev;
            corr = g.windErrorComponentCorrelation;
            spatial = g.windErrorSpatialScale;
            temporal = g.windErrorTemporalScale;
        }
        if (stdDev > 0) {
            uint64_t substep = (uint64_t)floor(elapsed / cfg.dti);
            double when = physicalTime + .5 * P.direction * stepDt;
            double first = forcing_error_normal(cfg.randomSeed, id, P.intervalKey, substep,
                                                WIND_U_COMPONENT, longitude, latitude, when,
                                                spatial, temporal);
            double second = forcing_error_normal(cfg.randomSeed, id, P.intervalKey, substep,
                                                 WIND_V_COMPONENT, longitude, latitude, when,
                                                 spatial, temporal);
            windU = (float)(windU + stdDev * first);
            windV = (float)(windV + stdDev * correlated_normal(first, second, corr));
        }
    }
    float dn = 0.f, cn = 0.f;
    if (FULL && cfg.leewayCoefficientEnsemble) {
        uint64_t ens = key_prefix(cfg.randomSeed, id, ENSEMBLE_INTERVAL, 0);
        double n0 = prefix_normal(ens, 0);
        dn = (float)n0;
        cn = (float)correlated_normal(n0, prefix_normal(ens, 1), cfg.leewayResidualCorrelation);
    }
    du = dv = 0.f;
    const float speed = sqrtf(windU * windU + windV * windV);
    if (speed >= 1.0e-12f && side != 0 && type >= 0 && type <= 22) {
        const float *c = c_leeway_catalogue_f32[type];
        const bool right = side == 1;
        const float rs = 1.0f / speed;
        const float ux = windU * rs, uy = windV * rs;
        // (the ensemble's terms only where there is one)
        float downwind = __ldg(c + 0) * speed + __ldg(c + 1);
        float crosswind = right ? __ldg(c + 3) * speed + __ldg(c + 4) : __ldg(c + 6) * speed + __ldg(c + 7);
        if (FULL) {
            downwind += __ldg(c + 2) * dn;
            crosswind += right ? __ldg(c + 5) * cn : -__ldg(c + 8) * cn;
        }
        du = downwind * ux - crosswind * uy;
        dv = downwind * uy + crosswind * ux;
    }
    if (V.hasStokes) {
        du += at_f32(e1.su0 * w1 + e2.su0 * w2 + e3.su0 * w3 + e4.su0 * w4,
                     e1.su1 * w1 + e2.su1 * w2 + e3.su1 * w3 + e4.su1 * w4, a);
        dv += at_f32(e1.sv0 * w1 + e2.sv0 * w2 + e3.sv0 * w3 + e4.sv0 * w4,
                     e1.sv1 * w1 + e2.sv1 * w2 + e3.sv1 * w3 + e4.sv1 * w4, a);
    }
}

__device__ __forceinline__ float signf_of(float a, float b) {
    return fabsf(a) * (float)((b > 0.f) - (b < 0.f));
}

// The normals of a record drawn ahead (VAR_DRAWN): those of substep s at at[s * stride].
struct Draws {
    const float4 *at;
    unsigned steps, stride;
};

// VARIANT (VAR_*): the branches the run parameters can reach are compiled in, the rest out --
// fewer registers and a smaller instruction footprint for the common runs.
//
// A particle stays in its cell and level for tens of substeps, so the velocity stencil, the surface
// record and the metric of a cell are kept in registers and read again only by the lanes that
// changed cell or level: the L1 then serves a few lines per substep instead of 14 loads of every
// lane, and a midpoint across a cell edge takes the same arithmetic as one inside (the new cell's
// stencil takes the kept one's place; the destination is mostly in it too). Measured on a turning
// gyre flow, move kernel: 1.05 M records, FP32 storage 3.87 -> 2.57 ms (L1 throughput 83 -> 19 %,
// 521 -> 490 instructions per particle-step, issue 50 -> 70 %); random walk with the reference
// keys, 262,144 records 2.47 -> 1.76 ms; leeway drift, 400,000 records 3.00 -> 2.28 ms. Bound now
// by instruction issue.
template <int SEM, int STORE, int VARIANT>
__device__ int move_particle_fast(const wacomm_b200_config &cfg, const IntervalParams &P,
                                  const FastView<STORE> &F, const Draws draws, ParticleState &p,
                                  double &elapsed, int *err) {
    const PackedView &V = F.V;
    const CellView<STORE> &C = F.C;
    const StepConstants &K = F.X.K;
    const int xi = V.g.xi, sW = V.g.sW;
    const double kLower = P.kLower, length = P.length;
    const int direction = P.direction;
    const bool midpoint = cfg.integrator == INTEGRATOR_MIDPOINT;
    constexpr bool canDiffuse = VARIANT != VAR_LEAN, full = VARIANT == VAR_FULL;
    constexpr bool canDrift = VARIANT == VAR_DRIFT || full, drawn = VARIANT == VAR_DRAWN;
    const bool diffuse = canDiffuse && cfg.random && (direction > 0 || cfg.backwardDiffusion);
    const bool drift = canDrift && cfg.driftModel == 1 && p.type != 0;
    const bool jibe = full && cfg.leewayJibeProbabilityHourly > 0 && p.type != 0;
    if (drift && SEM == SEM_HOST && (p.type < 0 || p.type > 22)) atomicOr(err, ERR_DRIFT_OBJECT);
    bool lazy = false;
    int steps = 0;
    // Substeps left in which the lazy survival tests cannot change their outcome (age below
    // min(ageKillLo, ageUnder): neither dead nor without health), counted when the particle turns
    // lazy, two substeps short of the bound for rounding; skipped while it lasts and no closure
    // has ended the lazy tracking.
    int youngLeft = 0;

    if (P.firstChunk) {
        if (p.k > 0) close_upper(cfg, p.k, p.health, lazy);
        if (p.k < kLower) close_lower(cfg, kLower, p.k, p.health, lazy);
    }
    const uint64_t prefix = fold(fold(mix64(cfg.randomSeed), p.id), (uint64_t)P.intervalKey);
    const uint64_t philoxKey = p.id ^ mix64(cfg.randomSeed);
    const double stop = P.chunkEnd < length ? P.chunkEnd : length;
    // Not yet released: the first substep starts at the release time (the clock only advances from
    // there, so the test is not repeated).
    if (direction > 0 && elapsed < stop && p.time > P.start + elapsed)
        elapsed = fmin(length, p.time - P.start);

    // The kept records: stencil of (cell, level) keptColumn, surface and metric of keptCell.
    constexpr bool lean = VARIANT == VAR_LEAN;
    constexpr uint32_t NONE = 0xffffffffu;
    Stencil kept;
    CellSurface surf;
    float2 metric;
    uint32_t keptColumn = NONE, keptCell = NONE;
    auto keep_column = [&](uint32_t column) {
        if (column != keptColumn) {
            C.stencil(column, kept);
            keptColumn = column;
        }
    };
    auto keep_cell = [&](uint32_t cell) {
        if (cell != keptCell) {
            surf = C.surf(cell);
            metric = __ldg(F.X.invMetric + cell);
            keptCell = cell;
        }
    };
    // Surface sums, cell and fractional position of the previous step's destination, valid while
    // the particle still sits there: the next step starts from the same values.
    SurfaceSums here{0.f, 0.f};
    int jI = 0, iI = 0;
    float jF = 0.f, iF = 0.f;
    bool haveCarried = false;

    while (elapsed < stop) {
        const double left = length - elapsed;
        double stepDt = cfg.dti;
        float dt = K.dti;
        if (left < cfg.dti) {
            stepDt = left;
            dt = (float)stepDt;
        }
        const double physicalTime = P.start + direction * elapsed;
        if (!(lazy && youngLeft > 0)) {
            bool dead = lazy ? (p.age >= P.ageKillHi ||
                                (p.age > P.ageKillLo && exp(-p.age / cfg.tau0) < cfg.survprob))
                             : p.health < cfg.survprob;
            if (dead) {
                p.health = -1;
                lazy = false;
                elapsed = length;
                break;
            }
        }
        float kF;
        const int kI = split_level<SEM>(p.k, kF);
        bool valid = !(SEM == SEM_DEVICE && (kI > 0 || kI <= -sW + 1));
        if (!haveCarried) {
            valid = valid && on_axis<SEM>(p.j, K.jEdge) && on_axis<SEM>(p.i, K.iEdge);
            if (valid) {
                jI = split_axis<SEM>(p.j, jF);
                iI = split_axis<SEM>(p.i, iF);
                keep_cell((uint32_t)(jI * xi + iI));
                here = surface_from(surf, jF, iF);
            }
        }
        if (!valid) {
            p.health = -1;
            lazy = false;
            elapsed = length;
            break;
        }
        steps++;
        // the substep index keys the reference draws and the jibe draw; Philox streams are keyed
        // on the step's elapsed time instead (unique per step, no division)
        uint64_t stepKey = 0;
        const bool philox = P.rng == WACOMM_B200_RNG_PHILOX;
        float4 normals;
        if (drawn) {
            const unsigned substep = (unsigned)floor(elapsed / cfg.dti);
            const unsigned last = draws.steps - 1;
            normals = __ldg(draws.at + (size_t)(substep < last ? substep : last) * draws.stride);
        } else if ((diffuse && !philox) || jibe) {
            stepKey = fold(prefix, (uint64_t)floor(elapsed / cfg.dti));
        }
        const float alpha = (float)((elapsed + 0.5 * stepDt) * K.invLength);
        const float hc = here.height(alpha);
        if (hc <= K.shore && cfg.horizontalClosure == CLOSURE_KILL) {
            p.health = -1;
            lazy = false;
            if (SEM == SEM_DEVICE) {
                elapsed = length;
                break;
            }
        }
        const int kM = mem_level(kI, sW);
        const uint32_t startCell = (uint32_t)(jI * xi + iI);
        const uint32_t startColumn = startCell * (uint32_t)sW + (uint32_t)(kM + sW - 1);
        const float2 inv = metric;
        const float depthHere = __ldg(F.X.depthIntervals + (kM + sW - 2));
        const float sa = midpoint ? (float)(elapsed * K.invLength) : alpha;
        float uu, vv, ww;
        keep_column(startColumn);
        current_at(kept, sa, kF, jF, iF, uu, vv, ww);
        if (drift) {
            float du, dv;
            drift_velocity<full>(cfg, P, V, p.id, p.type, p.side, jI, jF, iI, iF, sa, elapsed,
                           physicalTime, stepDt, du, dv);
            uu += du;
            vv += dv;
        }
        float rx = 0.f, ry = 0.f, rz = 0.f;
        if (diffuse) {
            const float aa = akt_at_cell(C, startColumn, alpha, kF, jF, iF);
            float sigmaDepth = (float)(cfg.sigma * (1 - p.k * P.invKLower));
            const float scale = dt == K.dti ? 1.f : sqrtf(dt / K.dti);
            float n0, n1, n2;
            if (drawn) {
                n0 = normals.x;
                n1 = normals.y;
                n2 = normals.z;
            } else if (philox) {
                philox_normals3(philoxKey, P.intervalKey, (uint64_t)__double_as_longlong(elapsed),
                                n0, n1, n2);
            } else {
                n0 = prefix_normal_f32(stepKey, 0);
                n1 = prefix_normal_f32(stepKey, 1);
                n2 = prefix_normal_f32(stepKey, 2);
            }
            const float2 rxy = __fmul2_rn(
                __fmul2_rn(make_float2(sigmaDepth, sigmaDepth), make_float2(n0, n1)),
                make_float2(scale, scale));
            rx = rxy.x;
            ry = rxy.y;
            rz = sigmaDepth * n2 * aa * K.crid * scale;
        }
        const float zdist = hc * depthHere;
        const float rzdist = __frcp_rn(zdist);
        // index increments (i, j) and the vertical leap in metres
        float dI, dJ, zleap;
        if (midpoint) {
            float kHalf = K.direction * (K.sv + ww) * 0.5f * dt;
            if (fabsf(kHalf) > zdist) kHalf = signf_of(zdist, kHalf);
            // (direction u 0.5 dt) / dx for i and j as one packed FP32x2 chain (the same roundings)
            const float2 half = __fmul2_rn(
                __fmul2_rn(__fmul2_rn(make_float2(K.direction * uu, K.direction * vv),
                                      make_float2(0.5f, 0.5f)),
                           make_float2(dt, dt)),
                inv);
            const double iMid = p.i + (double)half.x;
            const double jMid = p.j + (double)half.y;
            const double kMid = fmin(0.0, fmax(kLower, p.k + (double)(kHalf * rzdist)));
            // the midpoint, or the start where the midpoint has no water
            int jMI = jI, iMI = iI, kMI = kM;
            float jMF = jF, iMF = iF, kMF = kF, hcMid = 0.f;
            float2 im = inv;
            float um, vm, wm;
            bool moved = false;  // the lean form's lanes whose midpoint left the kept column
            bool midValid = on_axis<SEM>(jMid, K.jEdge) && on_axis<SEM>(iMid, K.iEdge);
            if (midValid) {
                float jf, if_;
                const int j = split_axis<SEM>(jMid, jf), i = split_axis<SEM>(iMid, if_);
                keep_cell((uint32_t)(j * xi + i));
                hcMid = surface_from(surf, jf, if_).height(alpha);
                midValid = hcMid > K.shore && hcMid > 0.f;
                if (midValid) {
                    jMI = j;
                    iMI = i;
                    jMF = jf;
                    iMF = if_;
                    im = metric;
                    kMI = mem_level(split_level<SEM>(kMid, kMF), sW);
                    const uint32_t column = keptCell * (uint32_t)sW + (uint32_t)(kMI + sW - 1);
                    if (!lean) {
                        keep_column(column);
                    } else if (column != keptColumn) {
                        moved = true;
                        keptColumn = column;
                        C.stencil(column, kept);
                        current_at(kept, alpha, kMF, jMF, iMF, um, vm, wm);
                    }
                }
            }
            if (!lean) current_at(kept, alpha, kMF, jMF, iMF, um, vm, wm);
            else if (!moved) current_changed(kept, alpha, kMF, jMF, iMF, um, vm, wm);
            if (drift) {
                float du, dv;
                drift_velocity<full>(cfg, P, V, p.id, p.type, p.side, jMI, jMF, iMI, iMF, alpha,
                               elapsed, physicalTime, stepDt, du, dv);
                um += du;
                vm += dv;
            }
            const float2 d = __fmul2_rn(
                __fmul2_rn(make_float2(K.direction * um, K.direction * vm), make_float2(dt, dt)), im);
            dI = d.x;
            dJ = d.y;
            float detZ = K.direction * (K.sv + wm) * dt;
            if (midValid) {
                const float zdistMid =
                    hcMid * (kMI == kM ? depthHere : __ldg(F.X.depthIntervals + (kMI + sW - 2)));
                detZ = detZ * zdist * __frcp_rn(zdistMid);
            }
            dI += rx * inv.x;
            dJ += ry * inv.y;
            zleap = detZ + rz;
        } else {
            dI = (K.direction * uu * dt + rx) * inv.x;
            dJ = (K.direction * vv * dt + ry) * inv.y;
            zleap = K.direction * (K.sv + ww) * dt + rz;
        }
        if (fabsf(zleap) > zdist) zleap = signf_of(zdist, zleap);
        double jdet = p.j + (double)dJ;
        double idet = p.i + (double)dI;
        double kdet = p.k + (double)(zleap * rzdist);
        if (kdet > 0.) close_upper(cfg, kdet, p.health, lazy);
        if (kdet < kLower) close_lower(cfg, kLower, kdet, p.health, lazy);

        haveCarried = false;
        if (on_axis<SEM>(jdet, K.jEdge) && on_axis<SEM>(idet, K.iEdge)) {
            float jf, if_;
            const int jdetI = split_axis<SEM>(jdet, jf), idetI = split_axis<SEM>(idet, if_);
            keep_cell((uint32_t)(jdetI * xi + idetI));
            const SurfaceSums there = surface_from(surf, jf, if_);
            if (there.height(alpha) <= K.shore) {
                if (cfg.horizontalClosure == CLOSURE_CONSTRAINT) {
                    idet = p.i;
                    jdet = p.j;
                } else if (cfg.horizontalClosure == CLOSURE_KILL) {
                    p.health = -1;
                    lazy = false;
                } else if (cfg.horizontalClosure == CLOSURE_REFLECTION) {
                    idet = reflect_cell(p.i, iI, idet, idetI);
                    jdet = reflect_cell(p.j, jI, jdet, jdetI);
                }
            } else if (there.height(alpha) > K.shore) {
                // the next step starts here
                here = there;
                jI = jdetI;
                iI = idetI;
                jF = jf;
                iF = if_;
                haveCarried = true;
            }
            p.i = idet;
            p.j = jdet;
            p.k = kdet;
        } else {
            if (cfg.horizontalClosure == CLOSURE_CONSTRAINT) {
                p.k = kdet;
            } else if (cfg.horizontalClosure == CLOSURE_KILL) {
                p.health = -1;
                lazy = false;
            } else if (cfg.horizontalClosure == CLOSURE_REFLECTION) {
                p.i = reflect_domain(idet, K.iEdge);
                p.j = reflect_domain(jdet, K.jEdge);
                p.k = kdet;
            }
        }
        bool alive;
        if (lazy && youngLeft > 0) {  // still lazy: no closure ended the tracking this substep
            alive = true;
            youngLeft--;
        } else {
            alive = lazy ? (p.age < P.ageUnder || exp(-p.age / cfg.tau0) > 0) : p.health > 0;
            if (alive && !lazy) {
                // FP32 and an approximate division: the two-substep margin covers their error
                const float n = floorf(__fdividef((float)(K.ageSafe - p.age), K.dti)) - 2.f;
                youngLeft = n > 0.f ? (n < 1.0e9f ? (int)n : 1000000000) : 0;
            }
        }
        if (alive) {
            p.age = p.age + stepDt;
            lazy = true;
            if (jibe) {
                double probability = stepDt == cfg.dti
                                         ? P.jibeFullStep
                                         : jibe_step_probability(cfg.leewayJibeProbabilityHourly, stepDt);
                if (prefix_uniform(stepKey, JIBE_COMPONENT) < probability) p.side = -p.side;
            }
        }
        elapsed += stepDt;
    }
    if (lazy) p.health = exp(-p.age / cfg.tau0);
    return steps;
}

}  // namespace wb
