// The particle step: one particle over (a chunk of) one forcing interval, all substeps in
// registers.
//
// SEM selects the rules of the reference path being replaced: SEM_HOST follows
// Particle::move (Particle.cpp:71-824), SEM_DEVICE follows the reference kernel
// (kernel.cu:153-368); the few places where they differ are marked. The arithmetic is the
// reference's (FP64 with float-rounded corner terms; compiled with -fmad=false so that no product is
// fused except where it is written so).
#pragma once

#include "common.cuh"
#include "views.cuh"

namespace wb {

// Per-launch constants of one interval, computed by make_interval on the host (engine path)
// or by each thread from device memory (drop-in path, like kernel.cu:161-171).
struct IntervalParams {
    int t0, t1, direction;
    int rng;                  // WACOMM_B200_RNG_*
    int skip;                 // the interval lies before the restart checkpoint: no change
    double start, end, length;
    long long intervalKey;    // llround(min(start, end)) (Particle.cpp:523)
    double elapsed0;          // first elapsed of the interval after a restart clip
    double chunkEnd;          // substeps that start before this elapsed run in this launch
    int firstChunk, lastChunk;
    double kLower;            // -sW + 2
    double invKLower;         // 1 / kLower (FP32 step: depth factor of the random walk)
    // Survival test without a per-step exp: health = exp(-age/tau0) is below survprob for
    // age >= ageKillHi, above it for age <= ageKillLo, and evaluated exactly in between;
    // exp(-age/tau0) > 0 is certain for age < ageUnder.
    double ageKillLo, ageKillHi, ageUnder;
    double jibeFullStep;      // jibeStepProbability(hourly, dti)
};

// Interval bounds and restart clip (Particle.cpp:109-120 with NumericalHelpers.hpp:45-52 under
// the host rules; kernel.cu:161-171 under the device rules).
__host__ __device__ inline void make_interval(const wacomm_b200_config &cfg, const double *times,
                                              int nTimes, int timeIndex, int sW, int semantics,
                                              IntervalParams &P) {
    P.direction = cfg.trackingDirection;
    int next = timeIndex + P.direction;
    bool inside = next >= 0 && next < nTimes;
    P.start = times[timeIndex];
    P.end = inside ? times[next] : P.start + P.direction * cfg.deltat;
    P.length = fabs(P.end - P.start);
    P.t0 = timeIndex;
    P.t1 = inside ? next : timeIndex;
    P.intervalKey = llround(P.start < P.end ? P.start : P.end);
    P.skip = 0;
    P.elapsed0 = 0;
    double rc = cfg.restartCheckpoint;
    if (!isnan(rc)) {
        if (semantics == WACOMM_B200_SEMANTICS_HOST) {
            if (P.end > P.start) {
                if (P.end <= rc) P.skip = 1;
                else {
                    double a = P.end - P.start, b = rc - P.start;
                    b = b < 0.0 ? 0.0 : b;
                    P.elapsed0 = b < a ? b : a;
                }
            } else {
                if (P.end >= rc) P.skip = 1;
                else {
                    double a = P.start - P.end, b = P.start - rc;
                    b = b < 0.0 ? 0.0 : b;
                    P.elapsed0 = b < a ? b : a;
                }
            }
        } else {
            if ((P.direction > 0 && P.end <= rc) || (P.direction < 0 && P.end >= rc)) P.skip = 1;
            else P.elapsed0 = fmin(P.length, fmax(0.0, P.direction * (rc - P.start)));
        }
    }
    P.kLower = -sW + 2;
    P.invKLower = 1.0 / P.kLower;
    P.chunkEnd = INFINITY;
    P.firstChunk = 1;
    P.lastChunk = 1;
    P.rng = WACOMM_B200_RNG_REFERENCE;
    double tau0 = cfg.tau0;
    if (tau0 > 0 && isfinite(tau0)) {
        P.ageUnder = 700.0 * tau0;
        if (cfg.survprob > 0 && isfinite(cfg.survprob)) {
            double a = -tau0 * log(cfg.survprob);
            P.ageKillLo = a - 1e-9 * fabs(a) - 1e-300;
            P.ageKillHi = a + 1e-9 * fabs(a) + 1e-300;
        } else {
            // survprob <= 0 is never above exp(); NaN survprob never compares true
            P.ageKillLo = INFINITY;
            P.ageKillHi = INFINITY;
        }
    } else {
        P.ageUnder = -INFINITY;
        P.ageKillLo = -INFINITY;
        P.ageKillHi = INFINITY;
    }
    double hourly = cfg.leewayJibeProbabilityHourly, dt = cfg.dti;
    if (hourly <= 0 || dt <= 0) P.jibeFullStep = 0;
    else if (hourly >= 1) P.jibeFullStep = 1;
    else P.jibeFullStep = 1 - exp(log(1 - hourly) * dt / 3600);
}

struct ParticleState {
    uint64_t id;
    double k, j, i, health, age, time;
    int type, side;
};

// ------------------------------------------------------------------ interpolation pieces

// x rounded to float precision and range grid (the value of (float)x for every |x| below the float
// overflow bound): adding and subtracting 1.5 2^29 times the power of two of x (of 2^-126 for smaller
// x, the grid of the subnormal floats) rounds to nearest, ties to even, at the float's last place.
// Two FP64 adds and four integer instructions in place of a conversion to float and one back, both
// on the quarter-rate unit that bounds the reference arithmetic.
__device__ __forceinline__ double rounded_to_float(double x) {
    const int power = max(__double2hiint(x) & 0x7ff00000, (1023 - 126) << 20);
    const double shift = __hiloint2double(power + (29 << 20) + (1 << 19), 0);
    return __dadd_rn(__dadd_rn(x, shift), -shift);
}

// (float)interpolateTime(v0, v1, alpha) (NumericalHelpers.hpp:37-39, kernel.cu:71-74) as a double;
// v0 and v1 hold float values, as floats or as doubles.
template <class T>
__device__ __forceinline__ double at_ref(T v0, T v1, double a) {
    return rounded_to_float((1.0 - a) * (double)v0 + a * (double)v1);
}
__device__ __forceinline__ double at_ref(double2 v, double a) { return at_ref(v.x, v.y, a); }
__device__ __forceinline__ float at_f32(float v0, float v1, float a) { return fmaf(a, v1 - v0, v0); }

// a / b correctly rounded from r = 1 / b correctly rounded: the product with r, then two
// residual corrections (P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", 1990: a quotient within one unit in the last place, corrected once more
// with the correctly rounded reciprocal, is the rounded quotient). 5 FP64 instructions instead of a
// division's reciprocal iteration and range tests.
__device__ __forceinline__ double quotient(double a, double b, double r) {
    double q = a * r;
    if (!(fabs(q) <= DBL_MAX)) return a / b;
    q = __fma_rn(__fma_rn(-b, q, a), r, q);
    return __fma_rn(__fma_rn(-b, q, a), r, q);
}

// Adding 1.5 2^52 rounds |x| < 2^31 to an integer in the direction of the add and leaves it in the
// sum's low word: floor and ceil with their index in two FP64 adds, no conversion on the
// quarter-rate unit.
constexpr double INTEGER_SHIFT = 6755399441055744.0;

// floor(x) as to_index gives it, and x - floor(x) as x - index.
template <int SEM>
__device__ __forceinline__ int floor_index(double x, double &fraction) {
    if (fabs(x) < 2147483648.0) {
        const double shifted = __dadd_rd(x, INTEGER_SHIFT);
        fraction = x - (shifted - INTEGER_SHIFT);
        return __double2loint(shifted);
    }
    const int index = to_index<SEM>(floor(x));
    fraction = x - index;
    return index;
}

// ceil(k) as to_index gives it, and ceil(k) - k.
template <int SEM>
__device__ __forceinline__ int ceil_index(double k, double &fraction) {
    if (fabs(k) < 2147483648.0) {
        const double shifted = __dadd_ru(k, INTEGER_SHIFT);
        fraction = (shifted - INTEGER_SHIFT) - k;
        return __double2loint(shifted);
    }
    const double up = ceil(k);
    fraction = up - k;
    return to_index<SEM>(up);
}

// Float sum of four float-rounded corner terms c*(1-iF)*(1-jF) ... (Particle.cpp:271-277).
__device__ __forceinline__ float bilinear_ref(double c1, double c2, double c3, double c4, double jF,
                                              double iF) {
    float f1 = (float)(c1 * (1.0 - iF) * (1.0 - jF));
    float f2 = (float)(c2 * (1.0 - iF) * jF);
    float f3 = (float)(c3 * iF * jF);
    float f4 = (float)(c4 * iF * (1.0 - jF));
    return f1 + f2 + f3 + f4;
}

// Surface at a position: bilinear h (double) and zeta (float) (Particle.cpp:271-290;
// kernel.cu:197-198).
template <class View>
__device__ __forceinline__ void surface_at(const View &V, int jI, int iI, double jF, double iF,
                                           double alpha, double &hh, float &zz) {
    const auto s1 = V.surface(jI, iI), s2 = V.surface(jI + 1, iI);
    const auto s3 = V.surface(jI + 1, iI + 1), s4 = V.surface(jI, iI + 1);
    hh = s1.h * (1.0 - iF) * (1.0 - jF) + s2.h * (1.0 - iF) * jF + s3.h * iF * jF +
         s4.h * iF * (1.0 - jF);
    zz = bilinear_ref(at_ref(s1.z0, s1.z1, alpha), at_ref(s2.z0, s2.z1, alpha),
                      at_ref(s3.z0, s3.z1, alpha), at_ref(s4.z0, s4.z1, alpha), jF, iF);
}

// hcMid of the host rules: one double chain of four h and four zeta terms (Particle.cpp:601-604).
template <class View>
__device__ __forceinline__ double hc_mid_host(const View &V, int jI, int iI, double jF, double iF,
                                              double alpha) {
    const auto s1 = V.surface(jI, iI), s2 = V.surface(jI + 1, iI);
    const auto s3 = V.surface(jI + 1, iI + 1), s4 = V.surface(jI, iI + 1);
    return s1.h * (1.0 - iF) * (1.0 - jF) + s2.h * (1.0 - iF) * jF + s3.h * iF * jF +
           s4.h * iF * (1.0 - jF) + at_ref(s1.z0, s1.z1, alpha) * (1.0 - iF) * (1.0 - jF) +
           at_ref(s2.z0, s2.z1, alpha) * (1.0 - iF) * jF +
           at_ref(s3.z0, s3.z1, alpha) * iF * jF +
           at_ref(s4.z0, s4.z1, alpha) * iF * (1.0 - jF);
}

// Vertical field blend: host rules sum eight float terms (Particle.cpp:464-474, 490-500);
// device rules blend two float bilinears in double (kernel.cu:258-259, 265-266).
template <int SEM>
__device__ __forceinline__ double trilinear_ref(double u1, double u2, double u3, double u4,
                                                double l1, double l2, double l3, double l4, double kF,
                                                double jF, double iF) {
    if (SEM == SEM_HOST) {
        float w1 = (float)(u1 * (1.0 - iF) * (1.0 - jF) * (1.0 - kF));
        float w2 = (float)(u2 * (1.0 - iF) * jF * (1.0 - kF));
        float w3 = (float)(u3 * iF * jF * (1.0 - kF));
        float w4 = (float)(u4 * iF * (1.0 - jF) * (1.0 - kF));
        float w5 = (float)(l1 * (1.0 - iF) * (1.0 - jF) * kF);
        float w6 = (float)(l2 * (1.0 - iF) * jF * kF);
        float w7 = (float)(l3 * iF * jF * kF);
        float w8 = (float)(l4 * iF * (1.0 - jF) * kF);
        return (double)(w1 + w2 + w3 + w4 + w5 + w6 + w7 + w8);
    } else {
        return (double)bilinear_ref(u1, u2, u3, u4, jF, iF) * (1.0 - kF) +
               (double)bilinear_ref(l1, l2, l3, l4, jF, iF) * kF;
    }
}

__device__ __forceinline__ int mem_level(int kI, int sW) {
    return kI > 0 ? 0 : (kI < -sW + 2 ? -sW + 2 : kI);
}

// Keys a substep draws from: the ordered prefix (seed, particle, interval) folded once per
// interval, then the substep.
struct DrawKeys {
    uint64_t prefix;     // ordered-splitmix64 prefix through the interval coordinate
    uint64_t philoxKey;  // particle id mixed with the run seed
};

// ------------------------------------------------------------------ advective velocity

// Ocean current plus leeway and Stokes at a fractional position and forcing weight
// (Particle.cpp:352-475; kernel.cu:206-260). kI must already be a valid memory level.
template <int SEM, bool DRIFT, class View>
__device__ __forceinline__ void advective_velocity(const wacomm_b200_config &cfg,
                                                   const IntervalParams &P, const View &V,
                                                   const RefStencil &s, const ParticleState &p,
                                                   double kF, int jI, double jF, int iI, double iF,
                                                   double sa, double elapsed,
                                                   double physicalTime, double stepDt,
                                                   float &uu, float &vv, double &ww, int *err) {
    uu = bilinear_ref(at_ref(s.u[0], sa), at_ref(s.u[1], sa), at_ref(s.u[2], sa), at_ref(s.u[3], sa),
                      jF, iF);
    vv = bilinear_ref(at_ref(s.v[0], sa), at_ref(s.v[1], sa), at_ref(s.v[2], sa), at_ref(s.v[3], sa),
                      jF, iF);
    if (DRIFT && cfg.driftModel == 1 && p.type != 0) {
        if (SEM == SEM_HOST && (p.type < 0 || p.type > 22)) atomicOr(err, ERR_DRIFT_OBJECT);
        double windU = cfg.windU10, windV = cfg.windV10;
        EnvPair e1{}, e2{}, e3{}, e4{};
        bool env = V.hasWindU || V.hasWindV || V.hasStokes;
        if (env) {
            e1 = V.environment(jI, iI);
            e2 = V.environment(jI + 1, iI);
            e3 = V.environment(jI + 1, iI + 1);
            e4 = V.environment(jI, iI + 1);
        }
        // environmentAt: float corner sums per record, then the time blend
        // (Particle.cpp:384-395; kernel.cu:105-116)
        if (V.hasWindU) {
            float f = (float)((double)e1.wu0 * (1.0 - iF) * (1.0 - jF)) + (float)((double)e2.wu0 * (1.0 - iF) * jF) +
                      (float)((double)e3.wu0 * iF * jF) + (float)((double)e4.wu0 * iF * (1.0 - jF));
            float n = (float)((double)e1.wu1 * (1.0 - iF) * (1.0 - jF)) + (float)((double)e2.wu1 * (1.0 - iF) * jF) +
                      (float)((double)e3.wu1 * iF * jF) + (float)((double)e4.wu1 * iF * (1.0 - jF));
            windU = (1.0 - sa) * (double)f + sa * (double)n;
        }
        if (V.hasWindV) {
            float f = (float)((double)e1.wv0 * (1.0 - iF) * (1.0 - jF)) + (float)((double)e2.wv0 * (1.0 - iF) * jF) +
                      (float)((double)e3.wv0 * iF * jF) + (float)((double)e4.wv0 * iF * (1.0 - jF));
            float n = (float)((double)e1.wv1 * (1.0 - iF) * (1.0 - jF)) + (float)((double)e2.wv1 * (1.0 - iF) * jF) +
                      (float)((double)e3.wv1 * iF * jF) + (float)((double)e4.wv1 * iF * (1.0 - jF));
            windV = (1.0 - sa) * (double)f + sa * (double)n;
        }
        uint64_t substep = (uint64_t)floor(elapsed / cfg.dti);
        double longitude = V.lon(jI, iI) * (1.0 - iF) * (1.0 - jF) + V.lon(jI + 1, iI) * (1.0 - iF) * jF +
                           V.lon(jI + 1, iI + 1) * iF * jF + V.lon(jI, iI + 1) * iF * (1.0 - jF);
        double latitude = V.lat(jI, iI) * (1.0 - iF) * (1.0 - jF) + V.lat(jI + 1, iI) * (1.0 - iF) * jF +
                          V.lat(jI + 1, iI + 1) * iF * jF + V.lat(jI, iI + 1) * iF * (1.0 - jF);
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
            double when = physicalTime + .5 * P.direction * stepDt;
            double first = forcing_error_normal(cfg.randomSeed, p.id, P.intervalKey, substep,
                                                WIND_U_COMPONENT, longitude, latitude, when,
                                                spatial, temporal);
            double second = forcing_error_normal(cfg.randomSeed, p.id, P.intervalKey, substep,
                                                 WIND_V_COMPONENT, longitude, latitude, when,
                                                 spatial, temporal);
            windU += stdDev * first;
            windV += stdDev * correlated_normal(first, second, corr);
        }
        double downwindNormal = 0, crosswindNormal = 0;
        if (cfg.leewayCoefficientEnsemble) {
            uint64_t ens = key_prefix(cfg.randomSeed, p.id, ENSEMBLE_INTERVAL, 0);
            downwindNormal = prefix_normal(ens, 0);
            crosswindNormal = prefix_normal(ens, 1);
            crosswindNormal = correlated_normal(downwindNormal, crosswindNormal,
                                                cfg.leewayResidualCorrelation);
        }
        Leeway lw = compute_leeway(p.type, windU, windV, p.side, downwindNormal, crosswindNormal);
        uu += (float)lw.u;
        vv += (float)lw.v;
        if (V.hasStokes) {
            // waveAt: double corner sums (Particle.cpp:446-453; kernel.cu:118-129)
            double fu = (double)e1.su0 * (1.0 - iF) * (1.0 - jF) + (double)e2.su0 * (1.0 - iF) * jF +
                        (double)e3.su0 * iF * jF + (double)e4.su0 * iF * (1.0 - jF);
            double nu = (double)e1.su1 * (1.0 - iF) * (1.0 - jF) + (double)e2.su1 * (1.0 - iF) * jF +
                        (double)e3.su1 * iF * jF + (double)e4.su1 * iF * (1.0 - jF);
            double fv = (double)e1.sv0 * (1.0 - iF) * (1.0 - jF) + (double)e2.sv0 * (1.0 - iF) * jF +
                        (double)e3.sv0 * iF * jF + (double)e4.sv0 * iF * (1.0 - jF);
            double nv = (double)e1.sv1 * (1.0 - iF) * (1.0 - jF) + (double)e2.sv1 * (1.0 - iF) * jF +
                        (double)e3.sv1 * iF * jF + (double)e4.sv1 * iF * (1.0 - jF);
            uu += (float)((1.0 - sa) * fu + sa * nu);
            vv += (float)((1.0 - sa) * fv + sa * nv);
        }
    }
    ww = trilinear_ref<SEM>(at_ref(s.wUp[0], sa), at_ref(s.wUp[1], sa), at_ref(s.wUp[2], sa),
                            at_ref(s.wUp[3], sa), at_ref(s.wLo[0], sa), at_ref(s.wLo[1], sa),
                            at_ref(s.wLo[2], sa), at_ref(s.wLo[3], sa), kF, jF, iF);
}

// Vertical diffusivity at the particle (Particle.cpp:490-500; kernel.cu:265-266).
template <int SEM, class View>
__device__ __forceinline__ double akt_at(const View &V, int kI, double kF, int jI, double jF,
                                         int iI, double iF, double alpha) {
    return trilinear_ref<SEM>(
        at_ref(V.akt(kI, jI, iI), alpha), at_ref(V.akt(kI, jI + 1, iI), alpha),
        at_ref(V.akt(kI, jI + 1, iI + 1), alpha), at_ref(V.akt(kI, jI, iI + 1), alpha),
        at_ref(V.akt(kI - 1, jI, iI), alpha), at_ref(V.akt(kI - 1, jI + 1, iI), alpha),
        at_ref(V.akt(kI - 1, jI + 1, iI + 1), alpha), at_ref(V.akt(kI - 1, jI, iI + 1), alpha), kF,
        jF, iF);
}

__device__ __forceinline__ void close_upper(const wacomm_b200_config &cfg, double &k, double &health,
                                            bool &lazy) {
    if (cfg.upperClosure == CLOSURE_CONSTRAINT) k = 0;
    else if (cfg.upperClosure == CLOSURE_KILL) { health = -1; lazy = false; }
    else if (cfg.upperClosure == CLOSURE_REFLECTION) k = -k;
}

__device__ __forceinline__ void close_lower(const wacomm_b200_config &cfg, double kLower, double &k,
                                            double &health, bool &lazy) {
    if (cfg.lowerClosure == CLOSURE_CONSTRAINT) k = kLower;
    else if (cfg.lowerClosure == CLOSURE_KILL) { health = -1; lazy = false; }
    else if (cfg.lowerClosure == CLOSURE_REFLECTION) k = 2.0 * kLower - k;
}

// ------------------------------------------------------------------ the interval loop

// Integrates particle p from `elapsed` while substeps start before min(length, chunkEnd).
// On return `elapsed` is where the next chunk resumes (>= length when the particle is done).
// Returns the number of substeps taken (particle-steps of this launch). DRIFT false leaves the
// drifting objects' branch out, for runs without a drift model; KEEP holds the velocity stencil (64
// registers) from substep to substep, for launches with registers to spare.
template <int SEM, bool DRIFT, bool KEEP, class View>
__device__ int move_particle(const wacomm_b200_config &cfg, const IntervalParams &P,
                             const View &V, ParticleState &p, double &elapsed, int *err) {
    const int eta = V.g.eta, xi = V.g.xi, sW = V.g.sW;
    const double kLower = P.kLower, length = P.length;
    const int direction = P.direction;
    const double dir = (double)direction;
    const bool midpoint = cfg.integrator == INTEGRATOR_MIDPOINT;
    const bool diffuse = cfg.random && (dir > 0 || cfg.backwardDiffusion);
    bool lazy = false;  // true while health == exp(-age/tau0) is owed
    int steps = 0;

    if (P.firstChunk) {
        // Closures before the loop (Particle.cpp:134-176; kernel.cu:173-182)
        if (p.k > 0) close_upper(cfg, p.k, p.health, lazy);
        if (p.k < kLower) close_lower(cfg, kLower, p.k, p.health, lazy);
    }
    DrawKeys keys;
    keys.prefix = fold(fold(mix64(cfg.randomSeed), p.id), (uint64_t)P.intervalKey);
    keys.philoxKey = p.id ^ mix64(cfg.randomSeed);
    const double stop = P.chunkEnd < length ? P.chunkEnd : length;
    const double rLength = 1.0 / length;
    // The velocity stencil of the particle's cell and level; KEEP: read again only when either
    // changes.
    RefStencil kept;
    long long keptColumn = -1;
    auto keep_column = [&](int kI, int jI, int iI) {
        const long long column = ((long long)(kI + sW - 1) * eta + jI) * xi + iI;
        if (!KEEP || column != keptColumn) {
            V.stencil(kI, jI, iI, kept);
            keptColumn = column;
        }
    };

    while (elapsed < stop) {
        double stepDt = SEM == SEM_HOST ? smin(cfg.dti, length - elapsed)
                                        : fmin(cfg.dti, length - elapsed);
        double physicalTime = P.start + direction * elapsed;
        if (direction > 0 && p.time > physicalTime) {
            // Not yet released: jump to the release time (Particle.cpp:211-215)
            elapsed = SEM == SEM_HOST ? smin(length, p.time - P.start)
                                      : fmin(length, p.time - P.start);
            continue;
        }
        bool dead;
        if (lazy)
            dead = p.age >= P.ageKillHi ||
                   (p.age > P.ageKillLo && exp(-p.age / cfg.tau0) < cfg.survprob);
        else
            dead = p.health < cfg.survprob;
        if (dead) {
            p.health = -1;
            lazy = false;
            elapsed = length;
            break;
        }
        double kF, jF, iF;
        const int kI = ceil_index<SEM>(p.k, kF);
        const int jI = floor_index<SEM>(p.j, jF), iI = floor_index<SEM>(p.i, iF);
        if (!valid_cell(jI, iI, eta, xi)) {
            p.health = -1;
            lazy = false;
            elapsed = length;
            break;
        }
        if (SEM == SEM_DEVICE && (kI > 0 || kI <= -sW + 1)) {
            p.health = -1;  // device-only level test (kernel.cu:195)
            lazy = false;
            elapsed = length;
            break;
        }
        steps++;
        double alpha = length == 0 ? 0 : quotient(elapsed + 0.5 * stepDt, length, rLength);
        double alphaStart = length == 0 ? 0 : quotient(elapsed, length, rLength);
        double hh;
        float zz;
        surface_at(V, jI, iI, jF, iF, alpha, hh, zz);
        double hc = hh + zz;
        if (hc <= cfg.shoreLimit && cfg.horizontalClosure == CLOSURE_KILL) {
            p.health = -1;
            lazy = false;
            if (SEM == SEM_DEVICE) {  // the host rules finish the step (Particle.cpp:311-319)
                elapsed = length;
                break;
            }
        }
        const int kM = mem_level(kI, sW);
        float uu, vv;
        double ww;
        keep_column(kM, jI, iI);
        advective_velocity<SEM, DRIFT>(cfg, P, V, kept, p, kF, jI, jF, iI, iF,
                                       midpoint ? alphaStart : alpha, elapsed, physicalTime,
                                       stepDt, uu, vv, ww, err);
        double dxleap = dir * uu * stepDt, dyleap = dir * vv * stepDt;
        double dzleap = dir * (cfg.sv + ww) * stepDt;
        double rx = 0, ry = 0, rz = 0;
        uint64_t substep = 0;
        uint64_t stepKey = 0;
        bool keyed = diffuse || (cfg.leewayJibeProbabilityHourly > 0 && p.type != 0);
        if (keyed) {
            substep = (uint64_t)floor(elapsed / cfg.dti);
            stepKey = fold(keys.prefix, substep);
        }
        if (diffuse) {
            // Stochastic leap (Particle.cpp:518-533; kernel.cu:269-276)
            double aa = akt_at<SEM>(V, kM, kF, jI, jF, iI, iF, alpha);
            double sigmaDepth = cfg.sigma * (1 - quotient(p.k, kLower, P.invKLower));
            double scale = stepDt == cfg.dti ? 1.0 : sqrt(stepDt / cfg.dti);
            double n0, n1, n2;
            if (P.rng == WACOMM_B200_RNG_PHILOX) {
                float f0, f1, f2;
                philox_normals3(keys.philoxKey, P.intervalKey,
                                (uint64_t)__double_as_longlong(elapsed), f0, f1, f2);
                n0 = f0;
                n1 = f1;
                n2 = f2;
            } else {
                n0 = prefix_normal(stepKey, 0);
                n1 = prefix_normal(stepKey, 1);
                n2 = prefix_normal(stepKey, 2);
            }
            rx = sigmaDepth * n0 * scale;
            ry = sigmaDepth * n1 * scale;
            rz = sigmaDepth * n2 * aa * cfg.crid * scale;
        }
        double xleap = dxleap + rx, yleap = dyleap + ry, zleap = dzleap + rz;

        const CellMetric md = V.cell_metric(jI, iI);
        const double xdist = md.x, ydist = md.y;
        double zdist = hc * V.depth_interval(kM);

        if (midpoint) {
            // Explicit midpoint (Particle.cpp:585-641; kernel.cu:281-317)
            double kHalf = dir * (cfg.sv + ww) * 0.5 * stepDt;
            if (fabs(kHalf) > zdist) kHalf = sign_of(zdist, kHalf);
            double iMid = p.i + quotient(dir * uu * 0.5 * stepDt, xdist, md.rx);
            double jMid = p.j + quotient(dir * vv * 0.5 * stepDt, ydist, md.ry);
            double kMid = SEM == SEM_HOST ? smin(0.0, smax(kLower, p.k + kHalf / zdist))
                                          : fmin(0.0, fmax(kLower, p.k + kHalf / zdist));
            // the midpoint, or the start where the midpoint has no water: one evaluation for both
            double iMF, jMF, kMF = kF;
            int iMI = floor_index<SEM>(iMid, iMF), jMI = floor_index<SEM>(jMid, jMF), kMI = kM;
            bool midValid = valid_cell(jMI, iMI, eta, xi);
            double hcMid = 0;
            if (midValid) {
                if (SEM == SEM_HOST) {
                    hcMid = hc_mid_host(V, jMI, iMI, jMF, iMF, alpha);
                } else {
                    double hm;
                    float zm;
                    surface_at(V, jMI, iMI, jMF, iMF, alpha, hm, zm);
                    hcMid = hm + zm;
                }
                midValid = hcMid > cfg.shoreLimit && hcMid > 0;
            }
            if (midValid) {
                kMI = mem_level(ceil_index<SEM>(kMid, kMF), sW);
            } else {
                iMI = iI;
                jMI = jI;
                iMF = iF;
                jMF = jF;
            }
            float um, vm;
            double wm;
            keep_column(kMI, jMI, iMI);
            advective_velocity<SEM, DRIFT>(cfg, P, V, kept, p, kMF, jMI, jMF, iMI, iMF, alpha,
                                           elapsed, physicalTime, stepDt, um, vm, wm, err);
            double detX = dir * um * stepDt, detY = dir * vm * stepDt;
            double detZ = dir * (cfg.sv + wm) * stepDt;
            if (midValid) {
                const CellMetric mm = V.cell_metric(jMI, iMI);
                double zdistMid = hcMid * V.depth_interval(kMI);
                detX = quotient(detX * xdist, mm.x, mm.rx);
                detY = quotient(detY * ydist, mm.y, mm.ry);
                detZ = detZ * zdist / zdistMid;
            }
            if (SEM == SEM_HOST) {
                xleap = detX + rx;
                yleap = detY + ry;
                zleap = detZ + rz;
            } else {
                xleap += detX - dir * uu * stepDt;
                yleap += detY - dir * vv * stepDt;
                zleap += detZ - dir * (cfg.sv + ww) * stepDt;
            }
        }

        // Vertical cap, candidate position and vertical closures (Particle.cpp:644-704)
        if (fabs(zleap) > zdist) zleap = sign_of(zdist, zleap);
        double jdet = p.j + quotient(yleap, ydist, md.ry);
        double idet = p.i + quotient(xleap, xdist, md.rx);
        double kdet = p.k + zleap / zdist;
        if (kdet > 0.) close_upper(cfg, kdet, p.health, lazy);
        if (kdet < kLower) close_lower(cfg, kLower, kdet, p.health, lazy);

        // Horizontal landing and closures (Particle.cpp:706-791; kernel.cu:331-353)
        double jdetF, idetF;
        const int jdetI = floor_index<SEM>(jdet, jdetF), idetI = floor_index<SEM>(idet, idetF);
        if (valid_cell(jdetI, idetI, eta, xi)) {
            double hd;
            float zd;
            surface_at(V, jdetI, idetI, jdetF, idetF, alpha, hd, zd);
            double hcdet = hd + zd;
            if (hcdet <= cfg.shoreLimit) {
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
                p.i = reflect_domain(idet, xi - 1);
                p.j = reflect_domain(jdet, eta - 1);
                p.k = kdet;
            }
        }

        // Age, decay and jibing (Particle.cpp:797-814; kernel.cu:354-364)
        bool alive = lazy ? (p.age < P.ageUnder || exp(-p.age / cfg.tau0) > 0) : p.health > 0;
        if (alive) {
            p.age = p.age + stepDt;
            lazy = true;
            if (cfg.leewayJibeProbabilityHourly > 0 && p.type != 0) {
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
