// Drop-in replacement of the reference GPU launcher (kernel.cu:370-382): same arguments, same
// in-place update of the caller's particle_data records, device rules and reference arithmetic.
// The work is ordered by horizontal cell (and level) first -- key per record, histogram, exclusive
// scan, scatter into a work order -- so that the threads of a warp gather the same forcing cells, and
// the forcing pair and the cell metric are packed once per call (views.cuh) instead of being gathered
// from the window and recomputed by haversines in every substep; each record still moves
// independently, so neither changes a result. The scratch is stream-ordered
// (cudaMallocAsync/cudaFreeAsync on the caller's stream, served from the device's memory pool without
// a device-wide synchronization); what cannot be had is done without: the records are moved in
// caller order, or read the window directly. Compiled with -fmad=false.
#include "engine.h"
#include "move_kernels.cuh"
#include "wacomm_b200_kernel.h"

namespace wb {

// Sort key of each record (its cell, and its level where `levels` > 1; the last bin for records
// outside the interpolation cells) and the warp-aggregated histogram of the keys.
__global__ void dropin_key_kernel(const wacomm_b200_particle *particles, int n, int eta, int xi,
                                  int levels, uint32_t *keys, uint32_t *hist) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        const double fj = floor(particles[p].j), fi = floor(particles[p].i);
        uint32_t key = (uint32_t)((size_t)eta * xi * levels);
        if (fj >= 0.0 && fi >= 0.0 && fj < (double)(eta - 1) && fi < (double)(xi - 1)) {
            const double down = fmin(fmax(-ceil(particles[p].k), 0.0), (double)(levels - 1));
            key = (uint32_t)((int)fj * xi + (int)fi) * (uint32_t)levels + (uint32_t)down;
        }
        keys[p] = key;
        unsigned peers = __match_any_sync(__activemask(), key);
        if ((threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(hist + key, (uint32_t)__popc(peers));
    }
}

// The call's forcing pair and cell metric in the engine's layout. Like the move, each thread reads
// the tracking direction from the device copy of the config; one thread per (level, node).
__global__ void __launch_bounds__(256) dropin_pack_kernel(
    const wacomm_b200_config *__restrict__ config, int timeIndex, int oceanTime, RawView V,
    NodeRecord *nodes, SurfRecord *surf, CellMetric *metric, EnvPair *env) {
    __shared__ NodeStage stage;
    const int next = timeIndex + config->trackingDirection;
    V.t0 = timeIndex;
    V.t1 = next >= 0 && next < oceanTime ? next : timeIndex;
    const int eta = V.g.eta, xi = V.g.xi;
    const size_t plane = (size_t)eta * xi, total = plane * V.g.sW;
    for (size_t base = blockIdx.x * (size_t)256; base < total; base += gridDim.x * (size_t)256) {
        const size_t n = base + threadIdx.x;
        const int L = (int)(n / plane);
        const size_t c = n - (size_t)L * plane;
        const int j = (int)(c / xi), i = (int)(c - (size_t)j * xi);
        NodeRecord r;
        r.w = r.akt = r.u = r.v = make_double2(0.0, 0.0);
        if (n < total) {
            r.w = V.pair(V.w, L, V.g.sW, j, i);
            r.akt = V.pair(V.aktField, L, V.g.sW, j, i);
            if (L > 0) {
                r.u = V.pair(V.u, L - 1, V.g.sRho, j, i);
                r.v = V.pair(V.v, L - 1, V.g.sRho, j, i);
            }
        }
        store_nodes(stage, r, base, total, nodes);
        if (L == 0) {
            const SurfPair<float> s = V.surface(j, i);
            surf[c] = SurfRecord{s.h, s.z0, s.z1, 0.0};
            if (j + 1 < eta && i + 1 < xi) metric[c] = V.cell_metric(j, i);
            if (env) env[c] = V.environment(j, i);
        }
    }
}

// Work order: record slots grouped by key, from the exclusive offsets of the histogram.
__global__ void dropin_scatter_kernel(const uint32_t *keys, int n, uint32_t *cursor,
                                      uint32_t *order) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        uint32_t key = keys[p];
        unsigned peers = __match_any_sync(__activemask(), key);
        int lane = threadIdx.x & 31, leader = __ffs(peers) - 1;
        uint32_t base = 0;
        if (lane == leader) base = atomicAdd(cursor + key, (uint32_t)__popc(peers));
        base = __shfl_sync(peers, base, leader);
        order[base + __popc(peers & ((1u << lane) - 1u))] = (uint32_t)p;
    }
}

__device__ __forceinline__ RawView at_interval(RawView V, const IntervalParams &P) {
    V.t0 = P.t0;
    V.t1 = P.t1;
    return V;
}
__device__ __forceinline__ const PackedView &at_interval(const PackedView &V, const IntervalParams &) {
    return V;
}

// One work item per record, taken in the work order (null: caller order). Like the reference
// kernel, each thread derives the interval from the device copies of config and times
// (kernel.cu:158-171); the particle is read from and written back to the caller's AoS array.
// 524,287 records on 128 x 128 x 10, 120 substeps: 13.7 ms with the window read and two haversines
// per substep (244 registers), 3.9 ms with the packed pair (3.4 times faster per call). Bound by L1 (87 %
// of its throughput: two stencil reads per substep, and spills, because the config is on the device and
// the drift form is in the same kernel); up to a record per cell and level the packed form keeps its
// stencil (keeps_stencil: 100,000 records on 200 x 200 x 20 1.95 -> 1.22 ms). Whole calls at 244 registers
// without spills / now: with leeway drift 500,000 records 20.2 / 8.9 ms packed; read from a window of 12.3 M
// nodes 50,000 records 3.1 / 1.9 ms, 500,000 15.3 / 10.9 ms, with leeway drift 24.1 / 19.2 ms.
template <bool KEEP, class View>
__global__ void __launch_bounds__(128, KEEP ? 1 : 4) dropin_move_kernel(
    const wacomm_b200_config *__restrict__ config, wacomm_b200_particle *particles,
    const uint32_t *__restrict__ order, int timeIndex, int oceanTime,
    const double *__restrict__ times, const View V, const MoveLaunch L) {
    const unsigned t = launch_item(L, blockIdx.x * (blockDim.x >> 5) * L.lanes, L.count);
    if (t >= (unsigned)L.count) return;
    const wacomm_b200_config &cfg = *config;
    IntervalParams P;
    make_interval(cfg, times, oceanTime, timeIndex, V.g.sW, SEM_DEVICE, P);
    if (P.skip) return;
    const View &view = at_interval(V, P);
    uint32_t idx = order ? order[t] : (uint32_t)t;
    // the whole record as words, so that its padding bytes go back as they came
    union {
        unsigned long long words[8];
        wacomm_b200_particle rec;
    } held;
    static_assert(sizeof(wacomm_b200_particle) == 64, "record layout");
    unsigned long long *words = reinterpret_cast<unsigned long long *>(particles + idx);
    for (int w = 0; w < 8; w++) held.words[w] = words[w];
    wacomm_b200_particle &rec = held.rec;
    ParticleState p;
    p.id = rec.id;
    p.k = rec.k;
    p.j = rec.j;
    p.i = rec.i;
    p.health = rec.health;
    p.age = rec.age;
    p.time = rec.time;
    p.type = rec.driftObjectType;
    p.side = rec.driftSide;
    double elapsed = P.elapsed0;
    if (cfg.driftModel == 1)
        move_particle<SEM_DEVICE, true, KEEP>(cfg, P, view, p, elapsed, nullptr);
    else
        move_particle<SEM_DEVICE, false, KEEP>(cfg, P, view, p, elapsed, nullptr);
    rec.k = p.k;
    rec.j = p.j;
    rec.i = p.i;
    rec.health = p.health;
    rec.age = p.age;
    rec.driftSide = (int8_t)p.side;
    for (int w = 1; w < 8; w++)
        if (w != 6) words[w] = held.words[w];  // all but the id and the release time
}

template <class View>
cudaError_t launch_dropin(const wacomm_b200_config *config, wacomm_b200_particle *particles,
                          const uint32_t *order, int timeIndex, int oceanTime, const double *times,
                          const View &V, bool keep, int count, cudaStream_t stream) {
    MoveLaunch L{};
    L.count = count;
    int threads;
    spread_launch(count, 128, L.lanes, threads);
    const int items = threads / 32 * L.lanes, blocks = launch_blocks(count, items);
    if (keep)
        dropin_move_kernel<true><<<blocks, threads, 0, stream>>>(config, particles, order, timeIndex,
                                                                 oceanTime, times, V, L);
    else
        dropin_move_kernel<false><<<blocks, threads, 0, stream>>>(config, particles, order, timeIndex,
                                                                  oceanTime, times, V, L);
    return cudaGetLastError();
}

// The call's packed pair in `scratch` (null: no scratch, read the window), stream-ordered. The window is
// read where the scratch would be too large for the records (packs_pair) or a node record does not hold
// what the move reads: with other rho levels than one per layer, or without a field (the diffusivity of
// a run without random walk).
cudaError_t pack_window(const wacomm_b200_config *config, int timeIndex, int oceanTime,
                        const RawView &V, int count, PackedView &out, void **scratch,
                        cudaStream_t stream) {
    const size_t plane = (size_t)V.g.eta * V.g.xi, nodes = plane * V.g.sW;
    const bool env = V.hasWindU || V.hasWindV || V.hasStokes;
    *scratch = nullptr;
    if (V.g.eta < 2 || V.g.xi < 2 || V.g.sW != V.g.sRho + 1 || !V.zeta || !V.u || !V.v || !V.w ||
        !V.aktField || !V.hField || !V.lonRad || !V.latRad)
        return cudaSuccess;
    const size_t bytes = nodes * sizeof(NodeRecord) +
                         plane * (sizeof(SurfRecord) + sizeof(CellMetric) + (env ? sizeof(EnvPair) : 0));
    if (!packs_pair(bytes, (size_t)count)) return cudaSuccess;
    if (cudaMallocAsync(scratch, bytes, stream) != cudaSuccess) {
        *scratch = nullptr;
        (void)cudaGetLastError();  // no pool memory: read the window
        return cudaSuccess;
    }
    NodeRecord *n = static_cast<NodeRecord *>(*scratch);
    SurfRecord *s = reinterpret_cast<SurfRecord *>(n + nodes);
    CellMetric *m = reinterpret_cast<CellMetric *>(s + plane);
    EnvPair *e = env ? reinterpret_cast<EnvPair *>(m + plane) : nullptr;
    size_t blocks = (nodes + 255) / 256;
    if (blocks > 148 * 16) blocks = 148 * 16;
    dropin_pack_kernel<<<(unsigned)blocks, 256, 0, stream>>>(config, timeIndex, oceanTime, V, n, s, m, e);
    out.g = V.g;
    out.nodes = n;
    out.surf = s;
    out.env = e;
    out.hasWindU = V.hasWindU;
    out.hasWindV = V.hasWindV;
    out.hasStokes = V.hasStokes;
    out.lonRad = V.lonRad;
    out.latRad = V.latRad;
    out.depthIntervals = V.depthIntervals;
    out.metric = m;
    return cudaGetLastError();
}

int dropin_move(const wacomm_b200_config *config, wacomm_b200_particle *particles, int timeIndex,
                int oceanTime, int sW, int sRho, int eta, int xi, const double *times,
                const double *lonRad, const double *latRad, const double *depthIntervals,
                const double *h, const float *zeta, const float *u, const float *v,
                const float *w, const float *akt, const float *windU, const float *windV,
                const float *stokesU, const float *stokesV, int count, cudaStream_t stream) {
    if (count <= 0) return (int)cudaGetLastError();
    RawView V;
    V.g = GridShape{eta, xi, sW, sRho};
    V.t0 = V.t1 = 0;
    V.zeta = zeta;
    V.u = u;
    V.v = v;
    V.w = w;
    V.aktField = akt;
    V.windU = windU;
    V.windV = windV;
    V.stokesU = stokesU;
    V.stokesV = stokesV;
    V.hField = h;
    V.lonRad = lonRad;
    V.latRad = latRad;
    V.depthIntervals = depthIntervals;
    V.hasWindU = windU != nullptr;
    V.hasWindV = windV != nullptr;
    V.hasStokes = stokesU != nullptr && stokesV != nullptr;
    uint32_t *order = nullptr, *scratch = nullptr;
    if (eta >= 2 && xi >= 2) {
        // keys[count] | order[count] | histogram[bins] | offsets[bins + 1] | scan partials
        const int levels = sort_bins(eta, xi, sRho, (size_t)count, false, INFINITY).levels;
        size_t bins = (size_t)eta * xi * levels + 1;
        size_t words = 2 * (size_t)count + 2 * bins + 1 + scan_temp_words(bins);
        if (cudaMallocAsync((void **)&scratch, words * sizeof(uint32_t), stream) == cudaSuccess) {
            uint32_t *keys = scratch, *hist = scratch + 2 * (size_t)count;
            uint32_t *offsets = hist + bins, *partials = offsets + bins + 1;
            int blocks = (count + 255) / 256;
            if (blocks > 148 * 16) blocks = 148 * 16;
            cudaError_t e = cudaMemsetAsync(hist, 0, bins * sizeof(uint32_t), stream);
            if (e == cudaSuccess) {
                dropin_key_kernel<<<blocks, 256, 0, stream>>>(particles, count, eta, xi, levels,
                                                              keys, hist);
                e = exclusive_scan(hist, offsets, bins, offsets + bins, partials, stream);
            }
            if (e == cudaSuccess) {
                order = keys + count;
                dropin_scatter_kernel<<<blocks, 256, 0, stream>>>(keys, count, offsets, order);
            } else {
                cudaFreeAsync(scratch, stream);
                return (int)e;
            }
        } else {
            scratch = nullptr;
            (void)cudaGetLastError();  // no pool memory: caller order
        }
    }
    PackedView packed;
    void *pair = nullptr;
    cudaError_t e = pack_window(config, timeIndex, oceanTime, V, count, packed, &pair, stream);
    // Read from the window, 16 warps per SM hide the haversines of thinly spread records, too: 500,000
    // on 12.3 M nodes 10.9 ms, 13.2 ms with the stencil kept at 8 (100,000: 3.7 and 3.2, 50,000: 1.9 and 2.1).
    if (e == cudaSuccess)
        e = pair ? launch_dropin(config, particles, order, timeIndex, oceanTime, times, packed,
                                 keeps_stencil(count, eta, xi, sRho), count, stream)
                 : launch_dropin(config, particles, order, timeIndex, oceanTime, times, V,
                                 count <= KEEP_RECORDS, count, stream);
    for (void *held : {pair, (void *)scratch})
        if (held) {
            cudaError_t f = cudaFreeAsync(held, stream);
            if (e == cudaSuccess) e = f;
        }
    return (int)e;
}

}  // namespace wb

// The reference signature (cuda/kernel.h:7), C++ linkage, so that Wacomm.cpp and the reference
// parity test link against this library unchanged.
cudaError_t cudaMoveParticle(config_data *config, particle_data *particles, int timeIndex,
                             int oceanTime, int sW, int sRho, int eta, int xi, double *times,
                             double *mask, double *lonRad, double *latRad, double *depthIntervals,
                             double *h, float *zeta, float *u, float *v, float *w, float *akt,
                             float *windU10, float *windV10, float *stokesU, float *stokesV,
                             int particleCount, int numThread, int numGPU, cudaStream_t stream) {
    (void)mask;
    (void)numThread;
    (void)numGPU;
    return (cudaError_t)wb::dropin_move(
        reinterpret_cast<const wacomm_b200_config *>(config),
        reinterpret_cast<wacomm_b200_particle *>(particles), timeIndex, oceanTime, sW, sRho, eta,
        xi, times, lonRad, latRad, depthIntervals, h, zeta, u, v, w, akt, windU10, windV10,
        stokesU, stokesV, particleCount, stream);
}

extern "C" int wacomm_b200_cuda_move_particle(
    const wacomm_b200_config *config_device, wacomm_b200_particle *particles_device,
    int time_index, int ocean_time, int s_w, int s_rho, int eta, int xi, const double *times,
    const double *mask, const double *lon_rad, const double *lat_rad,
    const double *depth_intervals, const double *h, const float *zeta, const float *u,
    const float *v, const float *w, const float *akt, const float *wind_u10,
    const float *wind_v10, const float *stokes_u, const float *stokes_v, int particle_count,
    int num_thread, int num_gpu, void *stream) {
    (void)mask;
    (void)num_thread;
    (void)num_gpu;
    return wb::dropin_move(config_device, particles_device, time_index, ocean_time, s_w, s_rho,
                           eta, xi, times, lon_rad, lat_rad, depth_intervals, h, zeta, u, v, w,
                           akt, wind_u10, wind_v10, stokes_u, stokes_v, particle_count,
                           static_cast<cudaStream_t>(stream));
}
