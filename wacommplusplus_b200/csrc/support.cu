// Kernels around the move: forcing-pair packing, cell metric, scan, counting sort by cell,
// record layout conversion, stable dead-particle compaction and concentration grids.
#include "engine.h"
#include "move_kernels.cuh"

namespace wb {

static inline int grid_for(size_t n, int block, int maxBlocks = 148 * 16) {
    size_t blocks = (n + block - 1) / block;
    if (blocks > (size_t)maxBlocks) blocks = maxBlocks;
    return blocks < 1 ? 1 : (int)blocks;
}

size_t node_record_bytes() { return sizeof(NodeRecord); }
size_t surf_record_bytes() { return sizeof(SurfRecord); }

// ------------------------------------------------------------------ forcing pair packing

// Interleaves records t0 and t1 into the node records of the reference arithmetic.
__global__ void __launch_bounds__(256) pack_nodes_kernel(int eta, int xi, int sW, FrameDevice f0,
                                                         FrameDevice f1, NodeRecord *nodes) {
    __shared__ NodeStage stage;
    const size_t plane = (size_t)eta * xi, total = plane * sW;
    for (size_t base = blockIdx.x * (size_t)256; base < total; base += gridDim.x * (size_t)256) {
        const size_t n = base + threadIdx.x;
        NodeRecord r;
        r.w = r.akt = r.u = r.v = make_double2(0.0, 0.0);
        if (n < total) {
            r.w = make_double2(f0.w[n], f1.w[n]);
            r.akt = make_double2(f0.akt[n], f1.akt[n]);
            if (n >= plane) {  // W level 0 has no rho level below it
                r.u = make_double2(f0.u[n - plane], f1.u[n - plane]);
                r.v = make_double2(f0.v[n - plane], f1.v[n - plane]);
            }
        }
        store_nodes(stage, r, base, total, nodes);
    }
}

__global__ void pack_surface_kernel(int eta, int xi, FrameDevice f0, FrameDevice f1,
                                    const double *h, SurfRecord *surf) {
    size_t plane = (size_t)eta * xi;
    for (size_t n = blockIdx.x * (size_t)blockDim.x + threadIdx.x; n < plane;
         n += (size_t)gridDim.x * blockDim.x)
        surf[n] = SurfRecord{h[n], f0.zeta[n], f1.zeta[n], 0.0};
}

__global__ void pack_environment_kernel(int eta, int xi, FrameDevice f0, FrameDevice f1,
                                        EnvPair *env) {
    size_t plane = (size_t)eta * xi;
    for (size_t n = blockIdx.x * (size_t)blockDim.x + threadIdx.x; n < plane;
         n += (size_t)gridDim.x * blockDim.x) {
        EnvPair e;
        e.wu0 = f0.windU ? f0.windU[n] : 0.f;
        e.wv0 = f0.windV ? f0.windV[n] : 0.f;
        e.su0 = f0.stokesU ? f0.stokesU[n] : 0.f;
        e.sv0 = f0.stokesV ? f0.stokesV[n] : 0.f;
        e.wu1 = f1.windU ? f1.windU[n] : 0.f;
        e.wv1 = f1.windV ? f1.windV[n] : 0.f;
        e.su1 = f1.stokesU ? f1.stokesU[n] : 0.f;
        e.sv1 = f1.stokesV ? f1.stokesV[n] : 0.f;
        env[n] = e;
    }
}

cudaError_t pack_pair(int eta, int xi, int sW, const FrameDevice &f0, const FrameDevice &f1,
                      const double *h, NodeRecord *nodes, SurfRecord *surf, cudaStream_t stream) {
    const size_t plane = (size_t)eta * xi;
    pack_nodes_kernel<<<grid_for(plane * sW, 256), 256, 0, stream>>>(eta, xi, sW, f0, f1, nodes);
    pack_surface_kernel<<<grid_for(plane, 256), 256, 0, stream>>>(eta, xi, f0, f1, h, surf);
    return cudaGetLastError();
}

cudaError_t pack_environment(int eta, int xi, const FrameDevice &f0, const FrameDevice &f1,
                             EnvPair *env, cudaStream_t stream) {
    pack_environment_kernel<<<grid_for((size_t)eta * xi, 256), 256, 0, stream>>>(eta, xi, f0, f1,
                                                                               env);
    return cudaGetLastError();
}

// ------------------------------------------------------------------ cell-column packing

size_t cell_record_bytes(int storage) {
    return 2 * (storage == STORE_F32 ? sizeof(CellQuad<STORE_F32>) : sizeof(CellQuad<STORE_F16>));
}
size_t cell_surface_bytes() { return sizeof(CellSurface); }

// Four corners of one field at one record time, in the storage precision (16 or 8 bytes).
template <int STORE>
struct CornerQuad;
template <>
struct CornerQuad<STORE_F32> {
    using type = float4;
    static __device__ __forceinline__ type of(float a, float b, float c, float d) {
        return make_float4(a, b, c, d);
    }
};
template <>
struct CornerQuad<STORE_F16> {
    using type = uint2;
    static __device__ __forceinline__ type of(float a, float b, float c, float d) {
        const __half2 lo = __floats2half2_rn(a, b), hi = __floats2half2_rn(c, d);
        return make_uint2(*reinterpret_cast<const uint32_t *>(&lo), *reinterpret_cast<const uint32_t *>(&hi));
    }
};
template <>
struct CornerQuad<STORE_BF16> {
    using type = uint2;
    static __device__ __forceinline__ type of(float a, float b, float c, float d) {
        const __nv_bfloat162 lo = __floats2bfloat162_rn(a, b), hi = __floats2bfloat162_rn(c, d);
        return make_uint2(*reinterpret_cast<const uint32_t *>(&lo), *reinterpret_cast<const uint32_t *>(&hi));
    }
};

constexpr int PACK_CELLS = 32;   // cells of a block along i
constexpr int PACK_LEVELS = 8;   // W levels of a block
constexpr int PACK_FIELDS = 8;   // u, v, w, akt of two records, in the order of the cell records
// Shared-memory strides: eight fields by four levels fall on 32 banks.
constexpr int PACK_ROW = 36, PACK_LEVEL = 2 * PACK_ROW, PACK_FIELD = PACK_LEVELS * PACK_LEVEL + 1;

// Writes A(L) and B(L) (views.cuh) of 32 cells of a row and 8 W levels per block: the nodes of two
// rows come through shared memory in the fields' own order, the records leave in theirs (each eight
// quads per level, the levels of a cell consecutive), so that both sides of the transposition move
// whole lines. Cells on the last row or column (never valid) are zero. Bound by the record writes:
// 491,520 cells of 25 levels 0.73 ms with one thread per (level, cell) and 128 bytes each, 0.48 ms so
// (4.0 TB/s).
template <int STORE>
__global__ void __launch_bounds__(256) pack_cells_kernel(int eta, int xi, int sW, FrameDevice f0,
                                                         FrameDevice f1, CellQuad<STORE> *cells) {
    using Quads = CornerQuad<STORE>;
    __shared__ float nodes[PACK_FIELDS * PACK_FIELD];
    const int tiles = (xi + PACK_CELLS - 1) / PACK_CELLS;
    const int i0 = (int)(blockIdx.x % tiles) * PACK_CELLS, j = (int)(blockIdx.x / tiles);
    const int L0 = blockIdx.y * PACK_LEVELS;
    const size_t plane = (size_t)eta * xi;
    const bool row = j + 1 < eta;
    const float *fields[PACK_FIELDS] = {f0.u, f1.u, f0.v, f1.v, f0.w, f1.w, f0.akt, f1.akt};
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // warp w stages field w: 33 nodes of two rows per level
    const float *src = fields[warp];
    const int below = warp < 4 ? 1 : 0;  // u, v of rho level L - 1
    float first[PACK_LEVELS * 2], last[PACK_LEVELS * 2];
#pragma unroll
    for (int q = 0; q < PACK_LEVELS * 2; q++) {
        const int L = L0 + (q >> 1) - below, jj = j + (q & 1);
        const bool there = row && L >= 0 && L0 + (q >> 1) < sW;
        const float *line = src + (size_t)(there ? L : 0) * plane + (size_t)(there ? jj : 0) * xi;
        first[q] = there && i0 + lane < xi ? __ldg(line + i0 + lane) : 0.f;
        last[q] = there && lane == 0 && i0 + PACK_CELLS < xi ? __ldg(line + i0 + PACK_CELLS) : 0.f;
    }
#pragma unroll
    for (int q = 0; q < PACK_LEVELS * 2; q++) {
        float *dst = nodes + warp * PACK_FIELD + (q >> 1) * PACK_LEVEL + (q & 1) * PACK_ROW;
        dst[lane] = first[q];
        if (lane == 0) dst[PACK_CELLS] = last[q];
    }
    __syncthreads();
    auto *out = reinterpret_cast<typename Quads::type *>(cells);
    // thread: field f, level l of the cells c, c + 4, ..
    const int f = threadIdx.x & 7, l = (threadIdx.x >> 3) % PACK_LEVELS, c0 = threadIdx.x / 64;
    if (L0 + l >= sW) return;
    const float *n = nodes + f * PACK_FIELD + l * PACK_LEVEL;
    out += (((size_t)j * xi + i0) * sW + L0 + l) * PACK_FIELDS + f;
    const size_t cell = (size_t)sW * PACK_FIELDS;
    const int valid = row ? xi - 1 - i0 : 0, there = xi - i0;  // cells with a record, cells at all
#pragma unroll
    for (int c = c0; c < PACK_CELLS; c += 4) {
        if (c >= there) break;
        typename Quads::type quad = Quads::of(0.f, 0.f, 0.f, 0.f);
        if (c < valid) quad = Quads::of(n[c], n[PACK_ROW + c], n[PACK_ROW + c + 1], n[c + 1]);
        out[(unsigned)c * cell] = quad;
    }
}

__global__ void pack_cell_surface_kernel(int eta, int xi, FrameDevice f0, FrameDevice f1,
                                         const double *h, CellSurface *out) {
    size_t plane = (size_t)eta * xi;
    for (size_t cell = blockIdx.x * (size_t)blockDim.x + threadIdx.x; cell < plane;
         cell += (size_t)gridDim.x * blockDim.x) {
        int j = (int)(cell / xi), i = (int)(cell - (size_t)j * xi);
        CellSurface s;
        if (j + 1 < eta && i + 1 < xi) {
            size_t c1 = cell, c2 = cell + xi, c3 = cell + xi + 1, c4 = cell + 1;
            s.s0 = make_float4((float)h[c1] + f0.zeta[c1], (float)h[c2] + f0.zeta[c2],
                               (float)h[c3] + f0.zeta[c3], (float)h[c4] + f0.zeta[c4]);
            s.dz = make_float4(f1.zeta[c1] - f0.zeta[c1], f1.zeta[c2] - f0.zeta[c2],
                               f1.zeta[c3] - f0.zeta[c3], f1.zeta[c4] - f0.zeta[c4]);
        } else {
            s.s0 = s.dz = make_float4(0, 0, 0, 0);
        }
        out[cell] = s;
    }
}

cudaError_t pack_cells(int storage, int eta, int xi, int sW, const FrameDevice &f0,
                       const FrameDevice &f1, const double *h, void *cells, void *cellSurface,
                       cudaStream_t stream) {
    const dim3 blocks((unsigned)((size_t)((xi + PACK_CELLS - 1) / PACK_CELLS) * eta),
                      (sW + PACK_LEVELS - 1) / PACK_LEVELS);
    switch (storage) {
        case STORE_F16:
            pack_cells_kernel<STORE_F16><<<blocks, 256, 0, stream>>>(
                eta, xi, sW, f0, f1, static_cast<CellQuad<STORE_F16> *>(cells));
            break;
        case STORE_BF16:
            pack_cells_kernel<STORE_BF16><<<blocks, 256, 0, stream>>>(
                eta, xi, sW, f0, f1, static_cast<CellQuad<STORE_BF16> *>(cells));
            break;
        default:
            pack_cells_kernel<STORE_F32><<<blocks, 256, 0, stream>>>(
                eta, xi, sW, f0, f1, static_cast<CellQuad<STORE_F32> *>(cells));
    }
    pack_cell_surface_kernel<<<grid_for((size_t)eta * xi, 256), 256, 0, stream>>>(
        eta, xi, f0, f1, h, static_cast<CellSurface *>(cellSurface));
    return cudaGetLastError();
}

// ------------------------------------------------------------------ cell metric

// Cell sizes in metres along j (ydist) and i (xdist). Host rules: haversine along one grid axis
// with the cross difference dropped (Particle.cpp:548-574); device rules: full haversine between
// the nodes (kernel.cu:145-149,278-279). Cells on the last row/column are never valid.
__global__ void metric_kernel(int semantics, int eta, int xi, const double *lat,
                              const double *lon, CellMetric *metric, float2 *invMetric) {
    size_t plane = (size_t)eta * xi;
    for (size_t n = blockIdx.x * (size_t)blockDim.x + threadIdx.x; n < plane;
         n += (size_t)gridDim.x * blockDim.x) {
        int j = (int)(n / xi), i = (int)(n - (size_t)j * xi);
        if (j + 1 >= eta || i + 1 >= xi) {
            metric[n] = CellMetric{0.0, 0.0, 0.0, 0.0};
            invMetric[n] = make_float2(0.f, 0.f);
            continue;
        }
        double lat0 = lat[n], lon0 = lon[n];
        double latN = lat[n + xi], lonN = lon[n + xi];
        double latE = lat[n + 1], lonE = lon[n + 1];
        double xdist, ydist;
        if (semantics == SEM_HOST) {
            double s = sin(0.5 * (latN - lat0));
            double d = s * s;
            ydist = 2.0 * atan2(sqrt(d), sqrt(1.0 - d)) * 6371000.0;
            s = sin(0.5 * (lonE - lon0));
            d = s * s * cos(latE) * cos(lat0);
            xdist = 2.0 * atan2(sqrt(d), sqrt(1.0 - d)) * 6371000.0;
        } else {
            double dLat = latN - lat0, dLon = lonN - lon0;
            double value = sin(.5 * dLat) * sin(.5 * dLat) + sin(.5 * dLon) * sin(.5 * dLon) * cos(latN) * cos(lat0);
            ydist = 2.0 * atan2(sqrt(value), sqrt(1.0 - value)) * 6371000.0;
            dLat = latE - lat0;
            dLon = lonE - lon0;
            value = sin(.5 * dLat) * sin(.5 * dLat) + sin(.5 * dLon) * sin(.5 * dLon) * cos(latE) * cos(lat0);
            xdist = 2.0 * atan2(sqrt(value), sqrt(1.0 - value)) * 6371000.0;
        }
        metric[n] = CellMetric{xdist, ydist, 1.0 / xdist, 1.0 / ydist};
        invMetric[n] = make_float2((float)(1.0 / xdist), (float)(1.0 / ydist));
    }
}

cudaError_t build_metric(int semantics, int eta, int xi, const double *lonRad,
                         const double *latRad, CellMetric *metric, float2 *invMetric,
                         cudaStream_t stream) {
    metric_kernel<<<grid_for((size_t)eta * xi, 256), 256, 0, stream>>>(semantics, eta, xi, latRad,
                                                                      lonRad, metric, invMetric);
    return cudaGetLastError();
}

// ------------------------------------------------------------------ exclusive scan

constexpr int SCAN_THREADS = 1024;
constexpr int SCAN_ITEMS = 8;
constexpr size_t SCAN_TILE = (size_t)SCAN_THREADS * SCAN_ITEMS;

__device__ __forceinline__ uint32_t block_exclusive(uint32_t value, uint32_t *shared,
                                                    uint32_t &blockTotal) {
    int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t inclusive = value;
    for (int off = 1; off < 32; off <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, inclusive, off);
        if (lane >= off) inclusive += y;
    }
    if (lane == 31) shared[warp] = inclusive;
    __syncthreads();
    if (warp == 0) {
        uint32_t s = lane < (int)(blockDim.x >> 5) ? shared[lane] : 0;
        uint32_t inc = s;
        for (int off = 1; off < 32; off <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, inc, off);
            if (lane >= off) inc += y;
        }
        shared[lane] = inc - s;
        if (lane == 31) shared[32] = inc;
    }
    __syncthreads();
    uint32_t result = shared[warp] + inclusive - value;
    blockTotal = shared[32];
    __syncthreads();
    return result;
}

__global__ void __launch_bounds__(SCAN_THREADS) scan_reduce_kernel(const uint32_t *in, size_t n,
                                                                   uint32_t *sums) {
    __shared__ uint32_t shared[33];
    size_t base = blockIdx.x * SCAN_TILE + (size_t)threadIdx.x * SCAN_ITEMS;
    uint32_t s = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; k++)
        if (base + k < n) s += in[base + k];
    uint32_t total;
    block_exclusive(s, shared, total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(SCAN_THREADS) scan_apply_kernel(const uint32_t *in, uint32_t *out,
                                                                  size_t n,
                                                                  const uint32_t *offsets,
                                                                  uint32_t *total) {
    __shared__ uint32_t shared[33];
    size_t base = blockIdx.x * SCAN_TILE + (size_t)threadIdx.x * SCAN_ITEMS;
    uint32_t v[SCAN_ITEMS];
    uint32_t s = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; k++) {
        v[k] = base + k < n ? in[base + k] : 0;
        s += v[k];
    }
    uint32_t blockTotal;
    uint32_t run = block_exclusive(s, shared, blockTotal) + (offsets ? offsets[blockIdx.x] : 0);
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; k++) {
        if (base + k < n) out[base + k] = run;
        run += v[k];
    }
    if (total && blockIdx.x == gridDim.x - 1 && threadIdx.x == blockDim.x - 1) *total = run;
}

size_t scan_temp_words(size_t n) {
    size_t words = 0;
    while (n > SCAN_TILE) {
        size_t blocks = (n + SCAN_TILE - 1) / SCAN_TILE;
        words += 2 * blocks;
        n = blocks;
    }
    return words + 2;
}

cudaError_t exclusive_scan(const uint32_t *in, uint32_t *out, size_t n, uint32_t *total,
                           uint32_t *temp, cudaStream_t stream) {
    if (n == 0) {
        if (total) cudaMemsetAsync(total, 0, sizeof(uint32_t), stream);
        return cudaGetLastError();
    }
    size_t blocks = (n + SCAN_TILE - 1) / SCAN_TILE;
    if (blocks == 1) {
        scan_apply_kernel<<<1, SCAN_THREADS, 0, stream>>>(in, out, n, nullptr, total);
        return cudaGetLastError();
    }
    uint32_t *sums = temp, *sumOffsets = temp + blocks;
    scan_reduce_kernel<<<(unsigned)blocks, SCAN_THREADS, 0, stream>>>(in, n, sums);
    cudaError_t e = exclusive_scan(sums, sumOffsets, blocks, nullptr, temp + 2 * blocks, stream);
    if (e != cudaSuccess) return e;
    scan_apply_kernel<<<(unsigned)blocks, SCAN_THREADS, 0, stream>>>(in, out, n, sumOffsets, total);
    return cudaGetLastError();
}

// ------------------------------------------------------------------ counting sort by cell

// The bin of a record (SortBins): its cell, its level from the surface down when the bins are split by
// level, its release time; the last bin for a record that takes no step.
__device__ __forceinline__ uint32_t sort_key(const SortBins &B, double k, double j, double i,
                                             double time) {
    const double fj = floor(j), fi = floor(i);
    if (!(fj >= 0.0 && fi >= 0.0 && fj < (double)(B.eta - 1) && fi < (double)(B.xi - 1)) ||
        time >= B.end)
        return (uint32_t)((size_t)B.eta * B.xi * B.levels * B.late);
    uint32_t key = (uint32_t)((int)fj * B.xi + (int)fi);
    if (B.levels > 1) {
        const double down = fmin(fmax(-ceil(k), 0.0), (double)(B.levels - 1));
        key = key * (uint32_t)B.levels + (uint32_t)down;
    }
    if (B.late > 1) {
        key *= (uint32_t)B.late;
        if (time > B.start) {
            const float part = (float)(time - B.start) / (float)(B.end - B.start);
            key += 1 + (uint32_t)fminf(part * (float)(B.late - 1), (float)(B.late - 2));
        }
    }
    return key;
}

// Both passes walk the records in the sequence `seq` (a permutation of the slots, or the identity
// when null); keys are kept in sequence order. Walking in the previous interval's cell order puts
// the records of one cell next to each other, so a warp's atomics collapse to one per cell even
// where walls gather hundreds of thousands of records into a few cells.
__global__ void key_histogram_kernel(const ParticleSoA S, int n, const SortBins B,
                                     const uint32_t *seq, uint32_t *keys, uint32_t *hist) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const uint32_t p = seq ? seq[t] : (uint32_t)t;
        uint32_t key = sort_key(B, B.levels > 1 ? S.k[p] : 0.0, S.j[p], S.i[p], S.time[p]);
        keys[t] = key;
        unsigned active = __activemask();
        unsigned peers = __match_any_sync(active, key);
        if ((threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(hist + key, (uint32_t)__popc(peers));
    }
}

__global__ void key_scatter_kernel(const uint32_t *keys, int n, const uint32_t *seq,
                                   uint32_t *cursor, uint32_t *order) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        uint32_t key = keys[t];
        unsigned active = __activemask();
        unsigned peers = __match_any_sync(active, key);
        int lane = threadIdx.x & 31;
        int leader = __ffs(peers) - 1;
        uint32_t base = 0;
        if (lane == leader) base = atomicAdd(cursor + key, (uint32_t)__popc(peers));
        base = __shfl_sync(peers, base, leader);
        uint32_t rank = __popc(peers & ((1u << lane) - 1u));
        order[base + rank] = seq ? seq[t] : (uint32_t)t;
    }
}

cudaError_t sort_by_cell(const ParticleSoA &S, int n, const SortBins &bins, const uint32_t *seq,
                         uint32_t *keys, uint32_t *hist, uint32_t *offsets, uint32_t *temp,
                         uint32_t *order, cudaStream_t stream) {
    const size_t count = bins.count();
    cudaMemsetAsync(hist, 0, count * sizeof(uint32_t), stream);
    int blocks = grid_for((size_t)n, 256);
    key_histogram_kernel<<<blocks, 256, 0, stream>>>(S, n, bins, seq, keys, hist);
    cudaError_t e = exclusive_scan(hist, offsets, count, offsets + count, temp, stream);
    if (e != cudaSuccess) return e;
    key_scatter_kernel<<<blocks, 256, 0, stream>>>(keys, n, seq, offsets, order);
    return cudaGetLastError();
}

// ------------------------------------------------------------------ random draws ahead of the step

// The draws of the reference keys depend on the record, the interval and the substep alone, not on
// the path: a small launch, whose time is the latency of its substep chain, has them drawn here by
// one thread per (substep, record) instead of one after the other inside the chain. Bound by FP64
// issue (log, square root and cosine of three normals): 20,011 records x 121 substeps in about
// 0.05 ms; the move kernel they feed takes 0.26 ms instead of 0.48 ms (1,021 records: 0.18 instead of
// 0.40 ms).
__global__ void __launch_bounds__(256) draw_normals_kernel(const uint64_t *id, unsigned count,
                                                          uint64_t seed, long long interval,
                                                          unsigned steps, float4 *out) {
    const size_t total = (size_t)steps * count;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total;
         e += (size_t)gridDim.x * blockDim.x) {
        const unsigned s = (unsigned)(e / count), slot = (unsigned)(e - (size_t)s * count);
        const uint64_t key = key_prefix(seed, id[slot], interval, s);
        out[e] = make_float4(prefix_normal_f32(key, 0), prefix_normal_f32(key, 1),
                             prefix_normal_f32(key, 2), 0.f);
    }
}

cudaError_t draw_normals(const uint64_t *id, int count, uint64_t seed, long long interval,
                         unsigned steps, float4 *out, cudaStream_t stream) {
    if (count <= 0 || !steps) return cudaSuccess;
    draw_normals_kernel<<<grid_for((size_t)steps * count, 256), 256, 0, stream>>>(
        id, (unsigned)count, seed, interval, steps, out);
    return cudaGetLastError();
}

// ------------------------------------------------------------------ record layout

__global__ void aos_to_soa_kernel(const wacomm_b200_particle *aos, int n, ParticleSoA S) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        wacomm_b200_particle r = aos[p];
        S.id[p] = r.id;
        S.k[p] = r.k;
        S.j[p] = r.j;
        S.i[p] = r.i;
        S.health[p] = r.health;
        S.age[p] = r.age;
        S.time[p] = r.time;
        S.type[p] = r.driftObjectType;
        S.side[p] = r.driftSide;
    }
}

// 256 records per block and turn through shared memory, so that they leave as whole lines. Bound by
// memory (59 bytes in, 64 out). With 64 bytes stored per thread 43 us at 1 M records and 19 us at
// 0.4 M; so 17 and 10 us.
__global__ void __launch_bounds__(256) soa_to_aos_kernel(ParticleSoA S, int n, wacomm_b200_particle *aos) {
    static_assert(sizeof(wacomm_b200_particle) == 64 && offsetof(wacomm_b200_particle, driftObjectType) == 56 &&
                      offsetof(wacomm_b200_particle, driftSide) == 58,
                  "record layout");
    __shared__ unsigned long long words[256 * 9];  // a record's 8 words, 9 apart: no bank conflicts
    auto *out = reinterpret_cast<unsigned long long *>(aos);
    for (long long base = blockIdx.x * 256ll; base < n; base += gridDim.x * 256ll) {
        const long long p = base + threadIdx.x;
        if (p < n) {
            unsigned long long *w = words + threadIdx.x * 9;
            w[0] = S.id[p];
            w[1] = (unsigned long long)__double_as_longlong(S.k[p]);
            w[2] = (unsigned long long)__double_as_longlong(S.j[p]);
            w[3] = (unsigned long long)__double_as_longlong(S.i[p]);
            w[4] = (unsigned long long)__double_as_longlong(S.health[p]);
            w[5] = (unsigned long long)__double_as_longlong(S.age[p]);
            w[6] = (unsigned long long)__double_as_longlong(S.time[p]);
            // type, side, zero padding
            w[7] = (unsigned long long)S.type[p] | (unsigned long long)(uint8_t)S.side[p] << 16;
        }
        __syncthreads();
        const long long left = n - base < 256 ? n - base : 256;
        for (int e = threadIdx.x; e < left * 8; e += 256) out[base * 8 + e] = words[(e >> 3) * 9 + (e & 7)];
        __syncthreads();
    }
}

cudaError_t aos_to_soa(const wacomm_b200_particle *aos, int n, const ParticleSoA &S,
                       cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    aos_to_soa_kernel<<<grid_for(n, 256), 256, 0, stream>>>(aos, n, S);
    return cudaGetLastError();
}

cudaError_t soa_to_aos(const ParticleSoA &S, int n, wacomm_b200_particle *aos,
                       cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    soa_to_aos_kernel<<<grid_for(n, 256), 256, 0, stream>>>(S, n, aos);
    return cudaGetLastError();
}

// ------------------------------------------------------------------ dead-particle removal

__global__ void alive_flags_kernel(const double *health, int n, uint32_t *flags) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x)
        flags[p] = health[p] > 0 ? 1u : 0u;
}

__global__ void compact_kernel(ParticleSoA S, int n, const uint32_t *flags,
                               const uint32_t *positions, ParticleSoA T) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        if (!flags[p]) continue;
        uint32_t q = positions[p];
        T.id[q] = S.id[p];
        T.k[q] = S.k[p];
        T.j[q] = S.j[p];
        T.i[q] = S.i[p];
        T.health[q] = S.health[p];
        T.age[q] = S.age[p];
        T.time[q] = S.time[p];
        T.type[q] = S.type[p];
        T.side[q] = S.side[p];
    }
}

cudaError_t compact_alive(const ParticleSoA &S, int n, const ParticleSoA &tmp, uint32_t *flags,
                          uint32_t *positions, uint32_t *temp, uint32_t *kept,
                          cudaStream_t stream) {
    if (n <= 0) {
        cudaMemsetAsync(kept, 0, sizeof(uint32_t), stream);
        return cudaGetLastError();
    }
    int blocks = grid_for(n, 256);
    alive_flags_kernel<<<blocks, 256, 0, stream>>>(S.health, n, flags);
    cudaError_t e = exclusive_scan(flags, positions, n, kept, temp, stream);
    if (e != cudaSuccess) return e;
    compact_kernel<<<blocks, 256, 0, stream>>>(S, n, flags, positions, tmp);
    return cudaGetLastError();
}

// ------------------------------------------------------------------ concentration

__global__ void count_kernel(ParticleSoA S, int n, int concTime, int sRho, int eta, int xi,
                             uint32_t *conc) {
    for (int base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
        int p = base + threadIdx.x;
        long long cell = -1;
        if (p < n) {
            ParticleState s;
            s.k = S.k[p];
            s.j = S.j[p];
            s.i = S.i[p];
            s.health = S.health[p];
            cell = concentration_cell(s, concTime, sRho, eta, xi);
        }
        warp_count(conc, cell);
    }
}

__global__ void accumulate_steps_kernel(const unsigned long long *steps,
                                        unsigned long long *total) {
    *total += *steps;
}

cudaError_t accumulate_steps(const unsigned long long *steps, unsigned long long *total,
                             cudaStream_t stream) {
    accumulate_steps_kernel<<<1, 1, 0, stream>>>(steps, total);
    return cudaGetLastError();
}

cudaError_t count_concentration(const ParticleSoA &S, int n, int concTime, int sRho, int eta,
                                int xi, uint32_t *conc, cudaStream_t stream) {
    if (n <= 0) return cudaSuccess;
    count_kernel<<<grid_for(n, 256), 256, 0, stream>>>(S, n, concTime, sRho, eta, xi, conc);
    return cudaGetLastError();
}

// Float grid of the reference (counts as float, exact below 2^24) with the land mask of
// Wacomm.cpp:188-196,724-739 (mask != 1 -> 1e37 in every level).
__global__ void to_float_kernel(const uint32_t *conc, size_t n, int plane, const double *mask,
                                float *out) {
    for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < n;
         q += (size_t)gridDim.x * blockDim.x) {
        float value = (float)conc[q];
        if (mask && mask[q % plane] != 1.0) value = 1e37f;
        out[q] = value;
    }
}

cudaError_t concentration_to_float(const uint32_t *conc, size_t n, int nTimes, int sRho, int eta,
                                   int xi, const double *mask, float *out, cudaStream_t stream) {
    (void)nTimes;
    (void)sRho;
    if (n == 0) return cudaSuccess;
    to_float_kernel<<<grid_for(n, 256), 256, 0, stream>>>(conc, n, eta * xi, mask, out);
    return cudaGetLastError();
}

}  // namespace wb
