// Forcing views: how the step reads the bracketing forcing pair.
//
// PackedView is the engine layout of the reference arithmetic. For each interval the two bracketing
// records are interleaved into one node record per (W level L, j, i), as doubles:
//     {w(L), akt(L), u(L-1), v(L-1)} of record t0 and t1
// so that one particle's trilinear stencil (4 corners x 2 levels) is 8 records instead of 48 scalar
// gathers from four fields and two frames, and the step's FP64 products read their operands without
// a float-to-double conversion each (a quarter-rate instruction; there are more of them in a substep
// than anything else on that unit). Surface data sit in a {h, zeta(t0), zeta(t1)} record per node,
// the optional wind/Stokes pair in a 32-byte record, the cell metric in a per-cell table. The FP32
// step shares the wind/Stokes pair and the grid.
//
// RawView reads the reference device layout directly (kernel.cu:63-80): it serves the drop-in
// launcher, whose caller owns separate field arrays for the whole window.
#pragma once

#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"

namespace wb {

template <class T>
struct SurfPair {
    double h;
    T z0, z1;
};
struct EnvPair {
    float wu0, wv0, su0, sv0, wu1, wv1, su1, sv1;
};

// Records of the packed pair: {t0, t1} per field.
struct alignas(16) NodeRecord {
    double2 w, akt, u, v;
};
// The records of a block of 256 threads, nodes base .. base + 255, leave through shared memory as whole
// lines (all threads of the block call this). Bound by memory (32 bytes read and 64 written per node):
// 12.3 M nodes 0.251 ms with 64 bytes stored per thread, 0.183 ms so (6.5 TB/s).
struct NodeStage {
    double2 field[4][258];  // two pairs of padding: no bank conflicts on the way out
};
__device__ __forceinline__ void store_nodes(NodeStage &stage, const NodeRecord &r, size_t base,
                                            size_t total, NodeRecord *nodes) {
    static_assert(offsetof(NodeRecord, akt) == 16 && offsetof(NodeRecord, u) == 32 &&
                      offsetof(NodeRecord, v) == 48 && sizeof(NodeRecord) == 64, "record layout");
    stage.field[0][threadIdx.x] = r.w;
    stage.field[1][threadIdx.x] = r.akt;
    stage.field[2][threadIdx.x] = r.u;
    stage.field[3][threadIdx.x] = r.v;
    __syncthreads();
    double2 *out = reinterpret_cast<double2 *>(nodes + base);
    const int left = total - base < 256 ? (int)(total - base) * 4 : 1024;
    for (int e = threadIdx.x; e < left; e += 256) out[e] = stage.field[e & 3][e >> 2];
    __syncthreads();
}
struct alignas(16) SurfRecord {
    double h, z0, z1, unused;
};

// Cell sizes in metres along i and j and their correctly rounded reciprocals.
struct CellMetric {
    double x, y, rx, ry;
};

// The velocity stencil of one cell and level: u, v (rho level kI) and w (W levels kI and kI-1) at the
// corners (j,i), (j+1,i), (j+1,i+1), (j,i+1) of records t0 and t1.
struct RefStencil {
    double2 u[4], v[4], wUp[4], wLo[4];  // {t0, t1}
};

// Grid-level constants every view shares.
struct GridShape {
    int eta, xi, sW, sRho;
};

struct PackedView {
    GridShape g;
    const NodeRecord *nodes;         // [sW][eta][xi]
    const SurfRecord *surf;          // [eta][xi]
    const EnvPair *env;              // [eta][xi] or null
    bool hasWindU, hasWindV, hasStokes;
    const double *lonRad, *latRad;   // [eta][xi]
    const double *depthIntervals;    // [sW-1]
    const CellMetric *metric;        // [eta][xi]

    __device__ __forceinline__ size_t node_index(int L, int j, int i) const {
        return ((size_t)L * (size_t)g.eta + (size_t)j) * (size_t)g.xi + (size_t)i;
    }
    // Stencil of logical level kI, kI in [-sW+2, 0].
    __device__ __forceinline__ void stencil(int kI, int j, int i, RefStencil &s) const {
        const NodeRecord *up = nodes + node_index(kI + g.sW - 1, j, i);
        const NodeRecord *lo = nodes + node_index(kI + g.sW - 2, j, i);
        const int corner[4] = {0, g.xi, g.xi + 1, 1};
#pragma unroll
        for (int c = 0; c < 4; c++) {
            s.u[c] = __ldg(&up[corner[c]].u);
            s.v[c] = __ldg(&up[corner[c]].v);
            s.wUp[c] = __ldg(&up[corner[c]].w);
            s.wLo[c] = __ldg(&lo[corner[c]].w);
        }
    }
    // Diffusivity {t0, t1} at W level kI.
    __device__ __forceinline__ double2 akt(int kI, int j, int i) const {
        return __ldg(&nodes[node_index(kI + g.sW - 1, j, i)].akt);
    }
    __device__ __forceinline__ SurfPair<double> surface(int j, int i) const {
        const double2 *s = reinterpret_cast<const double2 *>(surf + ((size_t)j * g.xi + i));
        const double2 hz = __ldg(s), z = __ldg(s + 1);
        return SurfPair<double>{hz.x, hz.y, z.x};
    }
    __device__ __forceinline__ EnvPair environment(int j, int i) const {
        const float4 *p = reinterpret_cast<const float4 *>(env + (size_t)j * g.xi + i);
        float4 a = __ldg(p), b = __ldg(p + 1);
        return EnvPair{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    }
    __device__ __forceinline__ double lon(int j, int i) const { return __ldg(lonRad + (size_t)j * g.xi + i); }
    __device__ __forceinline__ double lat(int j, int i) const { return __ldg(latRad + (size_t)j * g.xi + i); }
    __device__ __forceinline__ double depth_interval(int kI) const {
        return __ldg(depthIntervals + (kI + g.sW - 2));
    }
    __device__ __forceinline__ CellMetric cell_metric(int j, int i) const {
        const double2 *m = reinterpret_cast<const double2 *>(metric + ((size_t)j * g.xi + i));
        const double2 size = __ldg(m), reciprocal = __ldg(m + 1);
        return CellMetric{size.x, size.y, reciprocal.x, reciprocal.y};
    }
};

// ------------------------------------------------------------------ cell-column layout
// FP32 step layout. For every cell (j, i) and W level L the bracketing pair is stored at the
// four corners of the cell, corner order (j,i), (j+1,i), (j+1,i+1), (j,i+1):
//     A(L) = u, v of rho level L-1        B(L) = w, akt of W level L
// each as {field0 @ t0, field0 @ t1, field1 @ t0, field1 @ t1} x 4 corners, and the records of a
// cell are consecutive in L: ... A(L-1) B(L-1) A(L) B(L) ... so the stencil of a particle at
// level kI (L = kI + sW - 1) is the contiguous run B(L-1), A(L), B(L) read from one address.
// Surface per cell: h at the corners, zeta at t0 and t1 at the corners.

template <int STORE>
struct CellQuad;  // one field pair at 4 corners x 2 records
template <>
struct alignas(16) CellQuad<STORE_F32> {
    float4 a0, a1, b0, b1;  // field a @t0 corners, a @t1, field b @t0, b @t1
};
template <>
struct alignas(16) CellQuad<STORE_F16> {
    __half2 a0[2], a1[2], b0[2], b1[2];
};
template <>
struct alignas(16) CellQuad<STORE_BF16> {
    __nv_bfloat162 a0[2], a1[2], b0[2], b1[2];
};

struct Quad {
    float c1, c2, c3, c4;
};
struct QuadPair {  // a field at 4 corners for the two bracketing records
    Quad t0, t1;
};

__device__ __forceinline__ Quad quad_of(float4 v) { return Quad{v.x, v.y, v.z, v.w}; }

__device__ __forceinline__ Quad quad_h(uint32_t x, uint32_t y) {
    float2 lo = __half22float2(*reinterpret_cast<__half2 *>(&x));
    float2 hi = __half22float2(*reinterpret_cast<__half2 *>(&y));
    return Quad{lo.x, lo.y, hi.x, hi.y};
}
__device__ __forceinline__ Quad quad_bf(uint32_t x, uint32_t y) {
    float2 lo = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162 *>(&x));
    float2 hi = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162 *>(&y));
    return Quad{lo.x, lo.y, hi.x, hi.y};
}

// The velocity stencil of one cell and level: u, v and the two w levels at the bracketing records.
struct Stencil {
    QuadPair u, v, wUp, wLo;
};

// The first field of a CellQuad only (u of an A record, w of a B record).
template <int STORE>
__device__ __forceinline__ void load_first(const CellQuad<STORE> *p, QuadPair &a);

template <>
__device__ __forceinline__ void load_first<STORE_F32>(const CellQuad<STORE_F32> *p, QuadPair &a) {
    const float4 *q = reinterpret_cast<const float4 *>(p);
    a.t0 = quad_of(__ldg(q));
    a.t1 = quad_of(__ldg(q + 1));
}

template <>
__device__ __forceinline__ void load_first<STORE_F16>(const CellQuad<STORE_F16> *p, QuadPair &a) {
    uint4 x = __ldg(reinterpret_cast<const uint4 *>(p));
    a.t0 = quad_h(x.x, x.y);
    a.t1 = quad_h(x.z, x.w);
}

template <>
__device__ __forceinline__ void load_first<STORE_BF16>(const CellQuad<STORE_BF16> *p, QuadPair &a) {
    uint4 x = __ldg(reinterpret_cast<const uint4 *>(p));
    a.t0 = quad_bf(x.x, x.y);
    a.t1 = quad_bf(x.z, x.w);
}

// The second field of a CellQuad only (v of an A record, akt of a B record).
template <int STORE>
__device__ __forceinline__ void load_second(const CellQuad<STORE> *p, QuadPair &b);

template <>
__device__ __forceinline__ void load_second<STORE_F32>(const CellQuad<STORE_F32> *p, QuadPair &b) {
    const float4 *q = reinterpret_cast<const float4 *>(p);
    b.t0 = quad_of(__ldg(q + 2));
    b.t1 = quad_of(__ldg(q + 3));
}

template <>
__device__ __forceinline__ void load_second<STORE_F16>(const CellQuad<STORE_F16> *p, QuadPair &b) {
    uint4 y = __ldg(reinterpret_cast<const uint4 *>(p) + 1);
    b.t0 = quad_h(y.x, y.y);
    b.t1 = quad_h(y.z, y.w);
}

template <>
__device__ __forceinline__ void load_second<STORE_BF16>(const CellQuad<STORE_BF16> *p, QuadPair &b) {
    uint4 y = __ldg(reinterpret_cast<const uint4 *>(p) + 1);
    b.t0 = quad_bf(y.x, y.y);
    b.t1 = quad_bf(y.z, y.w);
}

struct CellSurface {  // FP32 at the 4 corners: h + zeta@t0, and zeta@t1 - zeta@t0
    float4 s0, dz;
};

template <int STORE>
struct CellView {
    int eta, xi, sW;
    const CellQuad<STORE> *columns;   // [cell][sW][2] (A, B)
    const CellSurface *surface;       // [cell]

    // Columns are numbered cell * sW + L (L = kI + sW - 1, kI a valid memory level, cell =
    // j xi + i); 32 bits number more columns than the device's memory holds.

    // Velocity stencil of a column: u, v at rho level kI; w at W levels kI (up) and kI-1 (lo).
    __device__ __forceinline__ void stencil(uint32_t column, Stencil &s) const {
        const CellQuad<STORE> *col = columns + 2 * (size_t)column;
        load_first<STORE>(col - 1, s.wLo);  // B(L-1)
        load_first<STORE>(col, s.u);        // A(L)
        load_second<STORE>(col, s.v);
        load_first<STORE>(col + 1, s.wUp);  // B(L)
    }
    // Diffusivity at W levels kI (up) and kI-1 (lo) of a column.
    __device__ __forceinline__ void akt(uint32_t column, QuadPair &up, QuadPair &lo) const {
        const CellQuad<STORE> *col = columns + 2 * (size_t)column;
        load_second<STORE>(col - 1, lo);
        load_second<STORE>(col + 1, up);
    }
    __device__ __forceinline__ CellSurface surf(uint32_t cell) const {
        const float4 *q = reinterpret_cast<const float4 *>(surface + cell);
        return CellSurface{__ldg(q), __ldg(q + 1)};
    }
};

// Reference device layout (kernel.cu:63-69), whole window, records t0/t1 given per interval.
struct RawView {
    GridShape g;
    int t0, t1;
    const float *zeta, *u, *v, *w, *aktField;
    const float *windU, *windV, *stokesU, *stokesV;
    const double *hField, *lonRad, *latRad, *depthIntervals;
    bool hasWindU, hasWindV, hasStokes;

    __device__ __forceinline__ size_t plane() const { return (size_t)g.eta * (size_t)g.xi; }
    __device__ __forceinline__ size_t i3(int t, int j, int i) const {
        return ((size_t)t * g.eta + j) * g.xi + i;
    }
    __device__ __forceinline__ size_t i4(int t, int storageLevel, int levels, int j, int i) const {
        return (((size_t)t * levels + storageLevel) * g.eta + j) * g.xi + i;
    }
    __device__ __forceinline__ double2 pair(const float *field, int level, int levels, int j,
                                            int i) const {
        return make_double2(__ldg(field + i4(t0, level, levels, j, i)),
                            __ldg(field + i4(t1, level, levels, j, i)));
    }
    __device__ __forceinline__ void stencil(int kI, int j, int i, RefStencil &s) const {
        const int Lr = kI + g.sRho - 1, Lw = kI + g.sW - 1;
        const int dj[4] = {0, 1, 1, 0}, di[4] = {0, 0, 1, 1};
#pragma unroll
        for (int c = 0; c < 4; c++) {
            s.u[c] = pair(u, Lr, g.sRho, j + dj[c], i + di[c]);
            s.v[c] = pair(v, Lr, g.sRho, j + dj[c], i + di[c]);
            s.wUp[c] = pair(w, Lw, g.sW, j + dj[c], i + di[c]);
            s.wLo[c] = pair(w, Lw - 1, g.sW, j + dj[c], i + di[c]);
        }
    }
    __device__ __forceinline__ double2 akt(int kI, int j, int i) const {
        return pair(aktField, kI + g.sW - 1, g.sW, j, i);
    }
    __device__ __forceinline__ SurfPair<float> surface(int j, int i) const {
        return SurfPair<float>{__ldg(hField + (size_t)j * g.xi + i), __ldg(zeta + i3(t0, j, i)),
                        __ldg(zeta + i3(t1, j, i))};
    }
    __device__ __forceinline__ EnvPair environment(int j, int i) const {
        EnvPair e{0, 0, 0, 0, 0, 0, 0, 0};
        if (hasWindU) { e.wu0 = __ldg(windU + i3(t0, j, i)); e.wu1 = __ldg(windU + i3(t1, j, i)); }
        if (hasWindV) { e.wv0 = __ldg(windV + i3(t0, j, i)); e.wv1 = __ldg(windV + i3(t1, j, i)); }
        if (hasStokes) {
            e.su0 = __ldg(stokesU + i3(t0, j, i)); e.su1 = __ldg(stokesU + i3(t1, j, i));
            e.sv0 = __ldg(stokesV + i3(t0, j, i)); e.sv1 = __ldg(stokesV + i3(t1, j, i));
        }
        return e;
    }
    __device__ __forceinline__ double lon(int j, int i) const { return __ldg(lonRad + (size_t)j * g.xi + i); }
    __device__ __forceinline__ double lat(int j, int i) const { return __ldg(latRad + (size_t)j * g.xi + i); }
    __device__ __forceinline__ double depth_interval(int kI) const {
        return __ldg(depthIntervals + (kI + g.sW - 2));
    }
    // Full haversine between the nodes of the cell's edges (kernel.cu:145-149,278-279).
    __device__ __forceinline__ CellMetric cell_metric(int j, int i) const {
        double lat0 = lat(j, i), lon0 = lon(j, i);
        double latN = lat(j + 1, i), lonN = lon(j + 1, i);
        double latE = lat(j, i + 1), lonE = lon(j, i + 1);
        double dLat = latN - lat0, dLon = lonN - lon0;
        double value = sin(.5 * dLat) * sin(.5 * dLat) + sin(.5 * dLon) * sin(.5 * dLon) * cos(latN) * cos(lat0);
        double ydist = 2.0 * atan2(sqrt(value), sqrt(1.0 - value)) * 6371000.0;
        dLat = latE - lat0;
        dLon = lonE - lon0;
        value = sin(.5 * dLat) * sin(.5 * dLat) + sin(.5 * dLon) * sin(.5 * dLon) * cos(latE) * cos(lat0);
        double xdist = 2.0 * atan2(sqrt(value), sqrt(1.0 - value)) * 6371000.0;
        return CellMetric{xdist, ydist, 1.0 / xdist, 1.0 / ydist};
    }
};

}  // namespace wb
