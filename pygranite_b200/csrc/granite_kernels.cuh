// granite_kernels.cuh — sm_100a device code of the trajectory step path.
//
// One thread owns one particle.  A launch advances its particle through a range of steps
// (one or more snapshot windows) with the particle state in registers; the reference
// instead launches `integrate` once per step on a single 512-thread block and
// double-buffers AoS positions through global memory (TrajectoryIntegrator.tpp:108-457,
// 790-796, 978-984).  Per step the uniform data (time weights, save slots, ring slots)
// comes from a small device schedule.
//
// Arithmetic follows one fixed operation order, spelled out with __fmaf_rn and compiled
// with --fmad=false, so the float32 oracle build reproduces it bit for bit.  Wind is
// stored node-major: float4 {u,v,w,0} (3D) or float2 {u,v} (2D) per node for float32,
// four / two 16-bit values per node for bf16 / fp16.  Hardware texture filtering (8-bit
// weights, TrajectoryIntegrator.cpp:503-505) is replaced by float32 interpolation.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#ifdef __CUDACC_RTC__
// run-time compilation of the deferred volume / expression kernel (jit.cu): no host headers
typedef signed char int8_t;
typedef short int16_t;
typedef int int32_t;
typedef long long int64_t;
typedef unsigned char uint8_t;
typedef unsigned short uint16_t;
typedef unsigned int uint32_t;
typedef unsigned long long uint64_t;
namespace std {
template <class A, class B> struct is_same { static constexpr bool value = false; };
template <class A> struct is_same<A, A> { static constexpr bool value = true; };
}  // namespace std
#else
#include <cstdint>
#include <type_traits>
#endif

#include "expr.h"

namespace granite_b200 {

constexpr int GR_MAX_VOL = 8;
constexpr int GR_MAX_EXPR = 4;
constexpr int GR_MAX_CON = 4;

// Compile-time feature sets of the step kernel.  FT_GENERIC honours every runtime option.  A
// lean variant (FT_LEAN) is picked by the host (kernel_features in advance.h) when the launch has a
// dynamic windfield, no uplift, length abort, topography or per-step alive counts, and curvature
// Off or Total; without FT_BORDER also no sphere coordinates, loop borders, 1/256 filter weights or wide
// grid.  FT_CURV / FT_EXTRAS say whether it keeps total curvature and volume
// / expression values, FT_COMP Kahan-compensated positions (instantiated without extras: the
// precision form).  FT_DEFER (with FT_LEAN, instead of FT_EXTRAS) leaves the volume / expression
// values to deferred_extras_kernel after the launch: the step kernel only stores each moved step's
// stage-averaged velocity and step index, and hands them to the record at a save step.  The lean
// variants drop the dead state from registers; their arithmetic is the generic variant's.
// FT_BORDER (with FT_LEAN alone) keeps the loop borders, sphere coordinates, 1/256 filter weights and
// wide grids as runtime options: positions on a sphere or in a periodic domain.
constexpr int FT_GENERIC = 0, FT_LEAN = 1, FT_CURV = 2, FT_EXTRAS = 4, FT_COMP = 8, FT_DEFER = 16, FT_BORDER = 32;

// Step-schedule flags.
constexpr int SF_SAVE = 1;       // position / info record after this step
constexpr int SF_TIME_POS = 2;   // data.Time > 0 at the start of the step
constexpr int SF_CURV_REC = 4;   // curvature record after this step (IndividualAndTotal)

struct StepEntry {
    float t0, t1, t2;      // time weights of the RK4 stages (t1 also for k3)
    int32_t flags;
    int32_t slot_back, slot_front;   // ring slots of the window's snapshots
    int32_t rec, crec, irec;
    int32_t pad[3];
};   // read as 16-byte words (advance_particle)

struct KParams {
    // geometry (TrajectoryIntegrator.tpp:521-574)
    float inv_scale[3], off[3], dom[3], scale[3];
    int32_t nx, ny, nz, dim;
    float fn[3], flo;             // clamp of a sample's grid coordinates: [flo, fn] (clamp_cells)
    int32_t below;                // cells -below .. n + below - 1 are read as they are
    int32_t wide;                 // 1: a grid too large for make_pcell or the cell index (ring layouts only)
    // operand pairs of the paired instructions and -off: world position -> grid is
    // (p + noff) * inv_scale
    float2 noff2, inv2, h2, hh2, sixth2, i2h2, ihh2;
    float noffz;
    // ring buffers: slot s of quantity q starts at base + s * stride
    const void *wind;
    int64_t wind_stride;          // bytes per slot
    const void *pair;             // window-pair buffer of the launch's window (pair layouts)
    int32_t pnx, pnxy;            // window pair: padded row length (nx + 3) and plane size
                                  // ((nx + 3) * (ny + 3)); node (x, y, z) at
                                  // (z + 1) * pnxy + (y + 1) * pnx + (x + 1): zeros outside the
                                  // grid in 3D, the clamped edge node in 2D
    const float *vol;             // [slot][8][plane]
    int64_t vol_plane;            // floats per plane
    const float *cons;            // [slot][4][n_total]
    const float *lift;            // [slot][n_total * dim]
    const float *topo;            // (ny, nx)
    // particle state, slot order
    float *px, *py, *pz;          // position
    float *qx, *qy, *qz;          // previous position (curvature pm1)
    float *kx, *ky, *kz;          // Kahan compensation
    float *lx, *ly, *lz;          // last direction (FastTotal curvature)
    int32_t *status;
    float *length, *tc, *curv;
    float *volc;                  // [8][n_state]
    float *cmpc;                  // [4][n_state]
    float4 *vlast;                // FT_DEFER: (stage-averaged velocity, step index as int bits) of
                                  // each slot's last moved step; index -1: no step since the values
                                  // were last evaluated (or handed to a record)
    float4 *vrec;                 // FT_DEFER: [2 i] position, [2 i + 1] vlast as of the launch's
                                  // save step, for its record
    const int32_t *id;            // original particle index
    int64_t n;                    // particles in this launch (prefix of the state arrays)
    const int32_t *n_dev;         // if set: live prefix length on the device (<= n)
    const int32_t *life;          // if set: steps each slot may run (batched sets of uneven lifetime)
    const int32_t *birth;         // if set: first step each slot runs (served requests joining mid-window)
    int32_t grid_stride;          // 1: persistent grid striding over the live prefix
    int64_t n_state;              // stride of volc / cmpc
    int64_t n_total;              // original particle count (history / constants stride)
    // history, record-major: one row of n_total particles per record, so the rows a launch
    // writes are whole in L2 before they reach DRAM (the fetch transposes them)
    float *hpos;                  // [(rec * n_total + id) * dim + d]
    float *hcurv;                 // [crec * n_total + id]
    float *hvol;                  // [(k * Li + irec) * n_total + id]
    float *hcmp;                  // [(e * Li + irec) * n_total + id]
    int64_t L, Lc, Li;
    // schedule
    const StepEntry *sched;
    int32_t s0, s1;
    // options (runtime-uniform)
    float h, hh, sixth, max_length, sphere_radius;
    float inv_2h, inv_hh;         // 1 / (2 h) and 1 / (h h), rounded to float (curvature differences)
    int32_t wind_dynamic, dyn_any, border_mode, curvature_mode, abort_mode, uplift_mode;
    int32_t constants_mode, volume_mode, reverse, sphere, topography, compensated;
    int32_t nvol, ncon, nexpr;
    int32_t filter_weights;       // 1: interpolation fractions rounded to the nearest 1/256
    const Program *prog;          // [4]
    unsigned long long *counters; // [0] particle-steps
    unsigned *alive_at;           // if set: [step - s0][32 shards] particles alive after each step
};

// ------------------------------------------------------------------ helpers

__device__ __forceinline__ float lerp_(float a, float b, float t) { return __fmaf_rn(t, b - a, a); }

// Paired float32 operations (one instruction for two values); each half rounds like the scalar
// operation.  a - b is formed as fma(b, -1, a): the product is exact, so it rounds like the
// subtraction.
__device__ __forceinline__ float2 both(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

// Texture coordinate -> cell index and fraction.  Coordinates are clamped to [-2, n+1]
// first; every corner outside the grid is border (3D) or clamped (2D), so the clamp never
// changes a value and keeps the integer conversion in range.
// fw = 1 rounds the fraction to the nearest 1/256, the 8-bit weights of the texture unit the
// reference filters with (CUDA Programming Guide, linear filtering); 0 keeps it exact.
__device__ __forceinline__ void cell(float a, int n, int fw, int &i, float &f) {
    a = fminf(fmaxf(a, -2.0f), (float)(n + 1));
    const float fl = floorf(a);
    i = (int)fl;
    f = a - fl;
    if (fw) f = floorf(f * 256.0f + 0.5f) * (1.0f / 256.0f);
}

template <typename H> __device__ __forceinline__ float2 cvt16(unsigned q) {
    if constexpr (std::is_same<H, __half>::value)
        return __half22float2(*reinterpret_cast<const __half2 *>(&q));
    else
        return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&q));
}

// Ring nodes, (u, v) and w of one snapshot: 16-bit types, and float32 below.
template <typename H> struct Store {
    static __device__ __forceinline__ void load3(const void *node, float2 &uv, float &w) {
        const uint2 q = __ldg(reinterpret_cast<const uint2 *>(node));
        uv = cvt16<H>(q.x); w = cvt16<H>(q.y).x;
    }
    static __device__ __forceinline__ float2 load2(const void *node) { return cvt16<H>(__ldg(reinterpret_cast<const unsigned *>(node))); }
    static constexpr int bytes3 = 8, bytes2 = 4;
};

template <> struct Store<float> {
    // 3D node {u, v, w, 0}
    static __device__ __forceinline__ void load3(const void *node, float2 &uv, float &w) {
        const float4 q = __ldg(reinterpret_cast<const float4 *>(node));
        uv = make_float2(q.x, q.y); w = q.z;
    }
    static __device__ __forceinline__ float2 load2(const void *node) { return __ldg(reinterpret_cast<const float2 *>(node)); }
    static constexpr int bytes3 = 16, bytes2 = 8;
};

// Window-pair layouts: node n holds the back snapshot's (u, v), the front snapshot's (u, v) and
// the two w: {u_b, v_b, u_f, v_f, w_b, w_f, 0, 0} in 3D (32 bytes float32, 16 bytes 16-bit),
// {u_b, v_b, u_f, v_f} in 2D (16 / 8 bytes).  One load returns both snapshots, as the operand pairs
// of sm_100's paired float32 instructions (__ffma2_rn): (u, v) of a snapshot is interpolated in space
// at once and (w_b, w_f) likewise, and the horizontal wind leaves the sample as a pair, so the time
// interpolation, the stage positions, the coordinates and the curvature differences are paired
// operations on (x, y) too.  Built per window from the ring (pack_kernels.cuh), with a border
// (clamped_cell, fill_padded, fill_edge2).
template <typename W> struct Pair {};

template <typename W> struct IsPair { static constexpr bool value = false; };
template <typename W> struct IsPair<Pair<W>> { static constexpr bool value = true; };

template <> struct Store<Pair<float>> {
    // 3D node: (u_b, v_b), (u_f, v_f), (w_b, w_f), one 256-bit load
    static __device__ __forceinline__ void load3p(const void *node, float2 (&c)[3]) {
        float r[8];
        asm volatile("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7])
                     : "l"(node));
        c[0] = make_float2(r[0], r[1]); c[1] = make_float2(r[2], r[3]); c[2] = make_float2(r[4], r[5]);
    }
    // 2D node: (u_b, v_b), (u_f, v_f)
    static __device__ __forceinline__ void load2p(const void *base, int32_t idx, float2 (&c)[2]) {
        const float4 q = __ldg(reinterpret_cast<const float4 *>(base) + idx);
        c[0] = make_float2(q.x, q.y); c[1] = make_float2(q.z, q.w);
    }
    static constexpr int bytes3 = 32, bytes2 = 16;
};

template <typename H> struct Store<Pair<H>> {
    static __device__ __forceinline__ void load3p(const void *node, float2 (&c)[3]) {
        const uint4 q = __ldg(reinterpret_cast<const uint4 *>(node));
        c[0] = cvt16<H>(q.x); c[1] = cvt16<H>(q.y); c[2] = cvt16<H>(q.z);
    }
    static __device__ __forceinline__ void load2p(const void *base, int32_t idx, float2 (&c)[2]) {
        const uint2 q = __ldg(reinterpret_cast<const uint2 *>(base) + idx);
        c[0] = cvt16<H>(q.x); c[1] = cvt16<H>(q.y);
    }
    static constexpr int bytes3 = 16, bytes2 = 8;
};

// Trilinear corner weights of one sample: indices and border validity.
struct Cell3 {
    int32_t base;        // node index of corner (ix, iy, iz), clamped into the grid (< 2^31 nodes)
    int32_t sx, sy, sz;  // strides to the +x / +y / +z corner (0 where that corner is clamped)
    float fx, fy, fz;
    unsigned valid;      // bit (dz*4 + dy*2 + dx): corner inside the grid
};

__device__ __forceinline__ Cell3 make_cell3(const KParams &P, float ax, float ay, float az) {
    int ix, iy, iz;
    Cell3 c;
    cell(ax, P.nx, P.filter_weights, ix, c.fx);
    cell(ay, P.ny, P.filter_weights, iy, c.fy);
    cell(az, P.nz, P.filter_weights, iz, c.fz);
    const bool x0 = (unsigned)ix < (unsigned)P.nx, x1 = (unsigned)(ix + 1) < (unsigned)P.nx;
    const bool y0 = (unsigned)iy < (unsigned)P.ny, y1 = (unsigned)(iy + 1) < (unsigned)P.ny;
    const bool z0 = (unsigned)iz < (unsigned)P.nz, z1 = (unsigned)(iz + 1) < (unsigned)P.nz;
    // bit k = dz*4 + dy*2 + dx: per axis, the corners on each side form a fixed bit pattern
    const unsigned X = (x0 ? 0x55u : 0u) | (x1 ? 0xAAu : 0u);
    const unsigned Y = (y0 ? 0x33u : 0u) | (y1 ? 0xCCu : 0u);
    const unsigned Z = (z0 ? 0x0Fu : 0u) | (z1 ? 0xF0u : 0u);
    c.valid = X & Y & Z;
    const int cx = min(max(ix, 0), P.nx - 1), cy = min(max(iy, 0), P.ny - 1), cz = min(max(iz, 0), P.nz - 1);
    c.base = (cz * P.ny + cy) * P.nx + cx;
    c.sx = (x0 && x1) ? 1 : 0;
    c.sy = (y0 && y1) ? P.nx : 0;
    c.sz = (z0 && z1) ? P.nx * P.ny : 0;
    return c;
}

// Nodes of the last cell a particle sampled.  Consecutive samples of one particle (its RK4 stages,
// its next step) mostly fall in the same cell, whose nodes then need no new gathers; the values and
// the arithmetic are the same either way.  The cell is identified by its
// node index or by its negated first corner (wind_at); 3D keeps 24 float
// pairs (48 registers; 16-bit nodes converted when loaded; AdvBounds gives the launch shape), 2D 8
// pairs (16 registers).
// Corner k + 1 of each x pair (k even) is kept as its difference from corner k, formed once when
// the cell is loaded: the x lerps of every later sample are then one paired FMA each, with the
// difference lerp2_ would form (same instruction, same rounding).
struct SampleCache {
    int32_t base;      // pairs in 3D and of Euler steps: padded node index of the first corner
    float2 nxy;        // else: minus the first corner; NaN: no cell, or one not to be kept
    float nz;
    float2 c2d[2][4];  // 2D: (u, v) of the back and of the front snapshot at corners 0, 2; differences 1 - 0, 3 - 2
    float2 c2[3][8];   // 3D: (u, v) back, (u, v) front, (w_b, w_f) at even corners, differences at odd ones
    __device__ __forceinline__ void reset() {
        base = (int32_t)0x80000000;   // no cell's index
        nz = __int_as_float(0x7fffffff);
        nxy = both(nz);
    }
};

// 2D window pair with replicated edges: padded node (x, y), x in [-1, nx + 1] and y in
// [-1, ny + 1], of a (nx + 3) x (ny + 3) buffer holds node (clamp(x), clamp(y)), so a coordinate
// clamped to [-1, n] reads the clamp-addressed corners of make_cell2 without index clamps.  Same
// values: inside [-1, n] cell, fraction and corners are unchanged; outside it both corners of the
// axis are the same edge node, interpolated with any fraction to that node's value exactly.
//
// 3D window pair with a zero border (one node below, two above the grid on every axis): the
// coordinate is clamped to [-1, n], so every corner of the footprint is a node of the padded
// buffer and needs no validity test.
// Same values as make_cell3 + border addressing: inside [-1, n] the cell and fraction are
// identical; outside it every corner the original reads is outside the grid (0), and here the
// fraction is 0 with the weighted-away corner finite, so the interpolation is +0 either way.
// Padded node count of a window-pair buffer: (nx + 3) (ny + 3) (nz + 3) in 3D, (nx + 3) (ny + 3)
// in 2D.
#ifndef __CUDACC_RTC__
inline int64_t padded_pair_nodes(int dim, int64_t nx, int64_t ny, int64_t nz) {
    return (nx + 3) * (ny + 3) * (dim == 3 ? nz + 3 : 1);
}
#endif

// Cell of a coordinate without the conversion unit.  For |a| < 2^22, a + 1.5 * 2^23 rounded toward
// -infinity lies in [2^23, 2^24), where the floats are the integers, so it is floor(a) + 1.5 * 2^23
// exactly, its bit pattern is PCELL_BITS + floor(a), and 1.5 * 2^23 minus it is -floor(a).  The sum is
// monotonic, so no coordinate outside that range (nor NaN) has the pattern of a cell in it.
constexpr uint32_t PCELL_BITS = 0x4B400000u;   // bit pattern of 1.5 * 2^23
constexpr float PCELL_MAGIC = 12582912.0f;     // 1.5 * 2^23
struct PCell {
    uint32_t bx, by, bz;     // PCELL_BITS + cell
    float2 nxy;              // minus the cell
    float nz;
};

template <int DIM>
__device__ __forceinline__ PCell make_pcell(float2 axy, float az) {
    PCell c;
    const float2 t = __fadd2_rd(axy, both(PCELL_MAGIC));
    c.bx = __float_as_uint(t.x);
    c.by = __float_as_uint(t.y);
    c.nxy = sub2(both(PCELL_MAGIC), t);
    c.bz = 0;
    c.nz = 0.f;
    if (DIM == 3) {
        const float tz = __fadd_rd(az, PCELL_MAGIC);
        c.bz = __float_as_uint(tz);
        c.nz = PCELL_MAGIC - tz;
    }
    return c;
}

// The same by the conversion unit, for grids of 2^22 nodes and more along an axis (a clamped).
__device__ __forceinline__ uint32_t pcell1_wide(float a, float &neg) {
    const float fl = floorf(a);
    neg = -fl;
    return PCELL_BITS + (uint32_t)(int)fl;
}

__device__ __forceinline__ float frac256(float f) { return floorf(f * 256.0f + 0.5f) * (1.0f / 256.0f); }

// lerp_ on a pair with one weight: each half equals lerp_ on that half bit for bit.
__device__ __forceinline__ float2 lerp2_(float2 a, float2 b, float t) { return fma2(both(t), sub2(b, a), a); }

// Trilinear interpolation of 8 corner pairs (odd entries: differences, SampleCache): x, then y,
// then z (the order of tri3).
__device__ __forceinline__ float2 tri8p(const float2 (&c)[8], float fx, float fy, float fz) {
    const float2 tx = both(fx);
    const float2 a00 = fma2(tx, c[1], c[0]), a10 = fma2(tx, c[3], c[2]);
    const float2 a01 = fma2(tx, c[5], c[4]), a11 = fma2(tx, c[7], c[6]);
    return lerp2_(lerp2_(a00, a10, fy), lerp2_(a01, a11, fy), fz);
}

// Index of a cell's first corner in the padded pair: (iz + 1) pnxy + (iy + 1) pnx + (ix + 1) in wrapping
// 32-bit arithmetic, with the patterns' offset removed by one loop-invariant term.
template <int DIM>
__device__ __forceinline__ int32_t padded_index(const KParams &P, const PCell &c) {
    const uint32_t sy = (uint32_t)P.pnx, sz = DIM == 3 ? (uint32_t)P.pnxy : 0u;
    return (int32_t)(c.bz * sz + c.by * sy + c.bx - (PCELL_BITS - 1u) * (sz + sy + 1u));
}

// Loads the 8 padded corners of the cell at `base` into the sample cache as 24 float pairs
// ((u, v) back and front, w per corner); 16-bit nodes are converted once here, not per sample.
template <typename H>
__device__ __forceinline__ void fill_padded(const KParams &P, const void *pairs, int32_t base, SampleCache &cc) {
    constexpr int64_t bytes = Store<Pair<H>>::bytes3;
    const char *row = reinterpret_cast<const char *>(pairs) + base * bytes;
    const int64_t sy = P.pnx * bytes, sz = P.pnxy * bytes;
#pragma unroll
    for (int k = 0; k < 8; k += 2) {
        const char *r = row + ((k & 2) ? sy : 0) + ((k & 4) ? sz : 0);
        float2 a[3], b[3];
        Store<Pair<H>>::load3p(r, a);
        Store<Pair<H>>::load3p(r + bytes, b);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            cc.c2[q][k] = a[q];
            cc.c2[q][k + 1] = sub2(b[q], a[q]);
        }
    }
}

// The four corners of a 2D cell from the window pair.
template <typename H>
__device__ __forceinline__ void fill_edge2(const KParams &P, const void *pairs, int32_t base, SampleCache &cc) {
    const int32_t idx[4] = {base, base + 1, base + P.pnx, base + P.pnx + 1};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        float2 c[2];
        Store<Pair<H>>::load2p(pairs, idx[k], c);
        cc.c2d[0][k] = (k & 1) ? sub2(c[0], cc.c2d[0][k - 1]) : c[0];
        cc.c2d[1][k] = (k & 1) ? sub2(c[1], cc.c2d[1][k - 1]) : c[1];
    }
}

// The corners of a cell straight from two ring slots (unpadded grids, both snapshots): corner
// indices are clamped into the grid, which is the 2D addressing; in 3D the corners outside are then
// set to zero (the border).  16 loads where the window pair needs 8, but no pass over the grid
// before the launch.  Against loading every sample's 16 nodes: gr_advance_noalloc, 500,001
// particles x 20 RK4 steps on 192 x 192 x 64 nodes 1.81 -> 0.49 ms, 1,000 particles x 10 steps
// 85 -> 67 us; the engine on ring slots, 1e6 particles x 300 steps, 28.3 -> 12.1 ms.
template <int DIM, typename T>
__device__ __forceinline__ void fill_ring(const KParams &P, const void *wb, const void *wf, const PCell &c, SampleCache &cc) {
    constexpr int bytes = DIM == 3 ? Store<T>::bytes3 : Store<T>::bytes2;
    const int ix = (int)(c.bx - PCELL_BITS), iy = (int)(c.by - PCELL_BITS), iz = DIM == 3 ? (int)(c.bz - PCELL_BITS) : 0;
    const int x0 = min(max(ix, 0), P.nx - 1), x1 = min(max(ix + 1, 0), P.nx - 1);
    const int y0 = min(max(iy, 0), P.ny - 1), y1 = min(max(iy + 1, 0), P.ny - 1);
    const int32_t dx = (x1 - x0) * bytes;
    if constexpr (DIM == 2) {
        const int32_t row[2] = {y0 * P.nx + x0, y1 * P.nx + x0};
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const char *b = reinterpret_cast<const char *>(wb) + (int64_t)row[r] * bytes;
            const char *f = reinterpret_cast<const char *>(wf) + (int64_t)row[r] * bytes;
            const float2 b0 = Store<T>::load2(b), b1 = Store<T>::load2(b + dx);
            const float2 f0 = Store<T>::load2(f), f1 = Store<T>::load2(f + dx);
            cc.c2d[0][2 * r] = b0; cc.c2d[0][2 * r + 1] = sub2(b1, b0);
            cc.c2d[1][2 * r] = f0; cc.c2d[1][2 * r + 1] = sub2(f1, f0);
        }
    } else {
        const int z0 = min(max(iz, 0), P.nz - 1), z1 = min(max(iz + 1, 0), P.nz - 1);
        const int32_t row[4] = {(z0 * P.ny + y0) * P.nx + x0, (z0 * P.ny + y1) * P.nx + x0,
                                (z1 * P.ny + y0) * P.nx + x0, (z1 * P.ny + y1) * P.nx + x0};
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const char *b = reinterpret_cast<const char *>(wb) + (int64_t)row[r] * bytes;
            const char *f = reinterpret_cast<const char *>(wf) + (int64_t)row[r] * bytes;
            Store<T>::load3(b, cc.c2[0][2 * r], cc.c2[2][2 * r].x);
            Store<T>::load3(b + dx, cc.c2[0][2 * r + 1], cc.c2[2][2 * r + 1].x);
            Store<T>::load3(f, cc.c2[1][2 * r], cc.c2[2][2 * r].y);
            Store<T>::load3(f + dx, cc.c2[1][2 * r + 1], cc.c2[2][2 * r + 1].y);
        }
        if ((unsigned)ix >= (unsigned)(P.nx - 1) || (unsigned)iy >= (unsigned)(P.ny - 1) ||
            (unsigned)iz >= (unsigned)(P.nz - 1)) {
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const bool in = (unsigned)(ix + (k & 1)) < (unsigned)P.nx &&
                                (unsigned)(iy + ((k >> 1) & 1)) < (unsigned)P.ny &&
                                (unsigned)(iz + (k >> 2)) < (unsigned)P.nz;
#pragma unroll
                for (int q = 0; q < 3; ++q)
                    if (!in) cc.c2[q][k] = make_float2(0.f, 0.f);
            }
        }
#pragma unroll
        for (int k = 0; k < 8; k += 2)
#pragma unroll
            for (int q = 0; q < 3; ++q) cc.c2[q][k + 1] = sub2(cc.c2[q][k + 1], cc.c2[q][k]);
    }
}

template <typename W> struct Elem { using type = W; };
template <typename H> struct Elem<Pair<H>> { using type = H; };

// Loads the corners of cell c into the sample cache: from the window pair wb, or from the ring
// slots wb and wf.
template <int DIM, typename W>
__device__ __forceinline__ void fill(const KParams &P, const void *wb, const void *wf, const PCell &c, SampleCache &cc) {
    using H = typename Elem<W>::type;
    if constexpr (!IsPair<W>::value) fill_ring<DIM, H>(P, wb, wf, c, cc);
    else if constexpr (DIM == 3) fill_padded<H>(P, wb, padded_index<3>(P, c), cc);
    else fill_edge2<H>(P, wb, padded_index<2>(P, c), cc);
}

// Horizontal components as a pair.
struct V3 {
    float2 xy;
    float z;
};

// Trilinear interpolation of one scalar float32 plane.
__device__ __forceinline__ float tri1(const float *plane, const Cell3 &c) {
    float s[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int dx = k & 1, dy = (k >> 1) & 1, dz = (k >> 2) & 1;
        const int32_t idx = c.base + (dx ? c.sx : 0) + (dy ? c.sy : 0) + (dz ? c.sz : 0);
        s[k] = (c.valid & (1u << k)) ? __ldg(plane + idx) : 0.f;
    }
    const float a00 = lerp_(s[0], s[1], c.fx), a10 = lerp_(s[2], s[3], c.fx);
    const float a01 = lerp_(s[4], s[5], c.fx), a11 = lerp_(s[6], s[7], c.fx);
    return lerp_(lerp_(a00, a10, c.fy), lerp_(a01, a11, c.fy), c.fz);
}

// Bilinear footprint with clamped indices (2D pitch textures sample as clamp).
struct Cell2 {
    int32_t i00, i10, i01, i11;
    float fx, fy;
};

__device__ __forceinline__ Cell2 make_cell2(int nx, int ny, int fw, float ax, float ay) {
    int ix, iy;
    Cell2 c;
    cell(ax, nx, fw, ix, c.fx);
    cell(ay, ny, fw, iy, c.fy);
    const int x0 = min(max(ix, 0), nx - 1), x1 = min(max(ix + 1, 0), nx - 1);
    const int y0 = min(max(iy, 0), ny - 1), y1 = min(max(iy + 1, 0), ny - 1);
    c.i00 = y0 * nx + x0;
    c.i10 = y0 * nx + x1;
    c.i01 = y1 * nx + x0;
    c.i11 = y1 * nx + x1;
    return c;
}

__device__ __forceinline__ float bil1(const float *plane, const Cell2 &c) {
    return lerp_(lerp_(__ldg(plane + c.i00), __ldg(plane + c.i10), c.fx),
                 lerp_(__ldg(plane + c.i01), __ldg(plane + c.i11), c.fx), c.fy);
}

__device__ __forceinline__ float dot3(const V3 &a, const V3 &b, int dim) {
    float s = a.xy.x * b.xy.x;
    s = __fmaf_rn(a.xy.y, b.xy.y, s);
    if (dim == 3) s = __fmaf_rn(a.z, b.z, s);
    return s;
}

// World position -> grid coordinates.
__device__ __forceinline__ float2 grid_xy(const KParams &P, float2 p) { return mul2(add2(p, P.noff2), P.inv2); }
__device__ __forceinline__ float grid_z(const KParams &P, float z) { return (z + P.noffz) * P.inv_scale[2]; }

// Loads the cell of a sample at grid coordinates (axy, az) outside the cached one; f, fz: its
// fractions.  A coordinate outside the grid's range is clamped here, and the cell is not kept: a
// neighbouring sample's fraction in it would be another one.
template <int DIM, typename W>
__device__ __forceinline__ void load_cell(const KParams &P, float2 axy, float az, bool wide, const void *wb,
                                          const void *wf, float2 &f, float &fz, SampleCache &cc) {
    PCell c = make_pcell<DIM>(axy, az);
    const uint32_t first = PCELL_BITS - (uint32_t)P.below, more = 2u * (uint32_t)P.below;   // n + more cells
    bool keep = true;
    if (wide || c.bx - first >= (uint32_t)P.nx + more || c.by - first >= (uint32_t)P.ny + more ||
        (DIM == 3 && c.bz - first >= (uint32_t)P.nz + more)) {
        const float2 a = axy;
        const float b = az;
        axy.x = fminf(fmaxf(axy.x, P.flo), P.fn[0]);
        axy.y = fminf(fmaxf(axy.y, P.flo), P.fn[1]);
        if (DIM == 3) az = fminf(fmaxf(az, P.flo), P.fn[2]);
        if (wide) {
            c.bx = pcell1_wide(axy.x, c.nxy.x);
            c.by = pcell1_wide(axy.y, c.nxy.y);
            if (DIM == 3) c.bz = pcell1_wide(az, c.nz);
        } else {
            c = make_pcell<DIM>(axy, az);
        }
        keep = a.x == axy.x && a.y == axy.y && (DIM == 2 || b == az);
    }
    f = add2(axy, c.nxy);
    if (DIM == 3) fz = az + c.nz;
    if (!keep) cc.reset();
    else cc.nxy = c.nxy, cc.nz = c.nz;
    fill<DIM, W>(P, wb, wf, c, cc);
}

// The cell and fractions of every sample, clamped, and its padded node index for a key.
template <int DIM>
__device__ __forceinline__ PCell clamped_cell(const KParams &P, float2 axy, float az, float2 &f, float &fz) {
    axy.x = fminf(fmaxf(axy.x, -1.0f), P.fn[0]);
    axy.y = fminf(fmaxf(axy.y, -1.0f), P.fn[1]);
    if (DIM == 3) az = fminf(fmaxf(az, -1.0f), P.fn[2]);
    const PCell c = make_pcell<DIM>(axy, az);
    f = add2(axy, c.nxy);
    if (DIM == 3) fz = az + c.nz;
    return c;
}

// Wind at world position p, time weight t: interpolate() of TrajectoryIntegrator.icc:42-110.  The
// cell's corners come from the sample cache, reloaded when the cell changes (wb: the window pair; or
// wb, wf: the ring slots), interpolated in space, then in time.
// 2D RK4 and ring slots: a sample lies in the cached cell when its coordinates minus the cell's first
// corner are in [0, 1), one unsigned comparison of the bits each; those differences are then its
// fractions (a - floor(a) bit for bit: the same subtraction), and nothing of the cell's search is
// left on the way of such a sample.  (A fraction that rounds to 1 loads the same cell again.)
// Other pairs: some lane of nearly every warp loads a cell at nearly every sample (of an Euler step the
// only one), so the search is on the warp's way in any case and goes before the test, where it
// costs no latency.  Measured, search
// first against differences first: 1e6 particles x 300 steps 7.03 / 7.16 ms of step launches, 300,000 x 200
// 2.30 / 2.33, 10,000 x 1024 Euler steps in 2D 0.46 / 0.47, 10,000 x 1024 RK4 steps in 2D 0.80 / 0.75, 2D
// sphere 150,000 x 200 0.75 / 0.72, bf16 ring slots 777,777 x 100 2.66 / 2.61 ms.
// FT: the step kernel's feature set; lean variants but FT_BORDER run with filter_weights off (kernel_features).
template <int DIM, bool RK4, typename W, int FT>
__device__ __forceinline__ V3 wind_at(const KParams &P, const V3 &p, float t, const void *wb, const void *wf,
                                      SampleCache &cc) {
    constexpr bool options = !(FT & FT_LEAN) || (FT & FT_BORDER);
    const float2 axy = grid_xy(P, p.xy);
    const float az = DIM == 3 ? grid_z(P, p.z) : 0.f;
    float2 fr;
    float fz = 0.f;
    if constexpr (IsPair<W>::value && (DIM == 3 || !RK4)) {
        const PCell c = clamped_cell<DIM>(P, axy, az, fr, fz);
        const int32_t base = padded_index<DIM>(P, c);
        if (base != cc.base) {
            cc.base = base;
            fill<DIM, W>(P, wb, wf, c, cc);
        }
    } else {
        fr = add2(axy, cc.nxy);
        if (DIM == 3) fz = az + cc.nz;
        constexpr uint32_t one = 0x3f800000u;
        if (__float_as_uint(fr.x) >= one || __float_as_uint(fr.y) >= one || (DIM == 3 && __float_as_uint(fz) >= one))
            load_cell<DIM, W>(P, axy, az, options && !IsPair<W>::value && P.wide, wb, wf, fr, fz, cc);
    }
    if (options && P.filter_weights) {
        fr = make_float2(frac256(fr.x), frac256(fr.y));
        fz = frac256(fz);
    }
    const bool dynamic = IsPair<W>::value || (FT & FT_LEAN) || P.wind_dynamic;
    if constexpr (DIM == 3) {
        const float2 b = tri8p(cc.c2[0], fr.x, fr.y, fz), f = tri8p(cc.c2[1], fr.x, fr.y, fz);
        const float2 w = tri8p(cc.c2[2], fr.x, fr.y, fz);
        return dynamic ? V3{lerp2_(b, f, t), lerp_(w.x, w.y, t)} : V3{b, w.x};
    } else {
        const float2 tx = both(fr.x);
        const float2 b = lerp2_(fma2(tx, cc.c2d[0][1], cc.c2d[0][0]), fma2(tx, cc.c2d[0][3], cc.c2d[0][2]), fr.y);
        const float2 f = lerp2_(fma2(tx, cc.c2d[1][1], cc.c2d[1][0]), fma2(tx, cc.c2d[1][3], cc.c2d[1][2]), fr.y);
        return V3{dynamic ? lerp2_(b, f, t) : b, 0.f};
    }
}

// sphere_coordinates (TrajectoryIntegrator.tpp:98-104).
__device__ __forceinline__ V3 sphere_(const KParams &P, float py, V3 v) {
    const float pi = 3.14159265358979323846f;
    return V3{{(v.xy.x * 180.f) / (P.sphere_radius * cosf(py * (pi * 2.f) / 360.f) * pi),
               (v.xy.y * 180.f) / (pi * P.sphere_radius)}, 0.f};
}

__device__ __forceinline__ float ref_at(const float (&ref)[19], int i) {
    switch (i) {
        case 0: return ref[0]; case 1: return ref[1]; case 2: return ref[2]; case 3: return ref[3];
        case 4: return ref[4]; case 5: return ref[5]; case 6: return ref[6]; case 7: return ref[7];
        case 8: return ref[8]; case 9: return ref[9]; case 10: return ref[10]; case 11: return ref[11];
        case 12: return ref[12]; case 13: return ref[13]; case 14: return ref[14]; case 15: return ref[15];
        case 16: return ref[16]; case 17: return ref[17]; default: return ref[18];
    }
}

// Expression programs in kernel parameter space (deferred_extras_kernel): read through the
// constant cache at a warp-uniform index, so the dispatch below branches on uniform values and
// no global load sits on the evaluation's critical path.  Programs longer in total than
// GR_EXPR_PARAM_CODE are read from global memory (KParams::prog) instead.
constexpr int GR_EXPR_PARAM_CODE = 512;
struct ExprSet {
    int32_t in_params;                 // 1: code[] holds the programs
    int32_t start[GR_MAX_EXPR], len[GR_MAX_EXPR];
    Instr code[GR_EXPR_PARAM_CODE];
};

// Program sources of eval_program: expression e's length and instruction k; eval(e, ref) is the
// value of expression e (the interpreter here, straight-line code in a run-time compiled JitCode).
struct GlobalCode {
    const Program *prog;
    __device__ __forceinline__ int len(int e) const { return prog[e].len; }
    __device__ __forceinline__ Instr at(int e, int k) const { return prog[e].code[k]; }
    __device__ __forceinline__ float eval(int e, const float (&ref)[19]) const;
};
struct ParamCode {
    const ExprSet &X;
    __device__ __forceinline__ int len(int e) const { return X.len[e]; }
    __device__ __forceinline__ Instr at(int e, int k) const { return X.code[X.start[e] + k]; }
    __device__ __forceinline__ float eval(int e, const float (&ref)[19]) const;
};

// Postfix evaluation with an 8-register rotating stack (s0 = top); the program is uniform
// across the grid, so every branch here is uniform.
template <typename Code>
__device__ __forceinline__ float eval_program(const Code &code, int e, const float (&ref)[19]) {
    float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f, s4 = 0.f, s5 = 0.f, s6 = 0.f, s7 = 0.f;
    const int len = code.len(e);
    for (int k = 0; k < len; ++k) {
        const Instr in = code.at(e, k);
        float r;
        bool binary = false, push = false;
        switch (in.op) {
            case OP_REF: r = ref_at(ref, in.arg); push = true; break;
            case OP_CONST: r = in.value; push = true; break;
            case OP_ADD: r = s1 + s0; binary = true; break;
            case OP_SUB: r = s1 - s0; binary = true; break;
            case OP_MUL: r = s1 * s0; binary = true; break;
            case OP_DIV: r = s1 / s0; binary = true; break;
            case OP_RSUB: r = s0 - s1; binary = true; break;
            case OP_RDIV: r = s0 / s1; binary = true; break;
            case OP_ATAN2: r = atan2f(s1, s0); binary = true; break;
            case OP_RATAN2: r = atan2f(s0, s1); binary = true; break;
            case OP_SQRT: r = sqrtf(s0); break;
            case OP_EXP: r = expf(s0); break;
            case OP_LOG: r = logf(s0); break;
            case OP_SIN: r = sinf(s0); break;
            case OP_COS: r = cosf(s0); break;
            case OP_TAN: r = tanf(s0); break;
            case OP_ASIN: r = asinf(s0); break;
            case OP_ACOS: r = acosf(s0); break;
            case OP_ATAN: r = atanf(s0); break;
            default: r = s0; break;
        }
        if (push) {
            s7 = s6; s6 = s5; s5 = s4; s4 = s3; s3 = s2; s2 = s1; s1 = s0; s0 = r;
        } else if (binary) {
            s0 = r; s1 = s2; s2 = s3; s3 = s4; s4 = s5; s5 = s6; s6 = s7;
        } else {
            s0 = r;
        }
    }
    return s0;
}

__device__ __forceinline__ float GlobalCode::eval(int e, const float (&ref)[19]) const { return eval_program(*this, e, ref); }
__device__ __forceinline__ float ParamCode::eval(int e, const float (&ref)[19]) const { return eval_program(*this, e, ref); }

// The run's volume / expression options as the code below reads them: the KParams fields, or
// compile-time constants in the run-time compiled deferred kernel (jit.cu defines
// GR_JIT_OPTIONS and GR_JIT_<field>), where the loops and branches a run does not use drop out.
#ifdef GR_JIT_OPTIONS
#define GR_OPT(P, name) (GR_JIT_##name)
#else
#define GR_OPT(P, name) ((P).name)
#endif

// Volume samples and expression values of a particle, evaluated from the inputs of its last
// alive step: position p (that step's new position), stage-averaged velocity vc, curvature cv
// and the step's time weight / ring slots (tpp:363-447).  The kernel calls this only when the
// values become observable (a record, the end of a launch), which gives the same values as
// evaluating after every alive step, as the reference does.
template <int DIM, typename Code>
__device__ __forceinline__ void eval_extras(const KParams &P, const Code &code, const StepEntry &E, int64_t pid,
                                            const V3 &p, const V3 &vc, float cv, float (&vol)[GR_MAX_VOL],
                                            float (&cmp)[GR_MAX_EXPR]) {
    const float t0 = GR_OPT(P, dyn_any) ? E.t0 : 0.f;
    if (GR_OPT(P, volume_mode) != 0 && GR_OPT(P, nvol) > 0) {
        const int vb = GR_OPT(P, volume_mode) == 2 ? E.slot_back : 0, vf = GR_OPT(P, volume_mode) == 2 ? E.slot_front : 0;
        const float ax = (p.xy.x - P.off[0]) * P.inv_scale[0];
        const float ay = (p.xy.y - P.off[1]) * P.inv_scale[1];
        if (DIM == 3) {
            const float az = (p.z - P.off[2]) * P.inv_scale[2];
            const Cell3 c = make_cell3(P, ax, ay, az);
#pragma unroll
            for (int k = 0; k < GR_MAX_VOL; ++k) {
                if (k < GR_OPT(P, nvol)) {
                    const float b = tri1(P.vol + ((int64_t)vb * GR_MAX_VOL + k) * P.vol_plane, c);
                    vol[k] = GR_OPT(P, volume_mode) == 2 ? lerp_(b, tri1(P.vol + ((int64_t)vf * GR_MAX_VOL + k) * P.vol_plane, c), t0)
                                                : b;
                }
            }
        } else {
            const Cell2 c = make_cell2(P.nx, P.ny, P.filter_weights, ax, ay);
#pragma unroll
            for (int k = 0; k < GR_MAX_VOL; ++k) {
                if (k < GR_OPT(P, nvol)) {
                    const float b = bil1(P.vol + ((int64_t)vb * GR_MAX_VOL + k) * P.vol_plane, c);
                    vol[k] = GR_OPT(P, volume_mode) == 2 ? lerp_(b, bil1(P.vol + ((int64_t)vf * GR_MAX_VOL + k) * P.vol_plane, c), t0)
                                                : b;
                }
            }
        }
    }
    if (GR_OPT(P, nexpr) > 0) {
        float ref[19];
        ref[0] = p.xy.x; ref[1] = p.xy.y; ref[2] = DIM == 3 ? p.z : 0.f;
        ref[3] = GR_OPT(P, curvature_mode) == 3 ? cv : 0.f;
#pragma unroll
        for (int k = 0; k < 8; ++k) ref[4 + k] = k < GR_OPT(P, nvol) ? vol[k] : 0.f;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            float c = 0.f;
            if (k < GR_OPT(P, ncon) && GR_OPT(P, constants_mode) != 0) {
                const int cb = GR_OPT(P, constants_mode) == 2 ? E.slot_back : 0;
                const float b = __ldg(P.cons + ((int64_t)cb * GR_MAX_CON + k) * P.n_total + pid);
                if (GR_OPT(P, constants_mode) == 2) {
                    const float f = __ldg(P.cons + ((int64_t)E.slot_front * GR_MAX_CON + k) * P.n_total + pid);
                    c = lerp_(b, f, t0);
                } else {
                    c = b;
                }
            }
            ref[12 + k] = c;
        }
        ref[16] = vc.xy.x; ref[17] = vc.xy.y; ref[18] = DIM == 3 ? vc.z : 0.f;
#pragma unroll
        for (int e = 0; e < GR_MAX_EXPR; ++e)
            if (e < GR_OPT(P, nexpr)) cmp[e] = code.eval(e, ref);
    }
}

// The volume / expression values of slot i kept in the state arrays between evaluations.  For
// an evaluation (`evaluating`) only what eval_extras reads but does not overwrite is loaded:
// volumes when no volume is sampled (their stored values enter the expressions).
__device__ __forceinline__ void load_extras(const KParams &P, int64_t i, bool evaluating, float (&vol)[GR_MAX_VOL],
                                            float (&cmp)[GR_MAX_EXPR]) {
    const bool vols = !evaluating || GR_OPT(P, volume_mode) == 0;
#pragma unroll
    for (int k = 0; k < GR_MAX_VOL; ++k) vol[k] = (k < GR_OPT(P, nvol) && vols) ? P.volc[k * P.n_state + i] : 0.f;
#pragma unroll
    for (int k = 0; k < GR_MAX_EXPR; ++k) cmp[k] = (k < GR_OPT(P, nexpr) && !evaluating) ? P.cmpc[k * P.n_state + i] : 0.f;
}

__device__ __forceinline__ void store_extras(const KParams &P, int64_t i, const float (&vol)[GR_MAX_VOL],
                                             const float (&cmp)[GR_MAX_EXPR]) {
#pragma unroll
    for (int k = 0; k < GR_MAX_VOL; ++k)
        if (k < GR_OPT(P, nvol)) P.volc[k * P.n_state + i] = vol[k];
#pragma unroll
    for (int k = 0; k < GR_MAX_EXPR; ++k)
        if (k < GR_OPT(P, nexpr)) P.cmpc[k * P.n_state + i] = cmp[k];
}

// ------------------------------------------------------------------ the step kernel

// Volume / expression values at a record or at the end of a launch (tpp:363-435): evaluated if
// an alive step has passed since the last evaluation (`dirty`, then kept in the state arrays),
// else the state arrays' values; written to the record's rows when irec >= 0.
template <int DIM, typename Code>
__device__ __forceinline__ void extras_at(const KParams &P, const Code &code, int64_t i, int64_t pid, bool dirty,
                                          int last_s, const V3 &p, const V3 &vc_last, float cv, int32_t irec) {
    float vol[GR_MAX_VOL], cmp[GR_MAX_EXPR];
    load_extras(P, i, dirty, vol, cmp);
    if (dirty) {
        eval_extras<DIM>(P, code, P.sched[last_s], pid, p, vc_last, cv, vol, cmp);
        store_extras(P, i, vol, cmp);
    }
    if (irec < 0) return;
    if (GR_OPT(P, volume_mode) != 0) {
#pragma unroll
        for (int k = 0; k < GR_MAX_VOL; ++k)
            if (k < GR_OPT(P, nvol)) P.hvol[((int64_t)k * P.Li + irec) * P.n_total + pid] = vol[k];
    }
#pragma unroll
    for (int e = 0; e < GR_MAX_EXPR; ++e)
        if (e < GR_OPT(P, nexpr)) P.hcmp[((int64_t)e * P.Li + irec) * P.n_total + pid] = cmp[e];
}

// extras_at for the step kernel's in-kernel evaluation (FT_EXTRAS).  Not inlined: it runs once
// per record, and its register peak (the expression stack, the volume samples) then stays out
// of the step loop's allocation; the caller's live registers are saved around the call.
template <int DIM>
__device__ __noinline__ void record_extras(const KParams &P, int64_t i, int64_t pid, bool dirty, int last_s,
                                           V3 p, V3 vc_last, float cv, int32_t irec) {
    extras_at<DIM>(P, GlobalCode{P.prog}, i, pid, dirty, last_s, p, vc_last, cv, irec);
}

// Volume / expression values after a FT_DEFER step launch (tpp:363-435), from the inputs of a
// slot's last moved step: its position (a particle keeps it once it stops), the stored
// velocity and that step's schedule entry.  Same values as the in-kernel evaluation.
//  - rec >= 0: the launch saved record rec (info record irec) at one step: every slot of the live
//    prefix writes the record's rows, evaluating first if it moved since its last evaluation
//    (inputs and position in vrec, as of the save step).
//  - rec < 0: slots with pending inputs (vlast) are evaluated into the state arrays: all of them
//    (all = 1, the end of a run) or those about to retire (aborted, or lifetime over by k_end),
//    whose values are final.  (Folding this pass into the record kernel measured slower: the
//    second evaluation path doubles the kernel's code.)
template <int DIM, typename Code>
__device__ __forceinline__ void deferred_extras(const KParams &P, const Code &code, int32_t rec, int32_t irec,
                                                int32_t k_end, int32_t all) {
    const int64_t n = P.n_dev ? (int64_t)*P.n_dev : P.n;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        if (rec >= 0) {
            const int64_t pid = P.id[i];
            const float cv = GR_OPT(P, curvature_mode) == 3 ? P.curv[i] : 0.f;
            const float4 a = P.vrec[2 * i], v = P.vrec[2 * i + 1];
            const int32_t last_s = __float_as_int(v.w);
            extras_at<DIM>(P, code, i, pid, last_s >= 0, last_s < 0 ? 0 : last_s, V3{{a.x, a.y}, a.z},
                           V3{{v.x, v.y}, v.z}, cv, irec);
        } else {
            if (!all && P.status[i] == 0 && !(P.life && P.life[i] <= k_end)) continue;
            const float4 v = P.vlast[i];
            const int32_t last_s = __float_as_int(v.w);
            if (last_s < 0) continue;
            const int64_t pid = P.id[i];
            const float cv = GR_OPT(P, curvature_mode) == 3 ? P.curv[i] : 0.f;
            const V3 p{{P.px[i], P.py[i]}, DIM == 3 ? P.pz[i] : 0.f};
            extras_at<DIM>(P, code, i, pid, true, last_s, p, V3{{v.x, v.y}, v.z}, cv, -1);
            reinterpret_cast<int32_t *>(P.vlast + i)[3] = -1;
        }
    }
}

template <int DIM>
__global__ void __launch_bounds__(256, 3) deferred_extras_kernel(const __grid_constant__ KParams P,
                                                              const __grid_constant__ ExprSet X, int32_t rec,
                                                              int32_t irec, int32_t k_end, int32_t all) {
    if (X.in_params)
        deferred_extras<DIM>(P, ParamCode{X}, rec, irec, k_end, all);
    else
        deferred_extras<DIM>(P, GlobalCode{P.prog}, rec, irec, k_end, all);
}

constexpr int GR_ADV_MIN_BLOCKS = 2, GR_F32_BLOCKS = 4, GR_LIGHT_BLOCKS = 5;   // AdvBounds

// Advances the particle in slot i through steps [s0, s1) (or until its lifetime ends).
template <int DIM, bool RK4, typename W, int FT>
// Slots and particle ids are below 2^31 (checked where seeds are set).
__device__ __forceinline__ void advance_particle(const KParams &P, const int32_t i, const int32_t n_live,
                                                 unsigned &steps_acc) {
    // options: runtime values in the generic variant; in a lean variant (FT_LEAN) the ones the
    // host checked are off, and curvature / extras are the variant's compile-time choice
    constexpr bool LEAN = (FT & FT_LEAN) != 0;
    const int curvature_mode = LEAN ? ((FT & FT_CURV) ? 1 : 0) : P.curvature_mode;
    const int abort_mode = LEAN ? 0 : P.abort_mode;
    const int uplift_mode = LEAN ? 0 : P.uplift_mode;
    const bool compensated = LEAN ? (FT & FT_COMP) != 0 : P.compensated != 0;
    const bool topography = LEAN ? false : P.topography != 0;
    const int border_mode = LEAN && !(FT & FT_BORDER) ? 0 : P.border_mode;
    unsigned *const alive_at = LEAN ? nullptr : P.alive_at;
    const bool valid = i < n_live;
    int32_t st = valid ? P.status[i] : 1;
    bool alive = st == 0;
    const int32_t pid = valid && P.id ? P.id[i] : 0;   // no ids: a launch without records

    const V3 zero{{0.f, 0.f}, 0.f};
    V3 p = zero, q = zero, comp = zero, ld = zero;
    float len = 0.f, tc = 0.f, cv = 0.f;

    const bool curv_prev = curvature_mode == 1 || curvature_mode == 3;
    float seg = 0.f;   // |p - q| (curvature's ds): carried from the step that formed it
    if (valid) {
        p.xy = make_float2(P.px[i], P.py[i]);
        if (DIM == 3) p.z = P.pz[i];
        if (curv_prev) {
            q.xy = make_float2(P.qx[i], P.qy[i]); if (DIM == 3) q.z = P.qz[i];
            const V3 a{sub2(p.xy, q.xy), p.z - q.z};
            seg = sqrtf(dot3(a, a, DIM));
        }
        if (compensated) { comp.xy = make_float2(P.kx[i], P.ky[i]); if (DIM == 3) comp.z = P.kz[i]; }
        if (curvature_mode == 2) { ld.xy = make_float2(P.lx[i], P.ly[i]); if (DIM == 3) ld.z = P.lz[i]; }
        if (abort_mode != 0) len = P.length[i];
        if (curvature_mode != 0) tc = P.tc[i];
        if (curvature_mode == 3) cv = P.curv[i];
    }
    const bool was_alive = alive;
    unsigned my_steps = 0;
    const int32_t life = (valid && P.life) ? P.life[i] : 0x7fffffff;   // steps this particle may run
    // first step it runs: the request server's, which takes positions only
    constexpr bool births = (FT & (FT_CURV | FT_EXTRAS | FT_COMP | FT_DEFER)) == 0;
    const int32_t birth = births && valid && P.birth ? P.birth[i] : 0;
    const bool extras = LEAN ? (FT & FT_EXTRAS) != 0 : ((P.volume_mode != 0 && P.nvol > 0) || P.nexpr > 0);
    V3 vc_last = zero;
    int last_s = P.s0;
    bool dirty = false;   // volumes / expressions not yet evaluated for the last alive step
    const int sph = (!LEAN || (FT & FT_BORDER)) && P.sphere && DIM == 2;

    SampleCache cc;
    cc.reset();
    int slot = -1;   // ring layouts: back slot of the cached cell
    // the step's time weights and flags; with registers to spare also its ring slots and record
    // indices (a load at the record of every Euler step of 10,000 particles in 2D: 0.56 ms instead of 0.48),
    // in the 3D pair variants those where they are used, so that no register holds them over the step
    constexpr bool whole = DIM == 2 || !IsPair<W>::value;
    // An entry is the first touch of its sector, an L2 latency that a step of one sample does not hide:
    // Euler steps in 2D read it a step ahead (step launches of 1,000 particles x 300 steps 153 -> 113 us,
    // 10,000 x 1024 with a record a step 485 -> 424, 100,000 x 300 196 -> 184).  With four samples a step
    // the registers cost more: 400,000 RK4 particles in 2D 877 -> 935 us, 3D pairs 6.84 -> 7.00 ms.
    constexpr bool ahead = DIM == 2 && !RK4;
    const int4 *words = reinterpret_cast<const int4 *>(P.sched + P.s0);
    int4 head = make_int4(0, 0, 0, 0), tail = head;   // tail: slot_back, slot_front, rec, crec
    int4 next_head = head, next_tail = head;
    if (ahead && P.s0 < P.s1) {
        next_head = __ldg(words);
        next_tail = __ldg(words + 1);
    }
    for (int s = P.s0; s < P.s1; ++s) {
        const StepEntry *const entry = P.sched + s;
        words = reinterpret_cast<const int4 *>(ahead ? P.sched + min(s + 1, P.s1 - 1) : entry);
        if (ahead) {
            head = next_head;
            tail = next_tail;
            next_head = __ldg(words);
            next_tail = __ldg(words + 1);
        } else {
            head = __ldg(words);
            if (whole) tail = __ldg(words + 1);
        }
        const struct {
            float t0, t1, t2;
            int flags;
        } E{__int_as_float(head.x), __int_as_float(head.y), __int_as_float(head.z), head.w};
        const int sb = !IsPair<W>::value && P.wind_dynamic ? tail.x : 0;
        const int sf = !IsPair<W>::value && P.wind_dynamic ? tail.y : 0;
        const void *wb = IsPair<W>::value ? P.pair : reinterpret_cast<const char *>(P.wind) + (int64_t)sb * P.wind_stride;
        const void *wf = reinterpret_cast<const char *>(P.wind) + (int64_t)sf * P.wind_stride;
        // the cached cell belongs to the window's two snapshots
        if (!IsPair<W>::value && sb != slot) {
            cc.reset();
            slot = sb;
        }
        if (alive && s < life && (!births || s >= birth)) {
            ++my_steps;
            const float t0 = P.dyn_any ? E.t0 : 0.f;

            // integrator (tpp:135-231)
            V3 v, vc;
            if (RK4) {
                // stage k samples at a with its time weight, and the sum ((k1 + 2 k2) + 2 k3) + k4
                // is accumulated in that order (wgt * k is exact, so the fused sum rounds like the
                // separate one).  Unrolled in the lean variants, where the weights and time
                // selects become constants: 30 launches of the 1e6-particle plain configuration
                // take 7.63 ms against 8.08 ms as one loop of four and 7.94 ms two by two.  The
                // generic variant's longer step stays ahead two by two (65,000 particles with
                // every option: 1.007 ms against 1.018 ms unrolled).
                V3 a = p, acc = zero, accc = zero;
                constexpr int kUnroll = LEAN ? 4 : 2;
#pragma unroll kUnroll
                for (int stage = 0; stage < 4; ++stage) {
                    const float tw = stage == 0 ? t0 : (stage == 3 ? E.t2 : E.t1);
                    const V3 kc = wind_at<DIM, RK4, W, FT>(P, a, tw, wb, wf, cc);
                    const V3 k = sph ? sphere_(P, a.xy.y, kc) : kc;
                    if (stage == 0) {
                        acc = k;
                        accc = kc;
                    } else {
                        const float wgt = stage == 3 ? 1.f : 2.f;
                        acc.xy = fma2(both(wgt), k.xy, acc.xy);
                        if (DIM == 3) acc.z = __fmaf_rn(wgt, k.z, acc.z);
                        if (sph) accc.xy = fma2(both(wgt), kc.xy, accc.xy);
                    }
                    a.xy = fma2(k.xy, stage < 2 ? P.hh2 : P.h2, p.xy);
                    if (DIM == 3) a.z = __fmaf_rn(k.z, stage < 2 ? P.hh : P.h, p.z);
                }
                v = V3{mul2(acc.xy, P.sixth2), DIM == 3 ? acc.z * P.sixth : 0.f};
                vc = sph ? V3{mul2(accc.xy, P.sixth2), 0.f} : v;
            } else {
                vc = wind_at<DIM, RK4, W, FT>(P, p, t0, wb, wf, cc);
                v = sph ? sphere_(P, p.xy.y, vc) : vc;
            }

            // displacement, reverse and uplift (tpp:233-250).  A reversed step subtracts the
            // negated displacement: without uplift that is the forward step, bit for bit, so the
            // lean variants leave the option out.
            const bool reverse = !LEAN && P.reverse;
            V3 dp{mul2(v.xy, P.h2), DIM == 3 ? v.z * P.h : 0.f};
            if (reverse) { dp.xy = make_float2(-dp.xy.x, -dp.xy.y); dp.z = -dp.z; }
            if (DIM == 3 && uplift_mode != 0) {
                const int lb = uplift_mode != 2 ? 0 : whole ? tail.x : __ldg(&entry->slot_back);
                const int lf = uplift_mode != 2 ? 0 : whole ? tail.y : __ldg(&entry->slot_front);
                const float *LB = P.lift + ((int64_t)lb * P.n_total + pid) * 3;
                const float *LF = P.lift + ((int64_t)lf * P.n_total + pid) * 3;
                if (uplift_mode == 1) {
                    dp.xy = add2(dp.xy, make_float2(LB[0], LB[1])); dp.z = dp.z + LB[2];
                } else {
                    dp.xy = add2(dp.xy, lerp2_(make_float2(LB[0], LB[1]), make_float2(LF[0], LF[1]), t0));
                    dp.z = dp.z + lerp_(LB[2], LF[2], t0);
                }
            }

            // length abort (tpp:252-280)
            int32_t abort = 0;
            if (abort_mode != 0) {
                const float dpl = sqrtf(dot3(dp, dp, DIM));
                const float nl = len + dpl;
                if (abort_mode == 2) {
                    if (nl > P.max_length) {
                        const float sc = (P.max_length - len) / dpl;
                        dp.xy = mul2(both(sc), dp.xy); dp.z = sc * dp.z;
                        len = P.max_length;
                        abort = 1;
                    } else {
                        len = nl;
                    }
                } else {
                    if (nl > P.max_length) abort = 1;
                    len = nl;
                }
            }

            // new position (tpp:282); Kahan-compensated in the precision form
            V3 np = zero;
            if (compensated) {
                const V3 sd = reverse ? V3{{-dp.xy.x, -dp.xy.y}, -dp.z} : dp;
                const float2 y = sub2(sd.xy, comp.xy);
                np.xy = add2(p.xy, y);
                comp.xy = sub2(sub2(np.xy, p.xy), y);
                if (DIM == 3) { const float yz = sd.z - comp.z; np.z = p.z + yz; comp.z = (np.z - p.z) - yz; }
            } else {
                np.xy = reverse ? sub2(p.xy, dp.xy) : add2(p.xy, dp.xy);
                if (DIM == 3) np.z = reverse ? p.z - dp.z : p.z + dp.z;
            }

            // border and abort checks (tpp:284-323, icc:7-20, tpp:13-96)
            if (abort == 0) {
                const float dp2 = dot3(dp, dp, DIM);
                const int bm = DIM == 3 ? 0 : border_mode;
                const float2 rel = add2(np.xy, P.noff2);   // np - off
                if (bm == 0) {
                    bool topo = false;
                    if (DIM == 3 && topography) {
                        const Cell2 c = make_cell2(P.nx, P.ny, P.filter_weights, np.xy.x / P.scale[0], np.xy.y / P.scale[1]);
                        topo = bil1(P.topo, c) > np.z;
                    }
                    if (topo) abort = 3;
                    else if (dp2 < 1e-9f) abort = 4;
                    else {
                        bool out = rel.x > P.dom[0] || rel.x < 0.f || rel.y > P.dom[1] || rel.y < 0.f;
                        if (DIM == 3) {
                            const float rz = np.z + P.noffz;
                            out = out || rz > P.dom[2] || rz < 0.f;
                        }
                        if (out) abort = 2;
                    }
                } else if (dp2 < 1e-9f) {
                    abort = 4;
                } else {
                    const float ox = P.off[0], oy = P.off[1], DX = P.dom[0], DY = P.dom[1];
                    if (bm == 1) {
                        np.xy.x = fmodf(rel.x + DX, DX) + ox;
                        if (rel.y > DY || rel.y < 0.f) abort = 2;
                    } else if (bm == 2) {
                        if (sph) {
                            if (rel.x > DX || rel.x < 0.f || rel.y > DY || rel.y < 0.f) abort = 2;
                        } else {
                            np.xy.y = fmodf(rel.y + DY, DY) + oy;
                            if (rel.x > DX || rel.x < 0.f) abort = 2;
                        }
                    } else {
                        if (sph) {
                            const float px_ = p.xy.x - ox, py_ = p.xy.y - oy;
                            if (rel.y < 0.f) {
                                const float tx = (-py_) / (rel.y - py_) * (rel.x - px_) + px_;
                                np.xy.y = -rel.y + oy;
                                np.xy.x = fmodf(DX + 180.0f - rel.x + 2.f * tx, DX) + ox;
                            } else if (rel.y >= DY) {
                                const float tx = (DY - py_) / (rel.y - py_) * (rel.x - px_) + px_;
                                np.xy.y = (rel.y - DY) + oy;
                                np.xy.x = fmodf(DX + 180.0f - rel.x + 2.f * tx, DX) + ox;
                            }
                        } else {
                            np.xy.y = fmodf(rel.y + DY, DY) + oy;
                        }
                        np.xy.x = fmodf(np.xy.x - ox + DX, DX) + ox;
                    }
                }
            }

            st = abort;
            if (abort == 2 || abort == 3 || abort == 4) {
                // old position kept, total curvature flagged (tpp:327-332)
                if (curvature_mode != 0) tc = -1.f;
                alive = false;
            } else {
                // curvature (tpp:335-361)
                if (curvature_mode == 2) {
                    const float inv = 1.0f / sqrtf(dot3(v, v, DIM));
                    const V3 u{mul2(v.xy, both(inv)), v.z * inv};
                    if (E.flags & SF_TIME_POS) {
                        const float k = acosf(dot3(ld, u, DIM));
                        if (!isnan(k)) tc += k;
                    }
                    ld = u;
                } else if (curv_prev) {
                    // |np - p|: this segment's length, the next step's |p - q|
                    const V3 b{sub2(np.xy, p.xy), np.z - p.z};
                    const float nseg = sqrtf(dot3(b, b, DIM));
                    if (E.flags & SF_TIME_POS) {
                        float k = 0.f;
                        if (DIM == 3) {
                            // central differences scaled by the float reciprocals of 2 h and h h
                            // (the reference divides, icc:151-154: within one rounding of these);
                            // the fused (q + np) - 2 p rounds like the separate one (2 p is exact)
                            const V3 d1{mul2(sub2(np.xy, q.xy), P.i2h2), (np.z - q.z) * P.inv_2h};
                            const V3 d2{mul2(fma2(p.xy, both(-2.f), add2(q.xy, np.xy)), P.ihh2),
                                        __fmaf_rn(-2.f, p.z, q.z + np.z) * P.inv_hh};
                            const V3 x{{d1.xy.y * d2.z - d1.z * d2.xy.y, d1.z * d2.xy.x - d1.xy.x * d2.z},
                                       d1.xy.x * d2.xy.y - d1.xy.y * d2.xy.x};
                            const float l = sqrtf(dot3(d1, d1, 3));
                            k = fabsf(sqrtf(dot3(x, x, 3)) / (l * l * l));
                        }
                        const float ds = 0.5f * (seg + nseg);
                        if (curvature_mode == 3) cv = k;
                        if (!isnan(k)) tc += k * ds;
                    }
                    seg = nseg;
                }

                // volumes and expressions are evaluated lazily (eval_extras), or after the launch
                // from the stored inputs (FT_DEFER, deferred_extras_kernel)
                if constexpr ((FT & FT_DEFER) != 0)
                    P.vlast[i] = make_float4(vc.xy.x, vc.xy.y, DIM == 3 ? vc.z : 0.f, __int_as_float(s));
                vc_last = vc;
                last_s = s;
                dirty = true;

                q = p;
                p = np;
                if (abort != 0) alive = false;
            }
        }

        if (valid && (E.flags & SF_SAVE)) {
            float *hp = P.hpos + ((int64_t)(whole ? tail.z : __ldg(&entry->rec)) * P.n_total + pid) * DIM;
            hp[0] = p.xy.x; hp[1] = p.xy.y;
            if (DIM == 3) hp[2] = p.z;
            if (curvature_mode == 3 && (E.flags & SF_CURV_REC)) P.hcurv[(int64_t)(whole ? tail.w : __ldg(&entry->crec)) * P.n_total + pid] = cv;
            if constexpr ((FT & FT_DEFER) != 0) {
                // the record's inputs: the position and the last moved step's (if any since the
                // last evaluation)
                const float4 v = P.vlast[i];
                P.vrec[2 * (int64_t)i] = make_float4(p.xy.x, p.xy.y, DIM == 3 ? p.z : 0.f, 0.f);
                P.vrec[2 * (int64_t)i + 1] = v;
                if (__float_as_int(v.w) >= 0) reinterpret_cast<int32_t *>(P.vlast + i)[3] = -1;
            }
            if (extras) {
                record_extras<DIM>(P, i, pid, dirty, last_s, p, vc_last, cv, __ldg(&entry->irec));
                dirty = false;
                // refill the sample cache for the next step's first sample (at p): the cached
                // nodes are then dead while the values above are evaluated, which frees their
                // registers there.  RK4 steps on ring slots drop the cell instead: a second copy of the 16
                // loads in the loop costs them more (a record every 5 steps, 50,000 particles x 143 steps,
                // refilled / dropped: a volume and an expression 0.97 / 0.86 ms, every option 1.05 / 0.99;
                // Euler steps, records every 20 and 30: every option 0.33 / 0.36, a volume 0.40 / 0.46).
                if constexpr (DIM == 3 && RK4 && !IsPair<W>::value) {
                    cc.reset();
                } else if constexpr (DIM == 3) {
                    float2 f;
                    float fz;
                    const float2 axy = grid_xy(P, p.xy);
                    const float az = grid_z(P, p.z);
                    if constexpr (IsPair<W>::value) {
                        const PCell c = clamped_cell<3>(P, axy, az, f, fz);
                        cc.base = padded_index<3>(P, c);
                        fill<3, W>(P, wb, wf, c, cc);
                    } else {
                        load_cell<3, W>(P, axy, az, !LEAN && P.wide, wb, wf, f, fz, cc);
                    }
                }
            }
        }

        // MinimumAliveParticles: particles alive after this step, one atomic per warp, spread
        // over 32 counters so that one address does not serialise the warps of the grid
        if (alive_at) {
            const unsigned m = __ballot_sync(0xffffffffu, valid && alive);
            if ((threadIdx.x & 31) == 0 && m)
                atomicAdd(alive_at + (int64_t)(s - P.s0) * 32 + (blockIdx.x & 31), (unsigned)__popc(m));
        }
    }

    if (valid && was_alive) {
        if (extras && dirty) record_extras<DIM>(P, i, pid, true, last_s, p, vc_last, cv, -1);
        P.status[i] = st;
        P.px[i] = p.xy.x; P.py[i] = p.xy.y;
        if (DIM == 3) P.pz[i] = p.z;
        if (curv_prev) { P.qx[i] = q.xy.x; P.qy[i] = q.xy.y; if (DIM == 3) P.qz[i] = q.z; }
        if (compensated) { P.kx[i] = comp.xy.x; P.ky[i] = comp.xy.y; if (DIM == 3) P.kz[i] = comp.z; }
        if (curvature_mode == 2) { P.lx[i] = ld.xy.x; P.ly[i] = ld.xy.y; if (DIM == 3) P.lz[i] = ld.z; }
        if (abort_mode != 0) P.length[i] = len;
        if (curvature_mode != 0) P.tc[i] = tc;
        if (curvature_mode == 3) P.curv[i] = cv;
    }

    steps_acc += my_steps;
}

// One thread per particle, or (P.grid_stride) a persistent grid striding over the live
// prefix, whose size is read on the device: the launch shape then stays fixed while the live
// count shrinks, as a captured CUDA graph needs.
// Launch bounds: 256 threads, 2 blocks per SM (128 registers).  The float32 3D kernels keep 48
// cached floats in 128-thread blocks: 4 per SM (128 registers) in the generic variant and the lean
// ones with volume / expression values or with both Kahan positions and curvature, 5 per SM (96
// registers, 20 warps) in the other lean ones on window pairs, whose state fits there, but for 24 bytes of
// spill stores and 12 of loads in the RK4 variants with total curvature (0.65e6 of the 142e6 warp
// instructions of a 10-step launch of 1e6 particles); the extra warps hide more of the sampling and
// curvature latency.  Ring slots stay at 4 blocks: with 16
// loads in flight 96 registers spill in the step loop (gr_advance_noalloc, 500,001 particles x 20
// steps, 0.49 ms against 0.44).  16-bit 3D kernels: 128 x 5 for the lean variants
// with curvature or deferred values (measured 5-6% faster than 256 x 2 on the 3D benchmark
// configuration), 256 x 2 for the rest (the positions-only variant of the batching and serving forms
// measured 2% slower at 128 x 5).
template <int DIM, typename W, int FT> struct AdvBounds {
    static constexpr bool f32 = std::is_same<typename Elem<W>::type, float>::value;
    static constexpr bool light = (FT & FT_LEAN) != 0 && (FT & FT_EXTRAS) == 0 &&
                                  (FT & (FT_COMP | FT_CURV)) != (FT_COMP | FT_CURV) &&
                                  (f32 || (FT & (FT_CURV | FT_DEFER)) != 0);
    static constexpr bool small = DIM == 3 && (f32 || light);   // 128-thread blocks
    static constexpr int threads = small ? 128 : 256;
    static constexpr int blocks = !small ? GR_ADV_MIN_BLOCKS : light && IsPair<W>::value ? GR_LIGHT_BLOCKS : GR_F32_BLOCKS;
};

template <int DIM, bool RK4, typename W, int FT>
__global__ void __launch_bounds__(AdvBounds<DIM, W, FT>::threads, AdvBounds<DIM, W, FT>::blocks)
    advance_kernel(const __grid_constant__ KParams P) {
    const int32_t n_live = P.n_dev ? *P.n_dev : (int32_t)P.n;
    unsigned steps = 0;   // of this thread
    if (P.grid_stride) {
        const int64_t stride = (int64_t)gridDim.x * blockDim.x;
        for (int64_t base = (int64_t)blockIdx.x * blockDim.x; base < n_live; base += stride)
            advance_particle<DIM, RK4, W, FT>(P, (int32_t)(base + threadIdx.x), n_live, steps);
    } else {
        advance_particle<DIM, RK4, W, FT>(P, (int32_t)(blockIdx.x * blockDim.x + threadIdx.x), n_live, steps);
    }
    // particle-steps, warp-aggregated (a block may be less than a warp)
    const unsigned lanes = __activemask();
    const unsigned warp_steps = __reduce_add_sync(lanes, steps);
    if ((int)(threadIdx.x & 31) == __ffs(lanes) - 1 && warp_steps) atomicAdd(P.counters, (unsigned long long)warp_steps);
}

}  // namespace granite_b200
