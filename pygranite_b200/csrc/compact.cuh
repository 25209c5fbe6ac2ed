// compact.cuh — retirement of aborted particles and spatial re-sorting of the live ones.
//
// Between launches the live particles are counting-sorted by the Morton rank of the grid
// brick they sit in (4x4x2 nodes in 3D, 4x4 in 2D), so a warp samples neighbouring cells
// and the gathers of one warp share cache lines.  Aborted particles go to a separate
// retired store and are never launched again; the records they would have written later
// repeat their frozen state, substituted when the history is read (RowFill, engine.cu).  Per-particle arithmetic does
// not depend on the order, so results stay bit-identical.
//
// Kernels are static: every translation unit that includes this header owns its instances.
//
// One pass is three launches: bin (key + warp-aggregated histogram), scan (offsets of the bins within
// chunks) and move (the destination of every slot by a warp-aggregated ticket, its state written
// there; the last block commits the counts).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "granite_kernels.cuh"
#include "host_util.h"

namespace granite_b200 {

constexpr int SCAN_THREADS = 1024, SCAN_CHUNK = 4 * SCAN_THREADS;   // bins per block of the scan
constexpr int MAX_BINS = 1 << 20;                                    // bricks of a grid
constexpr int MAX_CHUNKS = MAX_BINS / SCAN_CHUNK + 1;

struct StateView {
    float *px, *py, *pz, *qx, *qy, *qz, *kx, *ky, *kz, *lx, *ly, *lz;
    float *length, *tc, *curv, *volc, *cmpc;
    float4 *vlast;    // deferred volume / expression inputs (KParams::vlast), or null
    int32_t *status, *id, *retire, *life, *birth;
    int64_t stride;   // per-array stride of volc / cmpc
};

struct CompactParams {
    StateView src, dst, ret;
    int32_t *key;              // bin of each active slot
    int32_t *hist;             // counters of nbins + 1 bins (whole chunks), zero between passes
    int32_t *cursor;           // next free place of each bin, within its chunk
    int32_t *chunk;            // per-chunk sums
    int32_t *ticket;           // blocks of the move done, zero between passes
    const int32_t *bintab;     // brick linear index -> Morton rank
    int32_t *n_act;            // active count (device)
    int32_t *n_new;            // live count after the pass (device)
    int32_t *n_ret;            // retired count (device)
    float off[3], inv_scale[3];
    int32_t nx, ny, nz, dim;
    int32_t bx, by, bz, nbx, nby, nbz, nbins;
    int32_t nvol, nexpr, curv_prev, compensated, fast_curv, abort_on, curv_on, curv_ind;
    int32_t rec_now;           // first record index not yet written
    int32_t k_end;             // steps run so far: a particle whose lifetime is over retires
    int32_t ret_by_id;         // 1: retired particles go to slot id of `ret` (final state only)
};

__device__ __forceinline__ int32_t bin_of(const CompactParams &C, int64_t i) {
    // retired bin (last): aborted, or its lifetime is over (status stays Time)
    if (C.src.status[i] != 0 || (C.src.life && C.src.life[i] <= C.k_end)) return C.nbins;
    const float ax = (C.src.px[i] - C.off[0]) * C.inv_scale[0];
    const float ay = (C.src.py[i] - C.off[1]) * C.inv_scale[1];
    const int ix = (int)fminf(fmaxf(floorf(ax), 0.f), (float)(C.nx - 1));
    const int iy = (int)fminf(fmaxf(floorf(ay), 0.f), (float)(C.ny - 1));
    int iz = 0;
    if (C.dim == 3) {
        const float az = (C.src.pz[i] - C.off[2]) * C.inv_scale[2];
        iz = (int)fminf(fmaxf(floorf(az), 0.f), (float)(C.nz - 1));
    }
    return C.bintab[((iz / C.bz) * C.nby + iy / C.by) * C.nbx + ix / C.bx];
}

// key + histogram (zero when the pass begins); lanes of a warp with the same key add once (sorted input: mostly one key per warp)
static __global__ void bin_kernel(const __grid_constant__ CompactParams C) {
    const int64_t n = *C.n_act;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t base = (int64_t)blockIdx.x * blockDim.x; base < n; base += stride) {
        const int64_t i = base + threadIdx.x;
        const bool ok = i < n;
        const int32_t k = ok ? bin_of(C, i) : -1;
        if (ok) C.key[i] = k;
        const unsigned peers = __match_any_sync(0xffffffffu, k);
        const int leader = __ffs(peers) - 1;
        if (ok && (int)(threadIdx.x & 31) == leader) atomicAdd(C.hist + k, __popc(peers));
    }
}

// Exclusive scan of the counters inside chunks of SCAN_CHUNK bins, one block each; leaves the
// counters zero.  The chunk totals are scanned by every block of the move for itself (at most
// MAX_CHUNKS of them), which is shorter than a second level here.  The last bin holds the retiring
// slots, so its counter gives the live count.
static __global__ void __launch_bounds__(SCAN_THREADS) scan_kernel(const __grid_constant__ CompactParams C) {
    __shared__ int32_t warp_sum[SCAN_THREADS / 32];
    const int t = blockIdx.x * SCAN_THREADS + threadIdx.x;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int4 v = reinterpret_cast<const int4 *>(C.hist)[t];
    reinterpret_cast<int4 *>(C.hist)[t] = make_int4(0, 0, 0, 0);
    if (t == C.nbins / 4) {
        const int q = C.nbins & 3;
        *C.n_new = *C.n_act - (q == 0 ? v.x : q == 1 ? v.y : q == 2 ? v.z : v.w);
    }
    const int32_t own = v.x + v.y + v.z + v.w;
    int32_t x = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sum[wid] = x;
    __syncthreads();
    if (wid == 0) {
        int32_t s = warp_sum[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        warp_sum[lane] = s;   // inclusive over warps
    }
    __syncthreads();
    const int32_t before = x - own + (wid > 0 ? warp_sum[wid - 1] : 0);
    reinterpret_cast<int4 *>(C.cursor)[t] = make_int4(before, before + v.x, before + v.x + v.y, before + v.x + v.y + v.z);
    if (threadIdx.x == SCAN_THREADS - 1) C.chunk[blockIdx.x] = before + own;
}

__device__ __forceinline__ void move_live(const CompactParams &C, int64_t i, int64_t d) {
    const StateView &S = C.src, &D = C.dst;
    D.px[d] = S.px[i]; D.py[d] = S.py[i];
    if (C.dim == 3) D.pz[d] = S.pz[i];
    if (C.curv_prev) { D.qx[d] = S.qx[i]; D.qy[d] = S.qy[i]; if (C.dim == 3) D.qz[d] = S.qz[i]; }
    if (C.compensated) { D.kx[d] = S.kx[i]; D.ky[d] = S.ky[i]; if (C.dim == 3) D.kz[d] = S.kz[i]; }
    if (C.fast_curv) { D.lx[d] = S.lx[i]; D.ly[d] = S.ly[i]; if (C.dim == 3) D.lz[d] = S.lz[i]; }
    if (C.abort_on) D.length[d] = S.length[i];
    if (C.curv_on) D.tc[d] = S.tc[i];
    if (C.curv_ind) D.curv[d] = S.curv[i];
    for (int k = 0; k < C.nvol; ++k) D.volc[k * D.stride + d] = S.volc[k * S.stride + i];
    for (int k = 0; k < C.nexpr; ++k) D.cmpc[k * D.stride + d] = S.cmpc[k * S.stride + i];
    if (S.vlast) D.vlast[d] = S.vlast[i];
    D.status[d] = S.status[i];
    D.id[d] = S.id[i];
    if (S.life) D.life[d] = S.life[i];
    if (S.birth) D.birth[d] = S.birth[i];
}

__device__ __forceinline__ void move_retired(const CompactParams &C, int64_t i, int64_t r) {
    const StateView &S = C.src, &R = C.ret;
    if (C.ret_by_id) {   // final state straight into the result slot of the particle
        const int64_t id = S.id[i];
        R.px[id] = S.px[i]; R.py[id] = S.py[i];
        if (C.dim == 3) R.pz[id] = S.pz[i];
        R.status[id] = S.status[i];
        return;
    }
    R.px[r] = S.px[i]; R.py[r] = S.py[i];
    if (C.dim == 3) R.pz[r] = S.pz[i];
    if (C.abort_on) R.length[r] = S.length[i];
    if (C.curv_on) R.tc[r] = S.tc[i];
    if (C.curv_ind) R.curv[r] = S.curv[i];
    for (int k = 0; k < C.nvol; ++k) R.volc[k * R.stride + r] = S.volc[k * S.stride + i];
    for (int k = 0; k < C.nexpr; ++k) R.cmpc[k * R.stride + r] = S.cmpc[k * S.stride + i];
    R.status[r] = S.status[i];
    R.id[r] = S.id[i];
    R.retire[r] = C.rec_now;
}

// Destination of every slot, and its state moved there; the last block commits the counts.
static __global__ void move_kernel(const __grid_constant__ CompactParams C) {
    __shared__ int32_t chunk_base[MAX_CHUNKS];
    const int64_t n = *C.n_act, live = *C.n_new, retired = *C.n_ret;
    if (threadIdx.x < 32) {
        const int chunks = (C.nbins + SCAN_CHUNK) / SCAN_CHUNK, per = (chunks + 31) / 32;
        const int c0 = min(threadIdx.x * per, chunks), c1 = min(c0 + per, chunks);
        int32_t own = 0;
        for (int c = c0; c < c1; ++c) own += C.chunk[c];
        int32_t x = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if ((int)threadIdx.x >= o) x += y;
        }
        x -= own;
        for (int c = c0; c < c1; ++c) {
            chunk_base[c] = x;
            x += C.chunk[c];
        }
    }
    __syncthreads();
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t base = (int64_t)blockIdx.x * blockDim.x; base < n; base += stride) {
        const int64_t i = base + threadIdx.x;
        const bool ok = i < n;
        const int32_t k = ok ? C.key[i] : -1;
        const unsigned peers = __match_any_sync(0xffffffffu, k);
        const int lane = threadIdx.x & 31;
        const int leader = __ffs(peers) - 1;
        int32_t first = 0;
        if (ok && lane == leader) first = atomicAdd(C.cursor + k, __popc(peers));
        first = __shfl_sync(0xffffffffu, first, leader);
        if (ok) {
            const int64_t d = chunk_base[k / SCAN_CHUNK] + first + __popc(peers & ((1u << lane) - 1));
            if (d < live) move_live(C, i, d);
            else move_retired(C, i, retired + (d - live));
        }
    }
    // every block has read the counts by the time the last one is done
    __syncthreads();
    if (threadIdx.x == 0) {
        if (atomicAdd(C.ticket, 1) == (int32_t)gridDim.x - 1) {
            *C.ticket = 0;
            if (!C.ret_by_id) *C.n_ret = (int32_t)(retired + (n - live));
            *C.n_act = (int32_t)live;
        }
    }
}

// Enqueues a pass over at most `n` active slots.
static inline void launch_compaction(const CompactParams &C, int64_t n, cudaStream_t stream) {
    const int threads = 256;
    // grid-stride kernels over the device count: a few resident waves cover any count
    const int blocks = std::min(grid_for(n, threads), 148 * 16);
    bin_kernel<<<blocks, threads, 0, stream>>>(C);
    scan_kernel<<<(C.nbins + SCAN_CHUNK) / SCAN_CHUNK, SCAN_THREADS, 0, stream>>>(C);
    move_kernel<<<blocks, threads, 0, stream>>>(C);
}
constexpr int COMPACTION_LAUNCHES = 3;

// Morton ranks of a box of nbx x nby x nbz bricks (each below 1024): a brick's rank is the number of
// bricks with smaller codes, summed level by level over the octants before its own, each clipped to
// the box.  (Sorting the codes of 73,728 bricks on the host took 3 ms of every engine's first run.)
static __global__ void morton_rank_kernel(int32_t *rank, int32_t nbx, int32_t nby, int32_t nbz) {
    const int32_t lin = blockIdx.x * blockDim.x + threadIdx.x;
    if (lin >= nbx * nby * nbz) return;
    const int32_t x = lin % nbx, y = lin / nbx % nby, z = lin / nbx / nby;
    int32_t below = 0, cx = 0, cy = 0, cz = 0;   // (cx, cy, cz): corner of the octant descended into
    for (int b = 9; b >= 0; --b) {
        const int32_t size = 1 << b;
        const int own = (x >> b & 1) | (y >> b & 1) << 1 | (z >> b & 1) << 2;
        for (int o = 0; o < own; ++o) {
            const int32_t ox = cx + (o & 1) * size, oy = cy + (o >> 1 & 1) * size, oz = cz + (o >> 2) * size;
            below += max(min(size, nbx - ox), 0) * max(min(size, nby - oy), 0) * max(min(size, nbz - oz), 0);
        }
        cx += (x >> b & 1) * size;
        cy += (y >> b & 1) * size;
        cz += (z >> b & 1) * size;
    }
    rank[lin] = below;
}

// The bricks of a grid that compaction sorts by: 4 x 4 x 2 nodes (4 x 4 in 2D), larger where there
// would be more than MAX_BINS of them, and their Morton ranks.
struct Bricks {
    int bx = 4, by = 4, bz = 2, nbx = 0, nby = 0, nbz = 0, nbins = 0;
    DevBuf<int32_t> rank;
    // nbins (0: not built) is set once the ranks are on their way: after an error the next call builds again.
    cudaError_t build(int dim, int64_t nx, int64_t ny, int64_t nz, cudaStream_t stream) {
        nbins = 0;
        bx = 4; by = 4; bz = dim == 3 ? 2 : 1;
        for (;;) {
            nbx = (int)((nx + bx - 1) / bx);
            nby = (int)((ny + by - 1) / by);
            nbz = (int)((nz + bz - 1) / bz);
            if ((int64_t)nbx * nby * nbz <= MAX_BINS && nbx <= 1024 && nby <= 1024 && nbz <= 1024) break;
            bx *= 2; by *= 2; if (dim == 3) bz *= 2;
        }
        const int n = nbx * nby * nbz;
        cudaError_t e = rank.alloc((size_t)n);
        if (e != cudaSuccess) return e;
        morton_rank_kernel<<<(n + 255) / 256, 256, 0, stream>>>(rank.p, nbx, nby, nbz);
        e = cudaGetLastError();
        if (e == cudaSuccess) nbins = n;
        return e;
    }
    void set(CompactParams &C) const {
        C.bx = bx; C.by = by; C.bz = bz;
        C.nbx = nbx; C.nby = nby; C.nbz = nbz;
        C.nbins = nbins;
        C.bintab = rank.p;
    }
};

// Scratch of the passes: zeroed when it is allocated, left zero by every pass.
struct CompactScratch {
    DevBuf<int32_t> hist, cursor, chunk, ticket;
    bool ready = false;   // allocated and zeroed
    cudaError_t alloc(int nbins) {
        if (ready) return cudaSuccess;
        const size_t chunks = ((size_t)nbins + SCAN_CHUNK) / SCAN_CHUNK, nb = chunks * SCAN_CHUNK;
        cudaError_t e = hist.alloc(nb);
        if (e == cudaSuccess) e = cursor.alloc(nb);
        if (e == cudaSuccess) e = chunk.alloc(chunks);
        if (e == cudaSuccess) e = cudaMemset(hist.p, 0, nb * sizeof(int32_t));
        if (e == cudaSuccess) e = ticket.alloc(1);
        if (e == cudaSuccess) e = cudaMemset(ticket.p, 0, sizeof(int32_t));
        if (e == cudaSuccess) e = cudaStreamSynchronize(cudaStreamLegacy);   // the runs' streams do not wait for it
        ready = e == cudaSuccess;
        return e;
    }
    void set(CompactParams &C) const {
        C.hist = hist.p;
        C.cursor = cursor.p;
        C.chunk = chunk.p;
        C.ticket = ticket.p;
    }
};

}  // namespace granite_b200
