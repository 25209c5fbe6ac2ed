// advance.h — the step-kernel variants, instantiated per wind storage type in advance.cu
// (compiled once per type so the variants build in parallel).
#pragma once

#include "granite_kernels.cuh"

namespace granite_b200 {

using AdvanceFn = void (*)(const KParams);

// The feature set (FT_* in granite_kernels.cuh) a launch with parameters P may use: a lean
// variant when every option it leaves out is off in P, else generic.
// defer: the caller runs deferred_extras_kernel after every launch, which ends at each record.
inline int kernel_features(const KParams &P, bool defer = false) {
    if (P.uplift_mode != 0 || P.abort_mode != 0 || P.topography || P.alive_at != nullptr || !P.wind_dynamic ||
        (P.curvature_mode != 0 && P.curvature_mode != 1))
        return FT_GENERIC;
    const bool extras = (P.volume_mode != 0 && P.nvol > 0) || P.nexpr > 0;
    if (P.sphere || P.border_mode != 0 || P.filter_weights || P.wide)
        return extras || P.compensated || P.curvature_mode != 0 ? FT_GENERIC : (FT_LEAN | FT_BORDER);
    if (P.compensated) return extras ? FT_GENERIC : (FT_LEAN | FT_COMP | (P.curvature_mode == 1 ? FT_CURV : 0));
    return FT_LEAN | (P.curvature_mode == 1 ? FT_CURV : 0) | (extras ? (defer ? FT_DEFER : FT_EXTRAS) : 0);
}

// Where samples of a grid are clamped to (KParams::flo, fn): every corner of the cell beyond is
// outside the grid.  Window pairs carry one border node below and two above, so their cells are
// clamped to [-1, n]; 3D ring slots read as such to [-2, n + 1].  Both give the border's zeros; they
// differ where a sample lies a cell outside beside an edge node that is not finite, which [-1, n]
// multiplies by a weight of zero.
inline void clamp_cells(KParams &P, bool as_pair) {
    const bool one = as_pair || P.dim == 2;
    P.flo = one ? -1.f : -2.f;
    P.below = one ? 1 : 2;
    const int32_t n[3] = {P.nx, P.ny, P.nz};
    for (int d = 0; d < 3; ++d) P.fn[d] = one ? (float)n[d] : (float)(n[d] + 1);
}

// The step constants of a time step h and the operand pairs of the paired instructions, from off and
// inv_scale.
inline void derive_params(KParams &P, float h) {
    auto both = [](float a) { return make_float2(a, a); };
    P.h = h;
    P.hh = 0.5f * h;
    P.sixth = 1.0f / 6;
    P.inv_2h = 1.0f / (2.0f * h);
    P.inv_hh = 1.0f / (h * h);
    P.h2 = both(P.h);
    P.hh2 = both(P.hh);
    P.sixth2 = both(P.sixth);
    P.i2h2 = both(P.inv_2h);
    P.ihh2 = both(P.inv_hh);
    P.noff2 = make_float2(-P.off[0], -P.off[1]);
    P.noffz = -P.off[2];
    P.inv2 = make_float2(P.inv_scale[0], P.inv_scale[1]);
}

// Grids that the fast cell arithmetic does not cover (make_pcell needs coordinates below 2^22).
inline bool wide_grid(int64_t nx, int64_t ny, int64_t nz) {
    return nx >= (1 << 22) - 2 || ny >= (1 << 22) - 2 || nz >= (1 << 22) - 2;
}

// Threads per block of a launch over few particles: blocks of 4, 8 or 16 threads, each a warp of its
// own, or 0 for whole warps.  A warp waits for a cell whenever one of its lanes changes cells, at 32
// lanes nearly every sample, so with schedulers idle fewer lanes a warp are faster: 100 RK4 steps of 1,000
// particles 0.21 -> 0.15 ms at 4 lanes, 4,097 0.26 -> 0.20 at 8 (0.20 at 4, but 1.01 against 0.85 with
// volumes and expressions over 240 steps), 10,000 0.34 -> 0.28 at 8, 20,000 0.32 -> 0.31 at 16.  The line
// lies where the warps would come in a second wave (16 an SM; 20,000 at 8 lanes: 0.48 ms) with some room.
inline int block_of_few(int64_t n) {
    constexpr int64_t sms = 148;
    if (n <= 4 * 4 * sms) return 4;
    if (n <= 8 * 9 * sms) return 8;
    if (n <= 16 * 9 * sms) return 16;
    return 0;
}

// Step kernel for a dimension, integrator, wind layout (pair = window-pair buffer) and feature
// set (kernel_features).
AdvanceFn advance_f32(int dim, bool rk4, bool pair, int ft);
AdvanceFn advance_bf16(int dim, bool rk4, bool pair, int ft);
AdvanceFn advance_f16(int dim, bool rk4, bool pair, int ft);

}  // namespace granite_b200
