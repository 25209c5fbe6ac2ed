// noalloc.cu — gr_advance_noalloc: advancing particles without allocating device memory.
//
// Some callers cannot call cudaMalloc: plug-in hosts whose device memory belongs to their own
// pool allocator (a cudaMalloc there would go around the host's accounting and limits), and
// real-time loops that forbid allocation after start-up (an allocation may synchronise the
// device or take an unbounded time).  This entry point gives them the plain integrator (Euler
// or RK4 between two snapshots, the border checks and abort codes) on buffers they own.  Its
// only scratch, the per-step time weights and a counter, is the file-scope array below:
// every GPU that loads the library keeps these GR_NOALLOC_SCRATCH_BYTES until the process
// exits, and every call shares them.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <string>

#include "../../include/granite_b200.h"
#include "advance.h"

namespace granite_b200 {
void set_last_error(const char *msg);   // engine.cu
}

using namespace granite_b200;

namespace {

struct NoAllocScratch {
    StepEntry sched[GR_NOALLOC_MAX_STEPS];
    unsigned long long counters[2];   // [0] particle-steps, [1] unused (GR_NOALLOC_SCRATCH_BYTES counts it)
};

static_assert(sizeof(NoAllocScratch) == GR_NOALLOC_SCRATCH_BYTES, "scratch size stated in granite_b200.h");

static __device__ __align__(256) NoAllocScratch g_scratch;

constexpr int MAX_DEVICES = 64;
std::mutex g_mutex;
NoAllocScratch *g_scratch_ptr[MAX_DEVICES] = {};   // device address of g_scratch, per device

int err(int code, const char *msg) {
    set_last_error(msg);   // reported by gr_last_error()
    return code;
}

// Time weights of `steps` steps from time_start, with the float32 arithmetic of
// TrajectoryIntegrator.tpp:126-144 (the file is built with --fmad=false, so nothing is
// contracted).  The time accumulator T = T + h is a dependent chain: thread 0 walks it and
// parks each step's start time in t0; then the block turns the start times into the weights.
__global__ void __launch_bounds__(256) noalloc_schedule_kernel(NoAllocScratch *S, float time_back, float time_front,
                                                               float time_start, float h, int32_t steps) {
    if (threadIdx.x == 0) {
        float T = time_start;
        for (int k = 0; k < steps; ++k) {
            S->sched[k].t0 = T;
            T = T + h;
        }
        S->counters[0] = 0ull;   // it keeps the previous call's value: clear it
    }
    __syncthreads();
    for (int k = threadIdx.x; k < steps; k += blockDim.x) {
        StepEntry E{};
        const float T = S->sched[k].t0;
        E.t0 = (T - time_back) / (time_front - time_back);
        E.t1 = ((T + 0.5f * h) - time_back) / (time_front - time_back);
        E.t2 = ((T + h) - time_back) / (time_front - time_back);
        E.slot_back = 0;
        E.slot_front = 1;
        S->sched[k] = E;
    }
}

}  // namespace

extern "C" int gr_advance_noalloc(const gr_settings *s, int64_t nz, int64_t ny, int64_t nx, const void *wind_back,
                                  const void *wind_front, float time_back, float time_front, float time_start,
                                  int32_t steps, float *px, float *py, float *pz, int32_t *status, int64_t n,
                                  void *stream, int64_t *particle_steps) {
    if (!s || !wind_back || !wind_front || !px || !py || !status) return err(GR_ERR_USER, "ERROR < USER INPUT | null argument >");
    const int dim = s->space == 0 ? 3 : 2;
    if (dim == 3 && !pz) return err(GR_ERR_USER, "ERROR < USER INPUT | null argument >");
    if (steps < 0 || steps > GR_NOALLOC_MAX_STEPS)
        return err(GR_ERR_USER, "ERROR < USER INPUT | steps must be between 0 and GR_NOALLOC_MAX_STEPS (4096) >");
    if (n < 0 || n > 0x7fffffffLL) return err(GR_ERR_USER, "ERROR < USER INPUT | invalid particle count >");
    if (s->curvature_mode != 0 || s->volume_mode != 0 || s->constants_mode != 0 || (dim == 3 && s->uplift_mode != 0) ||
        s->abort_mode != 0 || s->storage != GR_STORE_F32 || s->compensated || s->windfield_mode != 1 ||
        s->time_mode != 0 || s->minimum_alive > 0)
        return err(GR_ERR_USER, "ERROR < USER INPUT | the allocation-free entry point runs the plain integrator only "
                                "(dynamic wind, float32 storage and time weights; no curvature, volumes, constants, "
                                "uplift, length abort or MinimumAliveParticles) >");
    if (!(s->delta_t > 0.f) || !(time_front > time_back))
        return err(GR_ERR_USER, "ERROR < USER INPUT | DeltaT must be positive and time_front > time_back >");
    if (!(time_start >= time_back) || !(time_start < time_front))
        return err(GR_ERR_USER, "ERROR < USER INPUT | time_start must lie in [time_back, time_front) >");
    if (nx < 1 || ny < 1 || (dim == 3 && nz < 1) || nx * ny * (dim == 3 ? nz : 1) > 0x7fffffffLL)
        return err(GR_ERR_USER, "ERROR < USER INPUT | invalid grid >");
    if (s->device < 0 || s->device >= MAX_DEVICES) return err(GR_ERR_USER, "ERROR < USER INPUT | invalid device >");

    std::lock_guard<std::mutex> lock(g_mutex);
    if (cudaSetDevice(s->device) != cudaSuccess) return err(GR_ERR_RUNTIME, "ERROR < RUNTIME | cudaSetDevice failed >");
    // once per device, with that device current: the device address of the scratch array
    if (!g_scratch_ptr[s->device]) {
        void *ptr = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&ptr, g_scratch);
        if (e != cudaSuccess || !ptr) return err(GR_ERR_RUNTIME, "ERROR < RUNTIME | cudaGetSymbolAddress failed >");
        g_scratch_ptr[s->device] = static_cast<NoAllocScratch *>(ptr);
    }
    NoAllocScratch *S = g_scratch_ptr[s->device];
    cudaStream_t st = static_cast<cudaStream_t>(stream);

    // the step schedule and the cleared counter, built on the device in stream order
    noalloc_schedule_kernel<<<1, 256, 0, st>>>(S, time_back, time_front, time_start, s->delta_t, steps);
    if (cudaGetLastError() != cudaSuccess) return err(GR_ERR_RUNTIME, "ERROR < RUNTIME | schedule launch failed >");
    const float h = s->delta_t;

    KParams P;
    std::memset(&P, 0, sizeof P);
    float scale[3];
    if (s->grid_scale_len == 1) { scale[0] = scale[1] = scale[2] = s->grid_scale[0]; }
    else if (s->grid_scale_len == 2) { scale[0] = s->grid_scale[0]; scale[1] = s->grid_scale[1]; scale[2] = s->grid_scale[0]; }
    else if (s->grid_scale_len == 3) { scale[0] = s->grid_scale[0]; scale[1] = s->grid_scale[1]; scale[2] = s->grid_scale[2]; }
    else return err(GR_ERR_USER, "ERROR < USER INPUT | Invalid GridScale dimension. >");
    float off[3];
    if (s->offset_len == 1) { off[0] = off[1] = off[2] = s->offset[0]; }
    else if (s->grid_scale_len == 2 && s->offset_len >= 2) { off[0] = s->offset[0]; off[1] = s->offset[1]; off[2] = s->offset[0]; }
    else if (s->grid_scale_len == 3 && s->offset_len >= 3) { off[0] = s->offset[0]; off[1] = s->offset[1]; off[2] = s->offset[2]; }
    else return err(GR_ERR_USER, "ERROR < USER INPUT | Invalid Offset dimension. >");
    const float g[3] = {(float)nx, (float)ny, (float)(dim == 3 ? nz : 0)};
    for (int d = 0; d < 3; ++d) {
        P.scale[d] = scale[d];
        P.inv_scale[d] = 1.0f / scale[d];
        P.off[d] = off[d];
        P.dom[d] = g[d] * scale[d];
    }
    P.nx = (int32_t)nx; P.ny = (int32_t)ny; P.nz = (int32_t)(dim == 3 ? nz : 1); P.dim = dim;
    const int64_t padded = (nx + 3) * (ny + 3) * (dim == 3 ? nz + 3 : 1);
    P.wide = wide_grid(nx, ny, dim == 3 ? nz : 1) || padded > 0x7fffffffLL;
    P.pnx = (int32_t)(nx + 3);
    P.pnxy = P.wide ? 0 : (int32_t)((nx + 3) * (ny + 3));
    clamp_cells(P, false);
    P.wind = wind_back;
    P.wind_stride = reinterpret_cast<const char *>(wind_front) - reinterpret_cast<const char *>(wind_back);
    P.px = px; P.py = py; P.pz = pz; P.status = status;
    P.n = n;
    P.sched = S->sched;
    P.counters = S->counters;
    P.s0 = 0;
    P.s1 = steps;
    derive_params(P, h);
    P.sphere_radius = s->sphere_radius;
    P.filter_weights = s->filter_weights ? 1 : 0;
    P.wind_dynamic = 1;
    P.dyn_any = 1;
    P.border_mode = dim == 2 ? s->border_mode : 0;
    P.reverse = s->reverse ? 1 : 0;
    P.sphere = dim == 2 && s->sphere_radius > 0.f;
    // the step kernel of the engine, reading the caller's two snapshots as ring slots, one thread per
    // particle
    const AdvanceFn fn = advance_f32(dim, s->integrator == 1, false, kernel_features(P));
    int threads = block_of_few(n);
    if (threads == 0)
        for (threads = 128; threads > 32 && (n + threads - 1) / threads < 2 * 148;) threads /= 2;
    const unsigned blocks = (unsigned)std::max<int64_t>(1, (n + threads - 1) / threads);
    fn<<<blocks, threads, 0, st>>>(P);
    if (cudaGetLastError() != cudaSuccess) return err(GR_ERR_RUNTIME, "ERROR < RUNTIME | launch failed >");
    if (particle_steps) {
        unsigned long long c = 0;
        if (cudaMemcpyAsync(&c, &S->counters[0], sizeof c, cudaMemcpyDeviceToHost, st) != cudaSuccess ||
            cudaStreamSynchronize(st) != cudaSuccess)
            return err(GR_ERR_RUNTIME, "ERROR < RUNTIME | reading the step counter failed >");
        *particle_steps = (int64_t)c;
    }
    return GR_OK;
}
