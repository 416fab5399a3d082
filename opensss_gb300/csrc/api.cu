// Error handling, version, and the batched ray tracer entry point.
#include <cstdarg>
#include <cstdio>
#include <cstring>

#include "common.cuh"
#include "trace.cuh"

static thread_local char g_err[1024] = "";

int sss_set_error(int code, const char* fmt, ...)
{
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
    return code;
}

int sss_check_launch(const char* what)
{
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        return sss_set_error(SSS_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
    return SSS_OK;
}

extern "C" const char* sss_last_error(void) { return g_err; }

extern "C" int sss_abi_version(void) { return SSS300_ABI_VERSION; }

extern "C" int sss_status_code(int32_t s)
{
    using namespace sss;
    s &= ~kNoteMapSigned;
    if (s == 0) return SSS_OK;
    if (s & kErrOverrun)
        return sss_set_error(SSS_ERR_OVERRUN,
                             "a ray traversal would pass Nx+Ny+Nz voxels (the reference raises "
                             "IndexError here)");
    if (s & kErrVoxel)
        return sss_set_error(SSS_ERR_VOXEL, "a linear voxel index fell outside the volume");
    if (s & kErrTofRange)
        return sss_set_error(SSS_ERR_TOF_RANGE,
                             "a TOF offset fell beyond the 8001-entry table (reference: IndexError)");
    if (s & kErrEnergy)
        return sss_set_error(SSS_ERR_ENERGY, "a scattered energy row fell outside the tables");
    if (s & kErrCapacity)
        return sss_set_error(SSS_ERR_CAPACITY, "an internal capacity was exceeded");
    if (s & kErrNonFinite)
        return sss_set_error(SSS_ERR_NONFINITE,
                             "a detector pair's scatter term came out infinite or NaN (the result is not "
                             "usable)");
    if (s & kErrTable)
        return sss_set_error(SSS_ERR_TABLE,
                             "an index table (sampled rings or crystals, LOR coordinates, cell or slice "
                             "table) holds an entry outside its range");
    if (s & kErrEvent)
        return sss_set_error(SSS_ERR_EVENT,
                             "a list-mode event addresses a crystal or ring outside the sinogram tables "
                             "(the reference raises IndexError here)");
    return sss_set_error(SSS_ERR_INVALID, "unknown device status 0x%x", (unsigned)s);
}

namespace {

using namespace sss;

// One thread per ray.  Variant 0 = RayTracing3DTOF (f64 lengths + samples,
// eps 1e-20); variant 1 = RayTracing3D MEX (f32 lengths, eps 1e-23).
__global__ void __launch_bounds__(128) raytrace_kernel(Grid g, const double* __restrict__ lines,
                                                       int64_t n, int variant, int cap,
                                                       int32_t* __restrict__ counts,
                                                       double* __restrict__ len64,
                                                       float* __restrict__ len32,
                                                       int32_t* __restrict__ idx,
                                                       double* __restrict__ samples,
                                                       int32_t* status)
{
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double lc[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) lc[k] = lines[6 * i + k];
    Ray r;
    const double eps = variant == 0 ? 1e-20 : 1e-23;
    if (!ray_setup(g, lc, eps, r)) {
        counts[i] = 0;
        return;
    }
    const int64_t base = i * (int64_t)cap;
    double prev = 0.0;
    int c = ray_walk(g, r, cap, [&](int k, int64_t lin, double t0, double t1) {
        double d = ref_length(r, t0, t1);
        idx[base + k] = (int32_t)lin;
        if (variant == 0) {
            if (len64) len64[base + k] = d;
            prev = add64(prev, d / 2);
            if (samples) samples[base + k] = prev;
        } else {
            if (len32) len32[base + k] = (float)d;
        }
    });
    if (c < 0) raise_error(status, kErrOverrun);
    counts[i] = c;
}

// Variant 0 with lengths, in three passes of a warp: the rays are walked one a
// lane, leaving the parameter of each crossing where its length will stand; the
// FP64 lengths (a chain of multiplications and a square root) are evaluated 32
// segments at a time; the samples, a running sum in the walk's order, one ray a
// lane again.  With the length inside the walk every step waited for that chain:
// 3001 rays through 64x64x48 voxels took 205 us, now 80 us (the walk's serial
// chain and, at two warps a SM, its latency).
constexpr int kTraceWarps = 2;

__global__ void __launch_bounds__(32 * kTraceWarps) raytrace_staged_kernel(
    Grid g, const double* __restrict__ lines, int64_t n, int cap, int rays, int32_t* __restrict__ counts, double* len64,
    int32_t* __restrict__ idx, double* __restrict__ samples, int32_t* status)
{
    const int lane = threadIdx.x & 31;
    const int64_t first = ((int64_t)blockIdx.x * kTraceWarps + (threadIdx.x >> 5)) * rays;
    if (first >= n) return;
    const int64_t i = first + lane, base = i * (int64_t)cap;
    int segments = 0;
    Ray r;
    r.xv = r.yv = r.zv = r.tmin = 0.0;
    if (lane < rays && i < n) {
        double lc[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) lc[k] = lines[6 * i + k];
        int c = 0;
        if (ray_setup(g, lc, 1e-20, r)) {
            c = ray_walk(g, r, cap, [&](int k, int64_t lin, double, double t1) {
                idx[base + k] = (int32_t)lin;
                len64[base + k] = t1;
            });
            if (c < 0) raise_error(status, kErrOverrun);
            segments = c < 0 ? cap - 1 : c;  // an overrun visits cap - 1 voxels
        }
        counts[i] = c;
    }
    __syncwarp();
    for (int j = 0; j < rays; ++j) {
        const int m = __shfl_sync(0xffffffffu, segments, j);
        Ray q;
        q.xv = __shfl_sync(0xffffffffu, r.xv, j);
        q.yv = __shfl_sync(0xffffffffu, r.yv, j);
        q.zv = __shfl_sync(0xffffffffu, r.zv, j);
        double before = __shfl_sync(0xffffffffu, r.tmin, j);  // the crossing before the chunk
        double* const row = len64 + (first + j) * (int64_t)cap;
        for (int k0 = 0; k0 < m; k0 += 32) {
            const int k = k0 + lane;
            const double t1 = k < m ? row[k] : 0.0;
            const double left = __shfl_up_sync(0xffffffffu, t1, 1);
            const double t0 = lane ? left : before;
            before = __shfl_sync(0xffffffffu, t1, 31);
            if (k < m) row[k] = ref_length(q, t0, t1);
        }
    }
    __syncwarp();
    if (!samples) return;
    double prev = 0.0;
    int k = 0;
    for (; k + 8 <= segments; k += 8) {  // eight loads in flight
        double d[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) d[u] = len64[base + k + u] / 2;
#pragma unroll
        for (int u = 0; u < 8; ++u) samples[base + k + u] = prev = add64(prev, d[u]);
    }
    for (; k < segments; ++k) samples[base + k] = prev = add64(prev, len64[base + k] / 2);
}

}  // namespace

extern "C" int sss_raytrace(const int32_t grid[3], const double bounds[6], const double* lines,
                            int64_t n_rays, int32_t variant, int32_t capacity, int32_t* counts,
                            double* lengths, float* lengths_f32, int32_t* indices,
                            double* samples, int32_t* status, void* stream)
{
    if (!grid || !bounds || (!lines && n_rays > 0) || !counts || !indices)
        return sss_set_error(SSS_ERR_INVALID, "sss_raytrace: null argument");
    if (variant != 0 && variant != 1)
        return sss_set_error(SSS_ERR_INVALID, "sss_raytrace: variant must be 0 or 1");
    if (grid[0] < 1 || grid[1] < 1 || grid[2] < 1)
        return sss_set_error(SSS_ERR_INVALID, "sss_raytrace: grid must be positive");
    if (!(bounds[3] > bounds[0] && bounds[4] > bounds[1] && bounds[5] > bounds[2]))
        return sss_set_error(SSS_ERR_INVALID, "sss_raytrace: bounds must satisfy max > min");
    int64_t need = (int64_t)grid[0] + grid[1] + grid[2];
    if (capacity < need)
        return sss_set_error(SSS_ERR_CAPACITY, "sss_raytrace: capacity %d < Nx+Ny+Nz = %lld",
                             capacity, (long long)need);
    if (n_rays <= 0) return SSS_OK;
    const Grid g = grid_of(grid[0], grid[1], grid[2], bounds);
    if (variant == 0 && lengths) {
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        // few rays are spread over the SMs, 8 a warp (3001 rays: 80 us), from 128 rays a
        // SM on a warp is filled
        const int rays = n_rays < 128ll * sms ? 8 : 32, per_block = kTraceWarps * rays;
        raytrace_staged_kernel<<<(unsigned)((n_rays + per_block - 1) / per_block), 32 * kTraceWarps, 0,
                                 (cudaStream_t)stream>>>(g, lines, n_rays, capacity, rays, counts, lengths, indices,
                                                         samples, status);
        return sss_check_launch("sss_raytrace");
    }
    const int threads = 128;
    int64_t blocks = (n_rays + threads - 1) / threads;
    raytrace_kernel<<<(unsigned)blocks, threads, 0, (cudaStream_t)stream>>>(
        g, lines, n_rays, variant, capacity, counts, lengths, lengths_f32, indices, samples,
        status);
    return sss_check_launch("sss_raytrace");
}
