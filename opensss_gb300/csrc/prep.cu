// Image preparation on the GPU: crop or zero-pad about the volume centre, then
// resize with the anti-aliasing Gaussian and cubic B-spline interpolation that
// the reference reaches through skimage.transform.resize (Python/openSSS/
// Utils.py:212-267, CropAndDownscale; :30-74, PrepareImages).  resize(order=3,
// mode='edge', anti_aliasing=True, preserve_range=True, clip=True) is, step by
// step:
//   1. a Gaussian filter per axis, sigma = max(0, (in/out - 1)/2), kernel
//      radius int(4 sigma + 0.5), edge samples repeated past the ends;
//   2. cubic B-spline coefficients of the result, computed on a copy padded by
//      12 edge samples per side (recursive filter, pole sqrt(3) - 2);
//   3. the coefficients sampled at x = (o + 0.5) in/out - 0.5 per axis;
//   4. the result clipped to the [min, max] of the cropped input.
// Steps 1 to 3 are linear and separable, and along one axis they are one short
// filter per output sample, so an axis is done in one pass: every output sample
// is a weighted sum of the input samples around it, the weights (Gaussian,
// spline response and sampling multiplied out) formed once per axis in FP64.
// The passes run from the last axis to the first and shrink the volume by each
// axis' factor as they go, so the map is read once and nothing of its size is
// written.  Measured, 400x400x280 map, 376x376x240 window to 75x75x48: eight
// full-volume passes step by step 2.20 ms, this form 0.24 ms (0.18 of them the
// pass over the map; its bytes at copy rate: 0.02 ms).
// The step-by-step form remains for what the composed one does not cover (see
// composed_fits).
// Volumes are C-ordered float32 [n0][n1][n2].
#include <math.h>

#include "common.cuh"

namespace {

constexpr int kPad = 12;        // edge samples added per side before the spline filter
constexpr int kMaxRadius = 512; // Gaussian kernel radius limit (weights in shared memory)

struct Dims {
    int n[3];
    __host__ __device__ long long count() const { return (long long)n[0] * n[1] * n[2]; }
};

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

// out[i] = in[i - before + start] per axis where that lies inside the input, else 0.
__global__ void crop_kernel(const float* __restrict__ in, Dims din, float* __restrict__ out, Dims dout,
                            int3 start, int3 before)
{
    const long long total = dout.count();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int k = (int)(i % dout.n[2]);
        const int j = (int)((i / dout.n[2]) % dout.n[1]);
        const int h = (int)(i / ((long long)dout.n[2] * dout.n[1]));
        const int a = h - before.x + start.x, b = j - before.y + start.y, c = k - before.z + start.z;
        float v = 0.f;
        if (a >= 0 && a < din.n[0] && b >= 0 && b < din.n[1] && c >= 0 && c < din.n[2])
            v = in[((long long)a * din.n[1] + b) * din.n[2] + c];
        out[i] = v;
    }
}

// Per-block minimum and maximum of x[0..n) into part[2 * block].
__global__ void __launch_bounds__(256) minmax_partial_kernel(const float* __restrict__ x, long long n,
                                                             float* __restrict__ part)
{
    float lo = INFINITY, hi = -INFINITY;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const float v = x[i];
        lo = fminf(lo, v);
        hi = fmaxf(hi, v);
    }
    __shared__ float slo[256], shi[256];
    slo[threadIdx.x] = lo;
    shi[threadIdx.x] = hi;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) {
            slo[threadIdx.x] = fminf(slo[threadIdx.x], slo[threadIdx.x + s]);
            shi[threadIdx.x] = fmaxf(shi[threadIdx.x], shi[threadIdx.x + s]);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = slo[0];
        part[2 * blockIdx.x + 1] = shi[0];
    }
}

// Reduces nb per-block pairs to part[0] = min, part[1] = max (one block).
__global__ void __launch_bounds__(256) minmax_final_kernel(float* __restrict__ part, int nb)
{
    float lo = INFINITY, hi = -INFINITY;
    for (int i = threadIdx.x; i < nb; i += blockDim.x) {
        lo = fminf(lo, part[2 * i]);
        hi = fmaxf(hi, part[2 * i + 1]);
    }
    __shared__ float slo[256], shi[256];
    slo[threadIdx.x] = lo;
    shi[threadIdx.x] = hi;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) {
            slo[threadIdx.x] = fminf(slo[threadIdx.x], slo[threadIdx.x + s]);
            shi[threadIdx.x] = fmaxf(shi[threadIdx.x], shi[threadIdx.x + s]);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        part[0] = slo[0];
        part[1] = shi[0];
    }
}

// One axis of the Gaussian filter: out = sum_k w[k] in[clamp(i + k - r)] along
// `axis` (edge samples repeated).  Weights are FP32 copies of the normalised
// FP64 kernel, staged in shared memory.  I: the index type, 32-bit unsigned
// for volumes below 2^31 elements (the index arithmetic is most of the
// kernel's instructions), 64-bit above.
template <typename I>
__global__ void __launch_bounds__(256) gauss_axis_kernel(const float* __restrict__ in, float* __restrict__ out,
                                                         Dims d, int axis, const float* __restrict__ w, int r)
{
    __shared__ float sw[2 * kMaxRadius + 1];
    for (int i = threadIdx.x; i <= 2 * r; i += blockDim.x) sw[i] = w[i];
    __syncthreads();
    const I total = (I)d.count();
    const I stride = axis == 2 ? (I)1 : (axis == 1 ? (I)d.n[2] : (I)d.n[1] * (I)d.n[2]);
    const int len = d.n[axis];
    for (I i = (I)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (I)gridDim.x * blockDim.x) {
        const int p = (int)((i / stride) % (I)len);  // position along the axis
        const I base = i - (I)p * stride;
        float acc = 0.f;
        if (p >= r && p + r < len) {  // no sample past an end: a running offset
            I q = base + (I)(p - r) * stride;
            for (int k = 0; k <= 2 * r; ++k, q += stride) acc = fmaf(sw[k], in[q], acc);
        } else {
            for (int k = -r; k <= r; ++k) acc = fmaf(sw[k + r], in[base + (I)clampi(p + k, 0, len - 1) * stride], acc);
        }
        out[i] = acc;
    }
}

// Edge padding by kPad samples on every side: P[p] = F[clamp(p - kPad)].
__global__ void pad_edge_kernel(const float* __restrict__ f, Dims d, float* __restrict__ P, Dims dp)
{
    const long long total = dp.count();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int k = (int)(i % dp.n[2]);
        const int j = (int)((i / dp.n[2]) % dp.n[1]);
        const int h = (int)(i / ((long long)dp.n[2] * dp.n[1]));
        const int a = clampi(h - kPad, 0, d.n[0] - 1), b = clampi(j - kPad, 0, d.n[1] - 1),
                  c = clampi(k - kPad, 0, d.n[2] - 1);
        P[i] = f[((long long)a * d.n[1] + b) * d.n[2] + c];
    }
}

// Cubic B-spline coefficients along `axis`, in place, one thread per line
// (Unser's recursive filter: gain 6, causal and anti-causal passes with pole
// z = sqrt(3) - 2, mirror-symmetric start values).  The 12 edge samples in
// front of the data make the start values' effect on the data below z^12.
constexpr int kSplineAhead = 8;  // values loaded ahead of the in-place recursion

__global__ void spline_axis_kernel(float* __restrict__ P, Dims d, int axis)
{
    const float z = -0.26794919243112270f;  // sqrt(3) - 2
    const long long stride = axis == 2 ? 1 : (axis == 1 ? d.n[2] : (long long)d.n[1] * d.n[2]);
    const int len = d.n[axis];
    const long long lines = d.count() / len;
    for (long long l = (long long)blockIdx.x * blockDim.x + threadIdx.x; l < lines;
         l += (long long)gridDim.x * blockDim.x) {
        // line l: the other two indices in C order
        long long base;
        if (axis == 2) {
            base = l * len;
        } else if (axis == 1) {
            const long long h = l / d.n[2], k = l % d.n[2];
            base = h * (long long)d.n[1] * d.n[2] + k;
        } else {
            base = l;  // l = j * n2 + k
        }
        float* x = P + base;
        // causal start: sum_k z^k c[k] over the first terms (z^28 < 1e-16)
        const int kmax = len < 28 ? len : 28;
        float zk = 1.f, c0 = 0.f;
        for (int k = 0; k < kmax; ++k) {
            c0 = fmaf(zk, 6.f * x[k * stride], c0);
            zk *= z;
        }
        x[0] = c0;
        float prev = c0;
        // The recursion runs in place, so each load would otherwise wait for
        // the store before it: kSplineAhead values are loaded together first
        // (none of them written yet), then filtered and stored.
        int k = 1;
        for (; k + kSplineAhead <= len; k += kSplineAhead) {
            float v[kSplineAhead];
#pragma unroll
            for (int j = 0; j < kSplineAhead; ++j) v[j] = x[(long long)(k + j) * stride];
#pragma unroll
            for (int j = 0; j < kSplineAhead; ++j) {
                prev = fmaf(z, prev, 6.f * v[j]);
                x[(long long)(k + j) * stride] = prev;
            }
        }
        for (; k < len; ++k) {
            prev = fmaf(z, prev, 6.f * x[(long long)k * stride]);
            x[(long long)k * stride] = prev;
        }
        // anti-causal start from the last two causal values
        float next = (z / (z * z - 1.f)) * fmaf(z, len > 1 ? x[(long long)(len - 2) * stride] : prev, prev);
        x[(long long)(len - 1) * stride] = next;
        k = len - 2;
        for (; k - kSplineAhead + 1 >= 0; k -= kSplineAhead) {
            float v[kSplineAhead];
#pragma unroll
            for (int j = 0; j < kSplineAhead; ++j) v[j] = x[(long long)(k - j) * stride];
#pragma unroll
            for (int j = 0; j < kSplineAhead; ++j) {
                next = z * (next - v[j]);
                x[(long long)(k - j) * stride] = next;
            }
        }
        for (; k >= 0; --k) {
            next = z * (next - x[(long long)k * stride]);
            x[(long long)k * stride] = next;
        }
    }
}

__device__ __forceinline__ void cubic_weights(double x, int& i0, float w[4])
{
    const double f = floor(x);
    const float t = (float)(x - f);
    const float t2 = t * t, t3 = t2 * t, u = 1.f - t;
    w[0] = u * u * u * (1.f / 6.f);
    w[1] = (3.f * t3 - 6.f * t2 + 4.f) * (1.f / 6.f);
    w[2] = (-3.f * t3 + 3.f * t2 + 3.f * t + 1.f) * (1.f / 6.f);
    w[3] = t3 * (1.f / 6.f);
    i0 = (int)f - 1 + kPad;
}

// Output voxel o: the coefficients sampled at x_d = (o_d + 0.5) in_d/out_d - 0.5,
// clipped to [lim[0], lim[1]] when clip is set; values below zero_below become 0.
__global__ void zoom_kernel(const float* __restrict__ P, Dims dp, Dims din, float* __restrict__ out, Dims dout,
                            const float* __restrict__ lim, int clip, float zero_below)
{
    const long long total = dout.count();
    const float lo = clip ? lim[0] : -INFINITY, hi = clip ? lim[1] : INFINITY;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int o2 = (int)(i % dout.n[2]);
        const int o1 = (int)((i / dout.n[2]) % dout.n[1]);
        const int o0 = (int)(i / ((long long)dout.n[2] * dout.n[1]));
        int a0, a1, a2;
        float w0[4], w1[4], w2[4];
        cubic_weights((o0 + 0.5) * ((double)din.n[0] / dout.n[0]) - 0.5, a0, w0);
        cubic_weights((o1 + 0.5) * ((double)din.n[1] / dout.n[1]) - 0.5, a1, w1);
        cubic_weights((o2 + 0.5) * ((double)din.n[2] / dout.n[2]) - 0.5, a2, w2);
        float acc = 0.f;
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            float accp = 0.f;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float* row = P + ((long long)(a0 + p) * dp.n[1] + (a1 + q)) * dp.n[2] + a2;
                const float s = fmaf(w2[0], row[0], fmaf(w2[1], row[1], fmaf(w2[2], row[2], w2[3] * row[3])));
                accp = fmaf(w1[q], s, accp);
            }
            acc = fmaf(w0[p], accp, acc);
        }
        acc = fminf(fmaxf(acc, lo), hi);
        out[i] = acc < zero_below ? 0.f : acc;
    }
}

// ---------------------------------------------------------------- composed form

// Samples either side of a coefficient that its spline response takes: the
// response falls as 0.268^distance, 3.6e-12 at this reach.  (The 12 repeated edge
// samples and the mirror beyond them are then the same as repeating the edge
// sample throughout.)
constexpr int kReach = 20;
constexpr int kTaps = 2 * kReach + 4;  // samples under an output sample's four coefficients
constexpr int kGroup = 4;              // neighbouring output samples computed together
constexpr int kLinePos = 512;          // samples of a line staged at once by line_axis_kernel
constexpr int kLines = 32;             // lines of a line_axis_kernel block

// One axis: n input samples, m output samples, Gaussian radius r (0: none).  A
// group of kGroup output samples takes the input samples from start[g] on,
// weight[g * span + u] being sample start[g] + u's weight in each of them.
struct Axis {
    int n, m, r, span, groups;
    double sigma;
    int* start;
    float4* weight;
};

struct Axes {
    Axis a[3];
};

__host__ __device__ inline int clamp_pos(long long v, int n) { return v < 0 ? 0 : (v >= n ? n - 1 : (int)v); }

// Position of output sample o on its axis (floor and remainder).
__host__ __device__ inline double sample_pos(const Axis& A, int o)
{
    return (o + 0.5) * ((double)A.n / A.m) - 0.5;
}

// Input samples of the group whose first output sample is o: [first, last].
__host__ __device__ inline void group_span(const Axis& A, int o, int& first, int& last)
{
    const int e = o + kGroup - 1 < A.m ? o + kGroup - 1 : A.m - 1;
    first = clamp_pos((long long)floor(sample_pos(A, o)) - 1 - kReach - A.r, A.n);
    last = clamp_pos((long long)floor(sample_pos(A, e)) + 2 + kReach + A.r, A.n);
}

constexpr int kWeightThreads = 320;

// The composed weights, one block a group; blocks 0.. of axis 0, then 1, then 2.
// limits: [0] min, [1] max (as ordered ints), [2] non-finite input seen; reset here.
__global__ void __launch_bounds__(kWeightThreads) axis_weights_kernel(Axes X, int* limits)
{
    __shared__ double gauss[2 * kMaxRadius + 1], cum[2 * kMaxRadius + 1];
    __shared__ double q[kGroup][kTaps], zp[kTaps];
    __shared__ double total;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        limits[0] = 0x7F800000;       // +infinity, ordered
        limits[1] = (int)0x807FFFFF;  // -infinity, ordered
        limits[2] = 0;
    }
    int g = blockIdx.x, d = 0;
    while (g >= X.a[d].groups) g -= X.a[d++].groups;
    const Axis A = X.a[d];
    const int r = A.r, nk = 2 * r + 1;
    for (int k = threadIdx.x; k < nk; k += blockDim.x)
        gauss[k] = r > 0 ? exp(-0.5 / (A.sigma * A.sigma) * (double)(k - r) * (double)(k - r)) : 1.0;
    // spline response: the weight of a sample at a distance from its coefficient
    const double z = -0.26794919243112270;
    if (threadIdx.x < kTaps) {
        double v = -6.0 * z / (1.0 - z * z), b = z;
        for (int e = threadIdx.x; e; e >>= 1, b *= b)
            if (e & 1) v *= b;
        zp[threadIdx.x] = v;
    }
    __syncthreads();
    if (threadIdx.x == kWeightThreads - 1) {
        double s = 0.0;
        for (int k = 0; k < nk; ++k) cum[k] = s += gauss[k];
        total = s;
    }
    // times the cubic weight of the coefficient in the output sample
    for (int i = threadIdx.x; i < kGroup * kTaps; i += blockDim.x) {
        const int o = g * kGroup + i / kTaps, m = i % kTaps;
        double v = 0.0;
        if (o < A.m) {
            const double x = sample_pos(A, o), t = x - floor(x), u = 1.0 - t;
            const double w[4] = {u * u * u / 6.0, (3.0 * t * t * t - 6.0 * t * t + 4.0) / 6.0,
                                 (-3.0 * t * t * t + 3.0 * t * t + 3.0 * t + 1.0) / 6.0, t * t * t / 6.0};
            for (int p = 0; p < 4; ++p) v += w[p] * zp[abs(m - kReach - p)];
        }
        q[i / kTaps][m] = v;
    }
    __syncthreads();
    const double norm = 1.0 / total;
    int first, last;
    group_span(A, g * kGroup, first, last);
    if (threadIdx.x == 0) A.start[g] = first;
    float* out = reinterpret_cast<float*>(A.weight + (long long)g * A.span);
    for (int i = threadIdx.x; i < A.span * kGroup; i += blockDim.x) {
        const int c = first + i / kGroup, j = i % kGroup, o = g * kGroup + j;
        double v = 0.0;
        if (o < A.m && c <= last) {
            const long long f0 = (long long)floor(sample_pos(A, o)) - 1 - kReach;
            int m0 = 0, m1 = kTaps;  // away from the ends only samples within r of c
            if (f0 >= 0 && f0 + kTaps <= A.n && c > 0 && c < A.n - 1) {
                m0 = max(0, (int)(c - r - f0));
                m1 = min(kTaps, (int)(c + r - f0) + 1);
            }
            for (int m = m0; m < m1; ++m) {
                // weight of input sample c in the Gaussian at sample f, whose
                // taps past an end all fall on that end
                const int f = clamp_pos(f0 + m, A.n), k = c - f + r;
                double gw = 0.0;
                if (A.n == 1) gw = total;
                else if (c == 0) gw = k < 0 ? 0.0 : (k >= nk ? total : cum[k]);
                else if (c == A.n - 1) gw = k >= nk ? 0.0 : (k <= 0 ? total : total - cum[k - 1]);
                else if (k >= 0 && k < nk) gw = gauss[k];
                v += q[j][m] * gw;
            }
            v *= norm;
        }
        out[i] = (float)v;
    }
}

// Order-preserving int of a float (NaN not compared).
__device__ __forceinline__ int ordered(float v)
{
    const int b = __float_as_int(v);
    return b < 0 ? b ^ 0x7FFFFFFF : b;
}
__device__ __forceinline__ float from_ordered(int b) { return __int_as_float(b < 0 ? b ^ 0x7FFFFFFF : b); }

struct Crop {
    const float* image;
    Dims image_dims, dims;
    int start[3], before[3];
    // window sample i of axis d in the image, or -1
    __device__ __forceinline__ int at(int d, int i) const
    {
        const int p = i - before[d] + start[d];
        return p >= 0 && p < image_dims.n[d] ? p : -1;
    }
};

__device__ __forceinline__ void copy_async4(float* dst, const float* src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

constexpr int kLineThreads = 128;

// The last (contiguous) axis, read from the image through the crop window: a
// block takes kLines lines, stages the samples of as many groups as fit and
// computes them lane = line, four outputs a sample read.  Also the window's
// minimum, maximum and whether it is finite.  Bound by the latency of its
// shared-memory and weight loads (11 weights a sample; issue 40%, L1 69%), at
// 0.8 TB/s of the window: 0.18 ms for 376x376x240 samples.
__global__ void __launch_bounds__(kLineThreads) line_axis_kernel(Crop K, Axis A, float* __restrict__ out, int* limits)
{
    extern __shared__ float xs[];  // [position][kLines + 1]
    constexpr int kWarps = kLineThreads / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long lines = (long long)K.dims.n[0] * K.dims.n[1], line0 = (long long)blockIdx.x * kLines;
    float lo = INFINITY, hi = -INFINITY;
    bool finite = true;
    for (int g0 = 0; g0 < A.groups;) {
        const int p0 = A.start[g0];
        int g1 = g0 + 1;
        while (g1 < A.groups && A.start[g1] + A.span - p0 <= kLinePos) ++g1;
        const int p1 = min(A.n, A.start[g1 - 1] + A.span);
        __syncthreads();
        for (int l = warp; l < kLines; l += kWarps) {
            const long long line = line0 + l;
            const float* src = nullptr;
            if (line < lines) {
                const int a = K.at(0, (int)(line / K.dims.n[1])), b = K.at(1, (int)(line % K.dims.n[1]));
                if (a >= 0 && b >= 0)
                    src = K.image + ((long long)a * K.image_dims.n[1] + b) * K.image_dims.n[2];
            }
            // asynchronous copies: all of a thread's samples are in flight at once
            for (int p = p0 + lane; p < p1; p += 32) {
                const int c = K.at(2, p);
                float* dst = xs + (p - p0) * (kLines + 1) + l;
                if (src && c >= 0) copy_async4(dst, src + c);
                else *dst = 0.f;
            }
        }
        copy_async_wait();
        __syncthreads();
        if (line0 + lane < lines)
            for (int p = warp; p < p1 - p0; p += kWarps) {
                const float v = xs[p * (kLines + 1) + lane];
                lo = fminf(lo, v);
                hi = fmaxf(hi, v);
                finite &= isfinite(v);
            }
        for (int g = g0 + warp; g < g1; g += kWarps) {
            const float4* w = A.weight + (long long)g * A.span;
            const float* x = xs + (A.start[g] - p0) * (kLines + 1) + lane;
            const int span = min(A.span, p1 - A.start[g]);
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
            for (int u = 0; u < span; ++u) {
                const float4 c = __ldg(w + u);
                const float v = x[u * (kLines + 1)];
                acc.x = fmaf(c.x, v, acc.x);
                acc.y = fmaf(c.y, v, acc.y);
                acc.z = fmaf(c.z, v, acc.z);
                acc.w = fmaf(c.w, v, acc.w);
            }
            const long long line = line0 + lane;
            if (line < lines) {
                float* o = out + line * A.m + g * kGroup;
                o[0] = acc.x;
                if (g * kGroup + 1 < A.m) o[1] = acc.y;
                if (g * kGroup + 2 < A.m) o[2] = acc.z;
                if (g * kGroup + 3 < A.m) o[3] = acc.w;
            }
        }
        g0 = g1;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    const bool bad = __any_sync(0xffffffffu, !finite);
    if (lane == 0) {
        if (lo <= hi) {
            atomicMin(limits, ordered(lo));
            atomicMax(limits + 1, ordered(hi));
        }
        if (bad) atomicOr(limits + 2, 1);
    }
}

// Minimum, maximum and finiteness of a window whose lines line_axis_kernel does
// not read completely (a factor above the filter's length).
__global__ void __launch_bounds__(256) crop_limits_kernel(Crop K, int* limits)
{
    const long long total = K.dims.count();
    float lo = INFINITY, hi = -INFINITY;
    bool finite = true;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int c = K.at(2, (int)(i % K.dims.n[2])), b = K.at(1, (int)(i / K.dims.n[2] % K.dims.n[1])),
                  a = K.at(0, (int)(i / ((long long)K.dims.n[2] * K.dims.n[1])));
        const float v = a >= 0 && b >= 0 && c >= 0
                            ? __ldg(K.image + ((long long)a * K.image_dims.n[1] + b) * K.image_dims.n[2] + c)
                            : 0.f;
        lo = fminf(lo, v);
        hi = fmaxf(hi, v);
        finite &= isfinite(v);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    const bool bad = __any_sync(0xffffffffu, !finite);
    if ((threadIdx.x & 31) == 0) {
        if (lo <= hi) {
            atomicMin(limits, ordered(lo));
            atomicMax(limits + 1, ordered(hi));
        }
        if (bad) atomicOr(limits + 2, 1);
    }
}

// A strided axis: in [outer][n][inner] -> out [outer][m][inner], one thread per
// (outer, inner) and group of outputs (blockIdx.y).  FINAL: the result, clipped
// to [min, max] when clip is set, values below zero_below 0; a window with a
// non-finite sample has none that is finite (every line of coefficients through
// it would be NaN), which the clip turns into the minimum.
template <bool FINAL>
__global__ void __launch_bounds__(128) strided_axis_kernel(const float* __restrict__ in, float* __restrict__ out,
                                                           long long outer, long long inner, Axis A,
                                                           const int* __restrict__ limits, int clip, float zero_below)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= outer * inner) return;
    const long long oi = i / inner, ii = i % inner;
    const int g = blockIdx.y, first = A.start[g], span = min(A.span, A.n - first);
    const float4* w = A.weight + (long long)g * A.span;
    const float* x = in + (oi * A.n + first) * inner + ii;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
    for (int u = 0; u < span; ++u) {
        const float4 c = __ldg(w + u);
        const float v = __ldg(x + (long long)u * inner);
        acc.x = fmaf(c.x, v, acc.x);
        acc.y = fmaf(c.y, v, acc.y);
        acc.z = fmaf(c.z, v, acc.z);
        acc.w = fmaf(c.w, v, acc.w);
    }
    float r[kGroup] = {acc.x, acc.y, acc.z, acc.w};
    if (FINAL) {
        const float lo = clip ? from_ordered(limits[0]) : -INFINITY, hi = clip ? from_ordered(limits[1]) : INFINITY;
        const bool bad = limits[2];
#pragma unroll
        for (int k = 0; k < kGroup; ++k) {
            const float v = fminf(fmaxf(bad ? NAN : r[k], lo), hi);
            r[k] = v < zero_below ? 0.f : v;
        }
    }
    float* o = out + (oi * A.m + g * kGroup) * inner + ii;
#pragma unroll
    for (int k = 0; k < kGroup; ++k)
        if (g * kGroup + k < A.m) o[k * inner] = r[k];
}

int grid_for(long long n, int threads = 256)
{
    long long b = (n + threads - 1) / threads;
    return (int)(b < 1 ? 1 : (b > 152 * 64 ? 152 * 64 : b));
}

constexpr int kMinmaxBlocks = 1024;

size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

struct PrepLayout {
    size_t crop, tmp, padded, part, weights, total;
};

PrepLayout prep_layout(const int crop[3])
{
    const long long c = (long long)crop[0] * crop[1] * crop[2];
    const long long p = (long long)(crop[0] + 2 * kPad) * (crop[1] + 2 * kPad) * (crop[2] + 2 * kPad);
    PrepLayout L;
    L.crop = 0;
    L.tmp = L.crop + align256(c * sizeof(float));
    L.padded = L.tmp + align256(c * sizeof(float));
    L.part = L.padded + align256(p * sizeof(float));
    L.weights = L.part + align256(2 * kMinmaxBlocks * sizeof(float));
    L.total = L.weights + align256(3 * (2 * kMaxRadius + 1) * sizeof(float));
    return L;
}

// Workspace of the composed form: the volumes after the last and the middle
// axis, limits, starts and weights.
struct ComposedLayout {
    size_t after2, after1, limits, start[3], weight[3], total;
};

// Whether the composed form applies: its volumes fit the workspace (sized for
// the step-by-step form; strong enlargements do not) and a group of the last
// axis fits the staged samples (factors up to about 60).

bool composed_fits(const int crop[3], const int outd[3], const int radius[3], const double sigma[3], size_t have, Axes& X,
                   ComposedLayout& L)
{
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t at = off;
        off = align256(off + bytes);
        return at;
    };
    for (int d = 0; d < 3; ++d) {
        Axis& A = X.a[d];
        A.n = crop[d];
        A.m = outd[d];
        A.r = radius[d] > 0 ? radius[d] : 0;
        A.sigma = sigma[d];
        A.groups = (A.m + kGroup - 1) / kGroup;
        const double want = kTaps + 2.0 * A.r + 3.0 * (double)A.n / A.m + 2.0;  // samples a group can take
        A.span = want < A.n ? (int)want : A.n;
        if (A.groups > 65535) return false;
    }
    // a group of the last axis has to fit the staged samples
    if (X.a[2].span > kLinePos) return false;
    L.after2 = take(sizeof(float) * (size_t)crop[0] * crop[1] * outd[2]);
    L.after1 = take(sizeof(float) * (size_t)crop[0] * outd[1] * outd[2]);
    L.limits = take(3 * sizeof(int));
    for (int d = 0; d < 3; ++d) {
        L.start[d] = take(sizeof(int) * X.a[d].groups);
        L.weight[d] = take(sizeof(float4) * (size_t)X.a[d].groups * X.a[d].span);
    }
    L.total = off;
    return off <= have;
}

int composed_downscale(const Crop& K, Axes& X, const ComposedLayout& L, int clip, float zero_below, float* out,
                       unsigned char* ws, cudaStream_t st)
{
    for (int d = 0; d < 3; ++d) {
        X.a[d].start = (int*)(ws + L.start[d]);
        X.a[d].weight = (float4*)(ws + L.weight[d]);
    }
    int* limits = (int*)(ws + L.limits);
    float *after2 = (float*)(ws + L.after2), *after1 = (float*)(ws + L.after1);
    axis_weights_kernel<<<X.a[0].groups + X.a[1].groups + X.a[2].groups, kWeightThreads, 0, st>>>(X, limits);
    const size_t smem = sizeof(float) * kLinePos * (kLines + 1);
    if (cudaFuncSetAttribute((const void*)line_axis_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
        cudaSuccess)
        return sss_set_error(SSS_ERR_CUDA, "sss_crop_downscale: %zu bytes of shared memory refused", smem);
    const long long lines = (long long)K.dims.n[0] * K.dims.n[1];
    const int used = X.a[2].n < kLinePos ? X.a[2].n : kLinePos;
    line_axis_kernel<<<(unsigned)((lines + kLines - 1) / kLines), kLineThreads, sizeof(float) * used * (kLines + 1), st>>>(
        K, X.a[2], after2, limits);
    // lines with gaps between the groups' samples: the limits need a pass of their own
    if ((double)X.a[2].n / X.a[2].m > kTaps)
        crop_limits_kernel<<<grid_for(K.dims.count()), 256, 0, st>>>(K, limits);
    auto strided = [&](auto kern, const float* in, float* to, long long outer, long long inner, const Axis& A) {
        kern<<<dim3((unsigned)((outer * inner + 127) / 128), (unsigned)A.groups), 128, 0, st>>>(in, to, outer, inner, A,
                                                                                              limits, clip, zero_below);
    };
    strided(strided_axis_kernel<false>, after2, after1, X.a[0].n, X.a[2].m, X.a[1]);
    strided(strided_axis_kernel<true>, after1, out, 1, (long long)X.a[1].m * X.a[2].m, X.a[0]);
    return sss_check_launch("sss_crop_downscale");
}

}  // namespace

extern "C" size_t sss_crop_downscale_workspace_size(const int crop_dims[3])
{
    if (!crop_dims || crop_dims[0] < 1 || crop_dims[1] < 1 || crop_dims[2] < 1) return 0;
    return prep_layout(crop_dims).total;
}

extern "C" int sss_crop_downscale(const float* image, const int image_dims[3], const int crop_start[3],
                                  const int crop_before[3], const int crop_dims[3], const int out_dims[3],
                                  const double sigma[3], int clip, float zero_below, float* out, void* workspace,
                                  size_t workspace_bytes, void* stream)
{
    if (!image || !image_dims || !crop_start || !crop_before || !crop_dims || !out_dims || !sigma || !out)
        return sss_set_error(SSS_ERR_INVALID, "sss_crop_downscale: null argument");
    for (int d = 0; d < 3; ++d) {
        if (image_dims[d] < 1 || crop_dims[d] < 1 || out_dims[d] < 1)
            return sss_set_error(SSS_ERR_INVALID, "sss_crop_downscale: empty dimension %d", d);
        if (!(sigma[d] >= 0.0) || sigma[d] > 100.0)
            return sss_set_error(SSS_ERR_INVALID, "sss_crop_downscale: sigma[%d] = %g outside [0, 100]", d, sigma[d]);
        if ((long long)crop_dims[d] + 2 * kPad > (1ll << 30))
            return sss_set_error(SSS_ERR_INVALID, "sss_crop_downscale: crop dimension %d too large", d);
    }
    const PrepLayout L = prep_layout(crop_dims);
    if (!workspace || workspace_bytes < L.total)
        return sss_set_error(SSS_ERR_WORKSPACE, "sss_crop_downscale: workspace of %zu bytes, %zu needed",
                             workspace_bytes, L.total);
    cudaStream_t st = (cudaStream_t)stream;
    unsigned char* ws = (unsigned char*)workspace;
    float* crop = (float*)(ws + L.crop);
    float* tmp = (float*)(ws + L.tmp);
    float* padded = (float*)(ws + L.padded);
    float* part = (float*)(ws + L.part);
    float* wdev = (float*)(ws + L.weights);

    const Dims din = {{image_dims[0], image_dims[1], image_dims[2]}};
    const Dims dc = {{crop_dims[0], crop_dims[1], crop_dims[2]}};
    const Dims dp = {{crop_dims[0] + 2 * kPad, crop_dims[1] + 2 * kPad, crop_dims[2] + 2 * kPad}};
    const Dims dout = {{out_dims[0], out_dims[1], out_dims[2]}};

    int radius[3];
    for (int d = 0; d < 3; ++d) {
        radius[d] = -1;
        if (sigma[d] <= 1e-15) continue;  // axes with a zero sigma are left unfiltered
        radius[d] = (int)(4.0 * sigma[d] + 0.5);
        if (radius[d] > kMaxRadius)
            return sss_set_error(SSS_ERR_INVALID, "sss_crop_downscale: kernel radius %d", radius[d]);
    }
    Axes X;
    ComposedLayout CL;
    if ((uintptr_t)workspace % 16 == 0 && composed_fits(crop_dims, out_dims, radius, sigma, workspace_bytes, X, CL)) {
        Crop K;
        K.image = image;
        K.image_dims = din;
        K.dims = dc;
        for (int d = 0; d < 3; ++d) {
            K.start[d] = crop_start[d];
            K.before[d] = crop_before[d];
        }
        return composed_downscale(K, X, CL, clip, zero_below, out, ws, st);
    }

    // Gaussian weights (FP64, normalised, then rounded to FP32) for every axis filtered
    float hw[3][2 * kMaxRadius + 1];
    for (int d = 0; d < 3; ++d) {
        if (radius[d] < 0) continue;
        const int r = radius[d];
        double sum = 0.0, tmpw[2 * kMaxRadius + 1];
        for (int k = -r; k <= r; ++k) sum += (tmpw[k + r] = exp(-0.5 / (sigma[d] * sigma[d]) * k * k));
        for (int k = 0; k <= 2 * r; ++k) hw[d][k] = (float)(tmpw[k] / sum);
    }
    for (int d = 0; d < 3; ++d)
        if (radius[d] >= 0 &&
            cudaMemcpyAsync(wdev + d * (2 * kMaxRadius + 1), hw[d], (2 * radius[d] + 1) * sizeof(float),
                            cudaMemcpyHostToDevice, st) != cudaSuccess)
            return sss_set_error(SSS_ERR_CUDA, "sss_crop_downscale: weight upload failed");

    const long long nc = dc.count();
    crop_kernel<<<grid_for(nc), 256, 0, st>>>(image, din, crop, dc,
                                              make_int3(crop_start[0], crop_start[1], crop_start[2]),
                                              make_int3(crop_before[0], crop_before[1], crop_before[2]));
    const int nb = (int)(nc / 256 + 1 < kMinmaxBlocks ? nc / 256 + 1 : kMinmaxBlocks);
    minmax_partial_kernel<<<nb, 256, 0, st>>>(crop, nc, part);
    minmax_final_kernel<<<1, 256, 0, st>>>(part, nb);
    // Gaussian per axis, ping-pong between crop and tmp (the cropped input is kept for nothing else)
    float* cur = crop;
    float* other = tmp;
    for (int d = 0; d < 3; ++d) {
        if (radius[d] < 0) continue;
        if (nc < (1ll << 31))
            gauss_axis_kernel<unsigned><<<grid_for(nc), 256, 0, st>>>(cur, other, dc, d,
                                                                      wdev + d * (2 * kMaxRadius + 1), radius[d]);
        else
            gauss_axis_kernel<long long><<<grid_for(nc), 256, 0, st>>>(cur, other, dc, d,
                                                                       wdev + d * (2 * kMaxRadius + 1), radius[d]);
        float* t = cur;
        cur = other;
        other = t;
    }
    const long long np = dp.count();
    pad_edge_kernel<<<grid_for(np), 256, 0, st>>>(cur, dc, padded, dp);
    for (int d = 0; d < 3; ++d) {
        const long long lines = np / dp.n[d];
        spline_axis_kernel<<<grid_for(lines, 128), 128, 0, st>>>(padded, dp, d);
    }
    zoom_kernel<<<grid_for(dout.count()), 256, 0, st>>>(padded, dp, dc, out, dout, part, clip, zero_below);
    return sss_check_launch("sss_crop_downscale");
}
