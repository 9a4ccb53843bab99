// fjb_scanner_post.cu -- scanner post effects on linear output-RGB planes.
//
// Restates src/Cuda/Scan/JuicerCudaScanPipeline.cu of the reference:
//   glare      :273-316  per-pixel lognormal glare percent from a Box-Muller normal of the
//                        Philox stream (seed, absolute x, medium, absolute y), :214-256;
//   blurs      :318-446  separable Gaussian, half-sample reflection repeated as needed
//                        (:258-270), taps summed in order in FP64, stored as float
//                        (0 when not finite);
//   unsharp    :586-655  vertical pass of the horizontally blurred plane combined as
//                        v + amount (v - blurred) in FP64;
//   schedule   :2586-2878 glare (+ its blur) before the scan to linear RGB, then lens blur
//                        and unsharp per plane, then output encoding.
// Planes are dense (width floats per row). Arithmetic order and rounding points follow the
// reference so results match it to the last bit.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "fjb_launches.h"
#include "fjb_line_pairs.cuh"
#include "fjb_philox.cuh"
#include "fjb_scanner_post.h"

namespace fjb {

namespace {

__device__ __forceinline__ int reflect_wide(long long i, int n) {
    if (n <= 1) return 0;
    while (i < 0 || i >= n) i = i < 0 ? -i - 1 : 2LL * n - i - 1;
    return (int)i;
}

__device__ __forceinline__ bool finite_d(double v) { return isfinite(v) && !isnan(v); }
__device__ __forceinline__ bool finite_f(float v) { return isfinite(v) && !isnan(v); }

__global__ void glare_kernel(float* out, int width, int height, uint64_t seed, uint32_t medium, int origin_x,
                             int origin_y, float percent, float roughness) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= width || y >= height) return;
    const float mean = fmaxf(0.0f, percent);
    const float stddev = fmaxf(0.0f, roughness * percent);
    const uint64_t ax = (uint64_t)((int64_t)origin_x + (int64_t)x);
    const uint64_t ay = (uint64_t)((int64_t)origin_y + (int64_t)y);
    Philox rng(seed, (uint32_t)ax, medium, (uint32_t)ay);
    float u1 = philox_u01(rng.next());
    u1 = fminf(fmaxf(u1, 1e-7f), 1.0f);
    const float u2 = philox_u01(rng.next());
    const float r = sqrtf(-2.0f * logf(u1));
    constexpr float kTwoPi = 6.28318530717958647692f;
    const float n = r * cosf(kTwoPi * u2);
    // lognormal with the given mean and standard deviation
    const float m2 = mean * mean;
    const float s2 = stddev * stddev;
    const float sigmaSq = logf(1.0f + (s2 / m2));
    const float sigma = sqrtf(fmaxf(0.0f, sigmaSq));
    const float mu = logf(fmaxf(1e-12f, mean)) - 0.5f * sigmaSq;
    const float glare = expf(mu + sigma * n);
    out[(size_t)y * width + x] = finite_f(glare) ? glare : 0.0f;
}

// ---------------------------------------------------------------------------
// Run form of the blurs: a thread computes kRun consecutive outputs. Its inputs sit in
// a ring of kRun doubles (each converted once), and output j still sums its taps in order,
// starting from zero.
// The taps are in shared memory as doubles, converted once per CTA.
//
// Bound by instruction issue at the ordinary radii, most of it around the sums: a warp
// takes a segment of one row (no divisions to place a run or an output), loads are
// asynchronous or unconditional where nothing is reflected. 1999x1333, glare, lens
// blur and unsharp (seven planes): rows 122 -> 46 us, columns 84 -> 73 us. Radius 80, three
// planes: 119 and 269 us (a 64-bit row index where rows are reflected: 306).
// ---------------------------------------------------------------------------
constexpr int kRun = 9; // odd: threads nine samples apart read distinct shared-memory banks
constexpr int kSegment = 32 * kRun;
constexpr int kRowWarps = 8, kColWarps = 8;

struct Planes {
    float* p[3];
};

__device__ __forceinline__ void stage_taps(double* taps, const float* __restrict__ w, int n) {
    for (int o = threadIdx.x; o < n; o += blockDim.x) taps[o] = (double)__ldg(w + o);
    __syncthreads();
}

// sum[j] = sum_o in(j + o) taps[o], o = 0 .. n-1 in order; get(i) is input i of the run
// (get(i) for i up to n - 1 + kRun is evaluated).
template <typename Get>
__device__ __forceinline__ void run_taps(const double* taps, int n, Get get, double (&sum)[kRun]) {
    double ring[kRun];
#pragma unroll
    for (int i = 0; i < kRun; ++i) {
        sum[i] = 0.0;
        ring[i] = (double)get(i);
    }
    for (int ob = 0; ob < n; ob += kRun) {
#pragma unroll
        for (int s = 0; s < kRun; ++s) {
            const int o = ob + s;
            if (o < n) {
                const double t = taps[o];
#pragma unroll
                for (int j = 0; j < kRun; ++j) sum[j] += ring[(s + j) % kRun] * t;
                ring[s] = (double)get(o + kRun); // input o leaves the run, input o + kRun enters
            }
        }
    }
}

// A row segment as staged: the inputs of kSegment outputs and what run_taps reads beyond.
__host__ __device__ inline int segment_floats(int radius) { return kSegment + 2 * radius + kRun + 1; }

size_t taps_bytes(int radius) { return (2 * (size_t)radius + 1) * sizeof(double); }
// 58 KB at radius 400, above which the segments of a row share their inputs
size_t rows_smem_bytes(int radius) {
    return taps_bytes(radius) + (size_t)kRowWarps * (segment_floats(radius) + kSegment) * sizeof(float);
}

// `count` inputs from sample q0 on of a row of `width`, reflected at its ends, asynchronously, by
// threads first, first + step, ...
__device__ __forceinline__ void stage_inputs(float* line, const float* row, int q0, int count, int width, int outputs,
                                             int radius, int first, int step) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(line);
    if (q0 >= 0 && q0 + count <= width) {
#pragma unroll 4
        for (int i = first; i < count; i += step)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d + 4u * (unsigned)i), "l"(row + q0 + i));
    } else {
        // what lies beyond the last output's inputs is not part of a sum that is kept
        const int last = outputs + 2 * radius;
        for (int i = first; i < count; i += step) {
            const int q = q0 + i;
            if (i < last)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d + 4u * (unsigned)i),
                             "l"(row + ((unsigned)q < (unsigned)width ? q : reflect_wide(q, width))));
            else
                line[i] = 0.0f;
        }
    }
    asm volatile("cp.async.commit_group;\n" ::);
}

// A warp's kSegment outputs of a row from its inputs at `in`, through its staging area `st`, to
// dst, of which `left` are inside the row.
__device__ __forceinline__ void segment_outputs(const double* taps, int n, const float* in, float* st, float* dst,
                                                int left, int lane) {
    if (lane * kRun < left) {
        double sum[kRun];
        run_taps(taps, n, [&](int i) { return in[lane * kRun + i]; }, sum);
#pragma unroll
        for (int j = 0; j < kRun; ++j) st[lane * kRun + j] = finite_d(sum[j]) ? (float)sum[j] : 0.0f;
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < kRun; ++i)
        if (i * 32 + lane < left) dst[i * 32 + lane] = st[i * 32 + lane];
}

// Horizontal pass (plane blockIdx.z): a warp stages the segment of a row, reflected at the
// row's ends, and its outputs leave through a staging area, so that the stores are coalesced.
__global__ void __launch_bounds__(32 * kRowWarps) blur_rows_run_kernel(const __grid_constant__ Planes in,
                                                                       const __grid_constant__ Planes out, int width,
                                                                       int height, const float* __restrict__ w,
                                                                       int radius) {
    extern __shared__ __align__(16) unsigned char post_smem[];
    double* taps = reinterpret_cast<double*>(post_smem);
    const int n = 2 * radius + 1, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int count = segment_floats(radius);
    float* line = reinterpret_cast<float*>(taps + n) + warp * (count + kSegment);
    float* st = line + count;
    const int x0 = blockIdx.x * kSegment, y = blockIdx.y * kRowWarps + warp;
    if (y < height)
        stage_inputs(line, in.p[blockIdx.z] + (size_t)y * width, x0 - radius, count, width, min(kSegment, width - x0),
                     radius, lane, 32);
    stage_taps(taps, w, n); // its barrier is the last one: warps go on by themselves
    if (y >= height) return;
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncwarp();
    segment_outputs(taps, n, line, st, out.p[blockIdx.z] + (size_t)y * width + x0, width - x0, lane);
}

// The same for large radii: the warps of a CTA take neighbouring segments of one row (blockIdx.x)
// and share its inputs, of which a segment by itself has more around it than in it. 1999x1333,
// three planes, a warp's own inputs and shared ones: radius 400 531 us both, 600 799 and 781,
// 1200 1684 and 1530, 2000, where the first leave room for eight warps per SM, 4230 and 2590.
constexpr int kSharedRadius = 400;
size_t shared_rows_smem_bytes(int radius, int warps) {
    return taps_bytes(radius) + ((size_t)segment_floats(radius) + (2 * (size_t)warps - 1) * kSegment) * sizeof(float);
}
__global__ void __launch_bounds__(32 * kRowWarps) blur_rows_shared_kernel(const __grid_constant__ Planes in,
                                                                          const __grid_constant__ Planes out, int width,
                                                                          int height, const float* __restrict__ w,
                                                                          int radius) {
    extern __shared__ __align__(16) unsigned char post_smem[];
    double* taps = reinterpret_cast<double*>(post_smem);
    const int n = 2 * radius + 1, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int count = segment_floats(radius) + (warps - 1) * kSegment;
    float* line = reinterpret_cast<float*>(taps + n);
    const int first = blockIdx.y * warps * kSegment, x0 = first + warp * kSegment;
    const size_t row = (size_t)blockIdx.x * width;
    stage_inputs(line, in.p[blockIdx.z] + row, first - radius, count, width, min(warps * kSegment, width - first), radius,
                 threadIdx.x, blockDim.x);
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    stage_taps(taps, w, n);
    if (x0 < width)
        segment_outputs(taps, n, line + warp * kSegment, line + count + warp * kSegment, out.p[blockIdx.z] + row + x0,
                        width - x0, lane);
}

// Vertical pass (plane blockIdx.z): a thread takes kRun rows of one column; the warp's
// loads are rows of 32 consecutive columns. The blurred value goes to `io`; with kUnsharp, `io`
// holds the plane and receives v + amount (v - blurred) in FP64; with kPairs it is a sum by pairs
// of columns and receives v + amount blurred.
enum ColumnsOut : int { kBlurred, kUnsharp, kPairs };
template <ColumnsOut kOut>
__global__ void __launch_bounds__(32 * kColWarps, 5) blur_cols_run_kernel(const __grid_constant__ Planes in,
                                                                       const __grid_constant__ Planes io, int width,
                                                                       int height, const float* __restrict__ w,
                                                                       int radius, float amount) {
    extern __shared__ __align__(16) unsigned char post_smem[];
    double* taps = reinterpret_cast<double*>(post_smem);
    const int n = 2 * radius + 1;
    stage_taps(taps, w, n);
    const int x = blockIdx.x * 32 + (threadIdx.x & 31);
    const int p0 = (blockIdx.y * kColWarps + (threadIdx.x >> 5)) * kRun;
    if (x >= width || p0 >= height) return;
    const float* src = in.p[blockIdx.z] + x;
    constexpr bool pairs = kOut == kPairs;
    float* dst = io.p[blockIdx.z] + (pairs ? ((size_t)(x >> 1) * lp::line_words(height) + p0) * 2 + (x & 1)
                                           : (size_t)p0 * width + x);
    const size_t step = pairs ? 2 : width;
    const int rows = min(kRun, height - p0);
    double sum[kRun];
    if (p0 >= radius && p0 - radius + n + kRun <= height) {
        const float* top = src + (size_t)(p0 - radius) * width;
        run_taps(taps, n, [&](int i) { return __ldg(top + (size_t)i * width); }, sum);
    } else {
        run_taps(taps, n, [&](int i) {
            const int q = p0 - radius + i;
            const int y = (unsigned)q < (unsigned)height ? q : reflect_wide(q, height);
            return __ldg(src + (size_t)y * width);
        }, sum);
    }
#pragma unroll
    for (int j = 0; j < kRun; ++j) {
        if (j >= rows) break;
        const float blurred = finite_d(sum[j]) ? (float)sum[j] : 0.0f;
        if constexpr (kOut == kUnsharp) {
            const double v = (double)dst[j * step];
            const double vb = (double)blurred;
            const double a = (double)amount;
            const double o = v + a * (v - vb);
            dst[j * step] = finite_d(o) ? (float)o : 0.0f;
        } else if constexpr (pairs) {
            dst[j * step] = fmaf(amount, blurred, dst[j * step]);
        } else {
            dst[j * step] = blurred;
        }
    }
}

dim3 plane_grid(int width, int height) { return dim3((width + 31) / 32, (height + 7) / 8); }

// Horizontal pass of `count` planes into `tmps`.
cudaError_t blur_rows(float* const* planes, float* const* tmps, int count, int width, int height, const float* w,
                      int radius, cudaStream_t stream) {
    Planes in{}, out{};
    for (int c = 0; c < count; ++c) {
        in.p[c] = planes[c];
        out.p[c] = tmps[c];
    }
    if (radius > kSharedRadius) {
        const int segments = (width + kSegment - 1) / kSegment, warps = std::min(segments, kRowWarps);
        const size_t smem = shared_rows_smem_bytes(radius, warps);
        const cudaError_t e = fjb::allow_dynamic_smem(blur_rows_shared_kernel, smem);
        if (e != cudaSuccess) return e;
        fjb::count_launch();
        blur_rows_shared_kernel<<<dim3(height, (segments + warps - 1) / warps, count), 32 * warps, smem, stream>>>(
            in, out, width, height, w, radius);
        return cudaGetLastError();
    }
    const size_t smem = rows_smem_bytes(radius);
    cudaError_t e = fjb::allow_dynamic_smem(blur_rows_run_kernel, smem);
    if (e != cudaSuccess) return e;
    fjb::count_launch();
    blur_rows_run_kernel<<<dim3((width + kSegment - 1) / kSegment, (height + kRowWarps - 1) / kRowWarps, count),
                           32 * kRowWarps, smem, stream>>>(in, out, width, height, w, radius);
    return cudaGetLastError();
}

template <ColumnsOut kOut>
cudaError_t blur_cols(float* const* planes, float* const* tmps, int count, int width, int height, const float* w,
                      int radius, float amount, cudaStream_t stream) {
    Planes in{}, io{};
    for (int c = 0; c < count; ++c) {
        in.p[c] = tmps[c];
        io.p[c] = planes[c];
    }
    const size_t smem = taps_bytes(radius); // 33 KB at the largest radius: no setting needed
    const int runs = (height + kRun - 1) / kRun;
    fjb::count_launch();
    blur_cols_run_kernel<kOut><<<dim3((width + 31) / 32, (runs + kColWarps - 1) / kColWarps, count), 32 * kColWarps,
                                 smem, stream>>>(in, io, width, height, w, radius, amount);
    return cudaGetLastError();
}

} // namespace

cudaError_t launch_glare(float* out, int width, int height, uint64_t seed, uint32_t medium, int origin_x,
                         int origin_y, float percent, float roughness, cudaStream_t stream) {
    if (width <= 0 || height <= 0) return cudaSuccess;
    fjb::count_launch();
    glare_kernel<<<plane_grid(width, height), dim3(32, 8), 0, stream>>>(out, width, height, seed, medium, origin_x,
                                                                       origin_y, percent, roughness);
    return cudaGetLastError();
}

cudaError_t launch_blur_planes(float* const* planes, float* const* tmps, int count, int width, int height,
                               const float* w, int radius, cudaStream_t stream) {
    if (width <= 0 || height <= 0 || radius <= 0 || !w || count <= 0) return cudaSuccess;
    if (count > 3) return cudaErrorInvalidValue;
    cudaError_t e = blur_rows(planes, tmps, count, width, height, w, radius, stream);
    if (e != cudaSuccess) return e;
    return blur_cols<kBlurred>(planes, tmps, count, width, height, w, radius, 0.0f, stream);
}

cudaError_t launch_unsharp_planes(float* const* planes, float* const* tmps, int count, int width, int height,
                                  const float* w, int radius, float amount, cudaStream_t stream) {
    if (width <= 0 || height <= 0 || radius <= 0 || !w || count <= 0) return cudaSuccess;
    if (count > 3) return cudaErrorInvalidValue;
    cudaError_t e = blur_rows(planes, tmps, count, width, height, w, radius, stream);
    if (e != cudaSuccess) return e;
    return blur_cols<kUnsharp>(planes, tmps, count, width, height, w, radius, amount, stream);
}

cudaError_t launch_blur_into_pairs(const float* const* planes, float* const* tmps, float* const* sums, int count,
                                   int width, int height, const float* w, int radius, float weight,
                                   cudaStream_t stream) {
    if (width <= 0 || height <= 0 || radius <= 0 || !w || count <= 0) return cudaSuccess;
    if (count > 3) return cudaErrorInvalidValue;
    float* in[3] = {};
    for (int c = 0; c < count; ++c) in[c] = const_cast<float*>(planes[c]); // read only
    cudaError_t e = blur_rows(in, tmps, count, width, height, w, radius, stream);
    if (e != cudaSuccess) return e;
    return blur_cols<kPairs>(sums, tmps, count, width, height, w, radius, weight, stream);
}

} // namespace fjb
