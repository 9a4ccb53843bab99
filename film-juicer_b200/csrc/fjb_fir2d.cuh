// fjb_fir2d.cuh -- short separable taps (radius 1..9), both axes in one pass.
//
// dst = sum_i weight_i columns_i(rows_i(src)) + src_weight src, each sum over taps in Acc
// precision and rounded to FP32 between the axes, half-sample reflection at the frame's
// edges. A CTA makes a 64 x 32 tile: the input with the widest halo goes to shared memory
// once, then for each set of taps every thread makes eight neighbouring row outputs from
// a register window (one shared-memory read per input instead of one per tap) and eight
// outputs of a column the same way. The result is stored by pairs of columns, each pair's
// samples of all rows together (fjb_line_pairs.cuh), 256 bytes at a time. One read and one
// write of a plane for all short Gaussians of a channel; as separate row and column passes
// each of them cost a plane written and read twice.
//
// What bounds it: FP32 sums, instruction issue and the barriers between the phases
// (3840x2160, three planes: 95 us for the scatter's Gaussians, 29 for the back-reflection's; two
// sums per packed instruction, in 76 registers, took 20 to 45 % longer); FP64 sums, the
// conversions between FP32 and FP64 (56 % of that unit) and the FP64 pipe (38 %): 147 us.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace fjb {
namespace fir {

constexpr int kMaxRadius = 9;
constexpr int kTileW = 64, kTileH = 32, kThreads = 256;
constexpr int kHalo = 12; // columns on each side: the widest halo in whole float4
constexpr int kInCols = kTileW + 2 * kHalo;
// Rows 4 banks apart (modulo 32): a quarter warp's 16-byte accesses to eight rows are
// conflict-free.
constexpr int kInPitch = kInCols + 4;
constexpr int kMidPitch = kTileW + 4;
static_assert(kInPitch % 32 == 28 && kMidPitch % 32 == 4, "eight rows in distinct banks");

constexpr int kMaxSets = 5;
struct Taps {
    float w[2 * kMaxRadius + 1]; // rows: tap o multiplies sample x + o - radius
    int radius;
    int flip_columns;            // columns: tap o multiplies sample y + radius - o
    float weight;
};
// One plane through the short Gaussians of its channel.
struct Job {
    const float* src;
    long long stride;
    float* dst;
    float src_weight;
    int count;
    Taps set[kMaxSets];
};
constexpr int kMaxJobs = 3;
struct Jobs {
    int width, height, count;
    int dst_pairs, dst_words; // pairs of columns of a result, words (row samples of a pair) of one
    Job job[kMaxJobs];
};

__device__ __forceinline__ int reflect(int i, int n) {
    if ((unsigned)i < (unsigned)n) return i;
    const int period = 2 * n;
    i %= period;
    if (i < 0) i += period;
    return i >= n ? period - 1 - i : i;
}

// FP64 sums that leave the finite range become 0, as the filters that use them ask for.
__device__ __forceinline__ float rounded(float v) { return v; }
__device__ __forceinline__ float rounded(double v) { return isfinite(v) ? (float)v : 0.0f; }

// The tile with a halo of `rad` rows and kHalo columns, asynchronously, all copies in flight
// at once: 16 bytes where the tile lies inside rows that are 16-byte aligned, else 4 bytes
// with the indexes reflected.
__device__ __forceinline__ void stage(const Jobs& P, const Job& J, int rad, float* in) {
    const int W = P.width, H = P.height;
    const int x0 = blockIdx.x * kTileW - kHalo, y0 = blockIdx.y * kTileH - rad;
    const int rows = kTileH + 2 * rad;
    const unsigned base = (unsigned)__cvta_generic_to_shared(in);
    if (x0 >= 0 && x0 + kInCols <= W && J.stride % 4 == 0 && (reinterpret_cast<uintptr_t>(J.src) & 15u) == 0) {
        for (int i = threadIdx.x; i < rows * (kInCols / 4); i += kThreads) {
            const int r = i / (kInCols / 4), c = i % (kInCols / 4) * 4;
            const float* src = J.src + (long long)reflect(y0 + r, H) * J.stride + x0 + c;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(base + 4u * (unsigned)(r * kInPitch + c)), "l"(src));
        }
    } else {
        for (int i = threadIdx.x; i < rows * kInCols; i += kThreads) {
            const int r = i / kInCols, c = i % kInCols;
            const float* src = J.src + (long long)reflect(y0 + r, H) * J.stride + reflect(x0 + c, W);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(base + 4u * (unsigned)(r * kInPitch + c)), "l"(src));
        }
    }
    asm volatile("cp.async.commit_group;\n" ::);
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}

// One set of taps on the staged tile (its first row is `rad` rows above the tile's): adds
// this thread's eight outputs, rows r .. r + 7 of column c.
template <typename Acc, int RAD>
__device__ __forceinline__ void taps(const Taps& T, int rad, const float* in, float* mid, float (&sum)[8]) {
    constexpr int kPad = (RAD + 3) / 4 * 4;
    constexpr int kRows = kTileH + 2 * RAD;
    Acc t[2 * RAD + 1];
#pragma unroll
    for (int o = 0; o <= 2 * RAD; ++o) t[o] = (Acc)T.w[o];
    __syncthreads();
    for (int task = threadIdx.x; task < kRows * (kTileW / 8); task += kThreads) {
        const int r = task % kRows, c = task / kRows * 8; // neighbouring lanes, neighbouring rows
        const float4* q = reinterpret_cast<const float4*>(in + (r + rad - RAD) * kInPitch + kHalo - kPad + c);
        Acc win[8 + 2 * kPad];
#pragma unroll
        for (int i = 0; i < (8 + 2 * kPad) / 4; ++i) {
            const float4 v = q[i];
            win[4 * i] = (Acc)v.x;
            win[4 * i + 1] = (Acc)v.y;
            win[4 * i + 2] = (Acc)v.z;
            win[4 * i + 3] = (Acc)v.w;
        }
        float o8[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            Acc s = 0;
#pragma unroll
            for (int o = 0; o <= 2 * RAD; ++o) s += win[kPad - RAD + j + o] * t[o];
            o8[j] = rounded(s);
        }
        float4* m = reinterpret_cast<float4*>(mid + r * kMidPitch + c);
        m[0] = make_float4(o8[0], o8[1], o8[2], o8[3]);
        m[1] = make_float4(o8[4], o8[5], o8[6], o8[7]);
    }
    __syncthreads();
    if (T.flip_columns) {
#pragma unroll
        for (int o = 0; o < RAD; ++o) {
            const Acc a = t[o];
            t[o] = t[2 * RAD - o];
            t[2 * RAD - o] = a;
        }
    }
    const float* col = mid + threadIdx.x / kTileW * 8 * kMidPitch + threadIdx.x % kTileW;
    Acc win[8 + 2 * RAD];
#pragma unroll
    for (int i = 0; i < 8 + 2 * RAD; ++i) win[i] = (Acc)col[i * kMidPitch];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        Acc s = 0;
#pragma unroll
        for (int o = 0; o <= 2 * RAD; ++o) s += win[j + o] * t[o];
        sum[j] = fmaf(T.weight, rounded(s), sum[j]);
    }
}

template <typename Acc>
__global__ void __launch_bounds__(kThreads, 3) kernel(const __grid_constant__ Jobs P) {
    __shared__ __align__(16) float in[(kTileH + 2 * kMaxRadius) * kInPitch];
    __shared__ __align__(16) float mid[(kTileH + 2 * kMaxRadius) * kMidPitch];
    const Job& J = P.job[blockIdx.z];
    int rad = 0;
    for (int i = 0; i < J.count; ++i) rad = max(rad, J.set[i].radius);
    stage(P, J, rad, in);
    __syncthreads();
    const int c = threadIdx.x % kTileW, r = threadIdx.x / kTileW * 8;
    float sum[8] = {};
#pragma unroll 1
    for (int i = 0; i < J.count; ++i) {
        const Taps& T = J.set[i];
        switch (T.radius) {
            case 1: taps<Acc, 1>(T, rad, in, mid, sum); break;
            case 2: taps<Acc, 2>(T, rad, in, mid, sum); break;
            case 3: taps<Acc, 3>(T, rad, in, mid, sum); break;
            case 4: taps<Acc, 4>(T, rad, in, mid, sum); break;
            case 5: taps<Acc, 5>(T, rad, in, mid, sum); break;
            case 6: taps<Acc, 6>(T, rad, in, mid, sum); break;
            case 7: taps<Acc, 7>(T, rad, in, mid, sum); break;
            case 8: taps<Acc, 8>(T, rad, in, mid, sum); break;
            default: taps<Acc, 9>(T, rad, in, mid, sum); break;
        }
    }
    // the source's own share last: it is the largest term as a rule
    if (J.src_weight != 0.0f)
#pragma unroll
        for (int j = 0; j < 8; ++j) sum[j] = fmaf(J.src_weight, in[(rad + r + j) * kInPitch + kHalo + c], sum[j]);
    // transposed through shared memory: a warp stores 32 rows of a pair of columns
    constexpr int kPitch = kTileH + 1;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 8; ++j) mid[c * kPitch + r + j] = sum[j];
    __syncthreads();
    const int lane = threadIdx.x & 31, y = blockIdx.y * kTileH + lane;
    float2* dst = reinterpret_cast<float2*>(J.dst);
#pragma unroll
    for (int p = threadIdx.x >> 5; p < kTileW / 2; p += kThreads / 32) {
        const int pair = blockIdx.x * (kTileW / 2) + p;
        if (pair < P.dst_pairs && y < P.height)
            dst[(size_t)pair * P.dst_words + y] = make_float2(mid[2 * p * kPitch + lane], mid[(2 * p + 1) * kPitch + lane]);
    }
}

inline dim3 grid(const Jobs& P) {
    return dim3((P.width + kTileW - 1) / kTileW, (P.height + kTileH - 1) / kTileH, P.count);
}

} // namespace fir
} // namespace fjb
