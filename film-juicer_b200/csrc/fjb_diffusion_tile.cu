// fjb_diffusion_tile.cu -- diffusion (a17) as an FFT convolution of tiles, radius 8 to 40.
//
// Same result as the other forms up to FP32 rounding (fjb_diffusion.cu, which states the
// semantics, and fjb_diffusion_fft.cu): a 128 x 128 tile of the reflect-extended frame
// convolved circularly with the PSF equals the linear convolution on its inner
// (128 - 2 r)^2 samples. A CTA takes two tiles of a channel as the real and the imaginary
// part of one complex tile -- the PSF is real and even, so its spectrum is real and the two
// stay apart -- and runs the whole convolution in shared memory, so a plane is read and
// written once.
//
// 1024 threads hold 16 complex values each. 128 = 16 x 8 along both axes: a radix-16 pass, a
// twiddle and a radix-8 pass, every pass in place (decimation in frequency forward, in time
// backward, so the spectrum stays permuted and nothing is reordered); the last forward
// pass, the product with the spectrum and the first backward pass share their registers.
// Rows are 136 words apart and their words swizzled so that every access is conflict-free.
//
// What bounds it: shared-memory bandwidth, twelve 128 KB sweeps a tile pair (about 14 000
// cycles), beside about 1500 instructions per thread (12 000 cycles per scheduler). The form
// over whole rows and columns of the frame moved its row spectra through memory three times
// (0.7 GB at 3840x2160, 780 us, and 185 us for the PSF's spectrum of a new frame size; here 233 us and 10 us). The
// inner share of a tile falls with the radius, (128 - 2 r)^2 / 128^2.
#include <cuda_runtime.h>

#include <cmath>

#include "fjb_diffusion.h"
#include "fjb_launches.h"
#include "fjb_packed.cuh"

namespace fjb {

namespace {

constexpr int N = kDiffusionTile;
constexpr int kPitch = N + 8;
constexpr int kThreads = 1024;
constexpr size_t kSmem = ((size_t)N * kPitch + N) * sizeof(float2); // the tile, the twiddles

__device__ __forceinline__ int reflect_whole(int i, int n) {
    if ((unsigned)i < (unsigned)n) return i;
    if (n <= 1) return 0;
    const int period = 2 * (n - 1);
    int v = i % period;
    if (v < 0) v += period;
    return v < n ? v : period - v;
}

struct TilePass {
    int width, height, radius, tiles_x, tiles; // tiles of one channel
    int ahead;                                 // CTAs between a CTA and the one after it
    float fraction;
    const float* spectrum; // per channel N x N reals, permuted as the tile is, scaled by 1 / N^2
    float* out;            // spectrum build
    const float* src[3];
    float* dst[3];
    long long stride;
    const float* psf[3]; // spectrum build: rows |dy| = 0..r, taps each
    int taps;
    float2 tw[N]; // exp(-2 pi i k / N)
};

__device__ __forceinline__ Pair cmul(Pair a, float wr, float wi) {
    const float2 f = unpack(a);
    return pack(f.x * wr - f.y * wi, f.x * wi + f.y * wr);
}
// times -i (forward) or i (inverse)
template <bool kInv>
__device__ __forceinline__ Pair rot(Pair a) {
    const float2 f = unpack(a);
    return kInv ? pack(-f.y, f.x) : pack(f.y, -f.x);
}

template <bool kInv>
__device__ __forceinline__ void dft4(Pair& a, Pair& b, Pair& c, Pair& d) {
    const Pair s = add2(a, c), t = sub2(a, c), u = add2(b, d), v = rot<kInv>(sub2(b, d));
    a = add2(s, u);
    b = add2(t, v);
    c = sub2(s, u);
    d = sub2(t, v);
}

// v[k] = sum_n v[n] exp(-+ 2 pi i n k / 8)
template <bool kInv>
__device__ __forceinline__ void dft8(Pair (&v)[8]) {
    constexpr float h = 0.70710678118654752440f;
    // n = 2 a + b: four-point transforms over a, then the pairs
    dft4<kInv>(v[0], v[2], v[4], v[6]);
    dft4<kInv>(v[1], v[3], v[5], v[7]);
    const Pair o1 = cmul(v[3], h, kInv ? h : -h), o2 = rot<kInv>(v[5]), o3 = cmul(v[7], -h, kInv ? h : -h);
    const Pair e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1];
    v[0] = add2(e0, o0);
    v[4] = sub2(e0, o0);
    v[1] = add2(e1, o1);
    v[5] = sub2(e1, o1);
    v[2] = add2(e2, o2);
    v[6] = sub2(e2, o2);
    v[3] = add2(e3, o3);
    v[7] = sub2(e3, o3);
}

// v[k] = sum_n v[n] exp(-+ 2 pi i n k / 16)
template <bool kInv>
__device__ __forceinline__ void dft16(Pair (&v)[16]) {
    constexpr float c1 = 0.92387953251128675613f, s1 = 0.38268343236508977173f, h = 0.70710678118654752440f;
    // n = 4 a + b: over a, twiddle exp(-+ 2 pi i b c / 16), then over b to k = c + 4 d
#pragma unroll
    for (int b = 0; b < 4; ++b) dft4<kInv>(v[b], v[4 + b], v[8 + b], v[12 + b]);
    constexpr float S = kInv ? 1.0f : -1.0f;
    v[5] = cmul(v[5], c1, S * s1);     // b c = 1
    v[6] = cmul(v[6], h, S * h);       // 2
    v[7] = cmul(v[7], s1, S * c1);     // 3
    v[9] = cmul(v[9], h, S * h);       // 2
    v[10] = rot<kInv>(v[10]);          // 4
    v[11] = cmul(v[11], -h, S * h);    // 6
    v[13] = cmul(v[13], s1, S * c1);   // 3
    v[14] = cmul(v[14], -h, S * h);    // 6
    v[15] = cmul(v[15], -c1, -S * s1); // 9
#pragma unroll
    for (int c = 0; c < 4; ++c) dft4<kInv>(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
    // v[4 c + d] holds k = c + 4 d
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int d = c + 1; d < 4; ++d) {
            const Pair t = v[4 * c + d];
            v[4 * c + d] = v[4 * d + c];
            v[4 * d + c] = t;
        }
}

// Word of row y that holds the j-th of eight values of group k (of 16).
__device__ __forceinline__ int word(int y, int k, int j) { return y * kPitch + k * 8 + (j ^ ((k >> 1) & 7)); }

// The tile's rows after the radix-16 pass of the loading thread (row y, n2): v[k1].
__device__ __forceinline__ void rows_out(Pair (&v)[16], Pair* z, const float2* tw, int y, int n2) {
    dft16<false>(v);
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        const float2 w = tw[n2 * k];
        z[word(y, k, n2)] = k == 0 ? v[0] : cmul(v[k], w.x, w.y);
    }
}

// Second forward row pass and both column passes up to the spectrum: afterwards this
// thread's column p holds rows (k1, j) = k1 * 8 + j for k1 = g and g + 8 in `a` and `b`.
__device__ __forceinline__ void forward(Pair* z, const float2* twc, int t, Pair (&a)[8], Pair (&b)[8]) {
    __syncthreads();
    {
        const int k = t & 15, y = t >> 4;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            Pair v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = z[word(y + 64 * i, k, j)];
            dft8<false>(v);
#pragma unroll
            for (int j = 0; j < 8; ++j) z[word(y + 64 * i, k, j)] = v[j];
        }
    }
    __syncthreads();
    Pair* col = z + (t & 127);
    const int g = t >> 7;
    {
        Pair v[16];
#pragma unroll
        for (int n = 0; n < 16; ++n) v[n] = col[(n * 8 + g) * kPitch];
        dft16<false>(v);
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const float2 w = twc[g * k];
            col[(k * 8 + g) * kPitch] = k == 0 ? v[0] : cmul(v[k], w.x, w.y);
        }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        a[j] = col[(g * 8 + j) * kPitch];
        b[j] = col[((g + 8) * 8 + j) * kPitch];
    }
    dft8<false>(a);
    dft8<false>(b);
}

__global__ void __launch_bounds__(kThreads, 1) tile_spectrum_kernel(const __grid_constant__ TilePass P) {
    extern __shared__ __align__(16) unsigned char sm[];
    Pair* z = reinterpret_cast<Pair*>(sm);
    float2* tw = reinterpret_cast<float2*>(z + N * kPitch);
    const int t = threadIdx.x, ch = blockIdx.x, r = P.radius;
    if (t < N) tw[t] = P.tw[t];
    __syncthreads();
    const int y = t >> 3, n2 = t & 7;
    // the PSF around the origin of the circular tile
    const int dy = y < N / 2 ? y : y - N;
    Pair v[16];
#pragma unroll
    for (int n = 0; n < 16; ++n) {
        const int x = n * 8 + n2, dx = x < N / 2 ? x : x - N;
        const bool in = dy >= -r && dy <= r && dx >= -r && dx <= r;
        v[n] = pack(in ? P.psf[ch][(size_t)(dy < 0 ? -dy : dy) * P.taps + dx + r] : 0.0f, 0.0f);
    }
    rows_out(v, z, tw, y, n2);
    Pair a[8], b[8];
    forward(z, P.tw, t, a, b);
    float* out = P.out + (size_t)ch * N * N + (t & 127);
    const int g = t >> 7;
    constexpr float scale = 1.0f / ((float)N * (float)N);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        out[(g * 8 + j) * N] = unpack(a[j]).x * scale;
        out[((g + 8) * 8 + j) * N] = unpack(b[j]).x * scale;
    }
}

__global__ void __launch_bounds__(kThreads, 1) tile_kernel(const __grid_constant__ TilePass P) {
    extern __shared__ __align__(16) unsigned char sm[];
    Pair* z = reinterpret_cast<Pair*>(sm);
    float2* tw = reinterpret_cast<float2*>(z + N * kPitch);
    const int t = threadIdx.x, ch = blockIdx.y, r = P.radius, inner = N - 2 * r;
    const int W = P.width, H = P.height;
    if (t < N) tw[t] = P.tw[t];
    const float* src = P.src[ch];
    // the two tiles' first extended samples
    int x0[2], y0[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int tile = min(2 * (int)blockIdx.x + i, P.tiles - 1);
        y0[i] = tile / P.tiles_x * inner - r;
        x0[i] = tile % P.tiles_x * inner - r;
    }
    const bool second = 2 * (int)blockIdx.x + 1 < P.tiles;
    {
        // what the CTA after this one loads, into L2: a 128-byte line per thread
        const int tile = 2 * (blockIdx.x + P.ahead) + (t >> 9);
        if (tile < P.tiles) {
            const int yy = tile / P.tiles_x * inner - r + ((t >> 2) & 127), xx = tile % P.tiles_x * inner - r + 32 * (t & 3);
            if (yy >= 0 && yy < H && xx >= 0 && xx < W)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(src + (long long)yy * P.stride + xx));
        }
    }
    const int y = t >> 3, n2 = t & 7;
    {
        float f[2][16];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float* row = src + (long long)reflect_whole(y0[i] + y, H) * P.stride;
            if (x0[i] >= 0 && x0[i] + N <= W) {
#pragma unroll
                for (int n = 0; n < 16; ++n) f[i][n] = row[x0[i] + n * 8 + n2];
            } else {
#pragma unroll
                for (int n = 0; n < 16; ++n) f[i][n] = row[reflect_whole(x0[i] + n * 8 + n2, W)];
            }
        }
        __syncthreads(); // the twiddles
        Pair v[16];
#pragma unroll
        for (int n = 0; n < 16; ++n) v[n] = pack(f[0][n], second ? f[1][n] : 0.0f);
        rows_out(v, z, tw, y, n2);
    }
    Pair* col = z + (t & 127);
    const int g = t >> 7;
    {
        Pair a[8], b[8];
        const float* spec = P.spectrum + (size_t)ch * N * N + (t & 127);
        forward(z, P.tw, t, a, b);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float sa = __ldg(spec + (g * 8 + j) * N), sb = __ldg(spec + ((g + 8) * 8 + j) * N);
            a[j] = mul2(a[j], pack(sa, sa));
            b[j] = mul2(b[j], pack(sb, sb));
        }
        dft8<true>(a);
        dft8<true>(b);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            col[(g * 8 + j) * kPitch] = a[j];
            col[((g + 8) * 8 + j) * kPitch] = b[j];
        }
    }
    __syncthreads();
    {
        Pair v[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const float2 w = P.tw[g * k];
            const Pair q = col[(k * 8 + g) * kPitch];
            v[k] = k == 0 ? q : cmul(q, w.x, -w.y);
        }
        dft16<true>(v);
#pragma unroll
        for (int n = 0; n < 16; ++n) col[(n * 8 + g) * kPitch] = v[n];
    }
    __syncthreads();
    // from here on only the inner rows are needed
    {
        const int k = t & 15;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int yy = (t >> 4) + 64 * i;
            if (yy >= r && yy < N - r) {
                Pair v[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = z[word(yy, k, j)];
                dft8<true>(v);
#pragma unroll
                for (int j = 0; j < 8; ++j) z[word(yy, k, j)] = v[j];
            }
        }
    }
    __syncthreads();
    if (y < r || y >= N - r) return;
    Pair v[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        const float2 w = tw[n2 * k];
        const Pair q = z[word(y, k, n2)];
        v[k] = k == 0 ? q : cmul(q, w.x, -w.y);
    }
    dft16<true>(v);
    const float f = P.fraction;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int yy = y0[i] + y;
        if (yy >= H || (i == 1 && !second)) continue;
        const float* cur = src + (long long)yy * P.stride + x0[i];
        float* out = P.dst[ch] + (long long)yy * P.stride + x0[i];
#pragma unroll
        for (int n = 0; n < 16; ++n) {
            const int x = n * 8 + n2;
            if (x < r || x >= N - r || x0[i] + x >= W) continue;
            const float2 c = unpack(v[n]);
            out[x] = (1.0f - f) * cur[x] + f * (i == 0 ? c.x : c.y);
        }
    }
}

void fill(TilePass& T, const DiffusionFftPlan& p) {
    T.width = p.width;
    T.height = p.height;
    T.radius = p.radius;
    const int inner = N - 2 * p.radius;
    T.tiles_x = (p.width + inner - 1) / inner;
    T.tiles = T.tiles_x * ((p.height + inner - 1) / inner);
    for (int k = 0; k < N; ++k) {
        const double a = -2.0 * 3.14159265358979323846 * (double)k / (double)N;
        T.tw[k] = make_float2((float)std::cos(a), (float)std::sin(a));
    }
}

} // namespace

cudaError_t launch_diffusion_tile_spectrum(const DiffusionFftPlan& p, const float* const psf_rows[3], int taps,
                                           float* spectrum, cudaStream_t stream) {
    TilePass T{};
    fill(T, p);
    T.out = spectrum;
    T.taps = taps;
    for (int c = 0; c < 3; ++c) T.psf[c] = psf_rows[c];
    cudaError_t e = cudaFuncSetAttribute(tile_spectrum_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
    if (e != cudaSuccess) return e;
    fjb::count_launch();
    tile_spectrum_kernel<<<3, kThreads, kSmem, stream>>>(T);
    return cudaGetLastError();
}

cudaError_t launch_diffusion_tile(const DiffusionFftPlan& p, const float* spectrum, float fraction, float* dst[3],
                                  const float* src[3], long long stride, cudaStream_t stream) {
    TilePass T{};
    fill(T, p);
    T.spectrum = spectrum;
    T.fraction = fraction;
    T.stride = stride;
    for (int c = 0; c < 3; ++c) {
        T.src[c] = src[c];
        T.dst[c] = dst[c];
    }
    int device = 0;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&T.ahead, cudaDevAttrMultiProcessorCount, device);
    cudaError_t e = cudaFuncSetAttribute(tile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
    if (e != cudaSuccess) return e;
    fjb::count_launch();
    tile_kernel<<<dim3((T.tiles + 1) / 2, 3), kThreads, kSmem, stream>>>(T);
    return cudaGetLastError();
}

} // namespace fjb
