// fjb_grain.cu -- density-space visual grain (a15).
//
// Per CMY channel the grain is the sum over up to three particle-size scales (fine,
// mid, coarse) of a correlated delta: a Poisson particle sample per pixel (one
// layer, or the three emulsion sublayers, each optionally blurred by its dye-cloud
// Gaussian) minus the developed density, blurred by the scale's correlation
// Gaussian and weighted; a shared (chroma-correlated) delta may be mixed in; the
// result is added back to the density planes in place.
//
// Arithmetic restates the reference's grain path so that results are bit-identical:
//   random draws     src/Cuda/Film/JuicerCudaFilmPipeline.cu:1892-1995 (static blue
//                    noise lookups keyed by splitmix64 of the draw index, or the
//                    Philox4x32-10 counter stream of third_party/openrand/philox.h)
//   Poisson / model  :1997-2075 (product-of-uniforms below lambda 10, rounded normal
//                    above; saturating particle count)
//   Wang offsets     :1674-1775, value noise / breathing / clump :1777-1890
//   frame uniforms   :2174-2352
//   layer lookup     :2077-2171
//   sample kernels   :2579-2986 (simple, one layer, layer triplet)
//   schedule, blurs  src/Cuda/Scan/JuicerCudaScanPipeline.cu:3141-3740, :317-380,
//                    :454-578, :705-775 (FMA chains in tap order, half-sample
//                    reflection, sanitising stores)
// The float contractions the reference's compiler forms (a + b * c -> fma) are
// written out as explicit __fmaf_rn here so that they do not depend on this
// compiler's choices. The layout is this project's: fewer passes (sample and
// accumulate/delta fused, the gain folded into the last weighted pass, mix and
// reconstruction in one pass) and taps passed as kernel parameters.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "fjb_grain.h"
#include "fjb_launches.h"
#include "fjb_philox.cuh"

namespace fjb {

namespace {

constexpr float kTwoPi = 6.28318530717958647692f;
constexpr float kInvU32 = 1.0f / 4294967296.0f;

__device__ __forceinline__ bool finite(float v) { return isfinite(v); }
__device__ __forceinline__ float sanitize(float v) { return isfinite(v) ? v : 0.0f; }
__device__ __forceinline__ float clamp01(float v, float lo, float hi) { return fminf(fmaxf(v, lo), hi); }

__device__ __forceinline__ uint64_t splitmix64(uint64_t v) {
    v += 0x9E3779B97F4A7C15ULL;
    v = (v ^ (v >> 30)) * 0xBF58476D1CE4E5B9ULL;
    v = (v ^ (v >> 27)) * 0x94D049BB133111EBULL;
    return v ^ (v >> 31);
}

__device__ __forceinline__ int wrap_coordinate(int64_t c, int size) {
    if (size <= 0) return 0;
    if ((size & (size - 1)) == 0) return (int)((uint64_t)c & (uint64_t)(size - 1));
    c %= (int64_t)size;
    if (c < 0) c += size;
    return (int)c;
}

__device__ __forceinline__ float smoothstep(float t) { return (t * t) * __fmaf_rn(-2.0f, t, 3.0f); }

__device__ __forceinline__ float hash01(int x, int y, uint64_t seed) {
    const uint64_t h = splitmix64(seed ^ ((uint64_t)x * 0x9E3779B97F4A7C15ULL) ^ ((uint64_t)y * 0xBF58476D1CE4E5B9ULL));
    return (float)(uint32_t)(h & 0xFFFFFFFFu) * kInvU32;
}

__device__ __forceinline__ float spatial_hash01(int x, int y, uint64_t seed) {
    const uint32_t lo = (uint32_t)seed, hi = (uint32_t)(seed >> 32);
    uint32_t h = lo ^ ((hi << 16) | (hi >> 16));
    h ^= (uint32_t)x * 0x9E3779B9u;
    h ^= (uint32_t)y * 0x85EBCA6Bu;
    h ^= h >> 16;
    h *= 0x7FEB352Du;
    h ^= h >> 15;
    h *= 0x846CA68Bu;
    h ^= h >> 16;
    return (float)h * kInvU32;
}

__device__ __forceinline__ uint32_t hash_u32(int x, int y, uint64_t seed, uint64_t salt) {
    const uint64_t h =
        splitmix64(seed ^ salt ^ ((uint64_t)x * 0x9E3779B97F4A7C15ULL) ^ ((uint64_t)y * 0xBF58476D1CE4E5B9ULL));
    return (uint32_t)(h & 0xFFFFFFFFu);
}

// A coordinate of a value-noise lattice: the cell and the smoothed position in it.
struct NoiseAxis {
    int i;
    float s;
};
__device__ __forceinline__ NoiseAxis noise_axis(float c) {
    const int i = (int)floorf(c);
    return {i, smoothstep(c - (float)i)};
}

// Value noise between the corners of a cell.
template <typename Corner>
__device__ __forceinline__ float value_noise(const NoiseAxis& x, const NoiseAxis& y, Corner corner) {
    const float v00 = corner(x.i, y.i);
    const float v10 = corner(x.i + 1, y.i);
    const float v01 = corner(x.i, y.i + 1);
    const float v11 = corner(x.i + 1, y.i + 1);
    const float v0 = __fmaf_rn(v10 - v00, x.s, v00);
    const float v1 = __fmaf_rn(v11 - v01, x.s, v01);
    return __fmaf_rn(v1 - v0, y.s, v0);
}

constexpr uint32_t kPhiloxGlobalSeed = 0xAAAAAAAAu;

// What a block of the sample kernel prepares for its pixels.
//
// The kernel is bound by integer instruction issue, and most of it was the same for many
// pixels: the blue-noise offsets of draw d hash the pass's seed and d alone; a blue-noise
// uniform has 256 values, so the normal's radius and cosine do too; Wang cells and noise
// lattice cells cover many pixels; coordinates (divisions and 64-bit conversions) depend on
// the column or the row. The block evaluates each once, with the functions the pixels would
// call, so the results keep their bits. 3840x2160, one pass of three sublayers: 2880 -> 1190
// instructions per warp of pixels, 857 -> 459 us. What is left waits on the scattered
// blue-noise bytes (the Wang shift differs from pixel to pixel) as much as on issue.
constexpr int kSampleColumns = 32, kSampleRows = 8;
constexpr int kSampleThreads = kSampleColumns * kSampleRows;
static_assert(kSampleThreads == 256, "one thread per value of a noise byte and sample of the axis");
constexpr int kBlockRows = 8 * kSampleRows; // rows of pixels of a tile, at most
constexpr int kTableDraws = 32; // a Poisson count of a mean below 10 draws rarely more
constexpr int kWangCells = kSampleThreads;
constexpr int kSampleBlocks = 3; // per SM (2: 586 us; 4, in 64 registers: 495; 3: 459)

// Value-noise fields and the coordinates they are read at: breathing at its small and its
// large cells with two seeds each, and the two uniforms of the clump normal.
constexpr int kNoiseCoords = 4; // breathing small, breathing large, clump, clump (shifted)
constexpr int kNoiseFields = 6; // small a, b, large a, b, clump, clump (shifted)
__host__ __device__ constexpr int noise_coord(int field) { return field < 4 ? field >> 1 : field - 2; }
constexpr int kLattice = 192; // corners held of a field: cells are at least 4 pixels wide

struct NoiseField {
    uint64_t seed;
    int x0, y0, nx, ny; // lattice corners held (nx 0: none)
};

struct WangRow {
    int cell, near, far; // row of cells held, rows of the tile
};

struct GrainTables {
    GrainFrameUniforms u;
    uint32_t draws[2][3][kTableDraws]; // [frame, next frame][sublayer][draw]: low word of the hash
    float radius[256], cosine[256];    // sqrt(-2 ln u), cos(2 pi u) of the noise byte's uniform u
    float axis[256];                   // layer lookup axis, in lookup sign
    const uint8_t* frame_base[2];      // the blue-noise frame's first row
    size_t frame_row[2];
    int64_t pitch_offset[2];
    NoiseField field[kNoiseFields];
    float lattice[kNoiseFields][kLattice];
    NoiseAxis row[kNoiseCoords][kBlockRows];
    int wang_tile[kWangCells];
    WangRow wang_row[kBlockRows];
    int64_t wang_x; // first column of cells
    int wang_nx;    // columns held (0: none)
};

__device__ __forceinline__ uint32_t draw_hash(uint64_t seed, uint32_t d) {
    return (uint32_t)splitmix64(seed + (uint64_t)d * 0x9E3779B97F4A7C15ULL);
}

// (v + 1/2) / 256, all steps exact
__device__ __forceinline__ float noise_uniform(uint32_t v) {
    return __uint_as_float(0x3f800000u + (v << 15)) - (1.0f - 0.5f / 256.0f);
}

// sqrt(-2 ln u1) and cos(2 pi u2) of the Box-Muller normal
__device__ __forceinline__ float normal_radius(float u1) {
    u1 = clamp01(u1, 1e-7f, 1.0f);
    return sqrtf(-2.0f * logf(u1));
}
__device__ __forceinline__ float normal_cosine(float u2) { return cosf(kTwoPi * u2); }

struct PixelContext {
    uint64_t ax, ay;
    int use_stbn, wang_x, wang_y;
    float breathing, clump;
    bool retime;
    float time_alpha;
};

// Where a pass's blue-noise draws fall for a pixel: the table is a power of two on both sides,
// so the masked coordinate keeps only low bits of the 64-bit sum, which the 32-bit sum of the
// addends' low words already has.
struct NoisePlace {
    const uint8_t* frame; // its first row
    uint32_t width, mask_x, mask_y, x, y;
    __device__ __forceinline__ uint32_t byte(uint32_t h) const {
        const uint32_t u = (x + (h & 0xFFFFu)) & mask_x, v = (y + (h >> 16)) & mask_y;
        return __ldg(frame + ((size_t)v * (size_t)width + u));
    }
};

// The low word of the hash of draw d of the pass's `seed`. `draws`: its table, or null.
__device__ __forceinline__ uint32_t draw_word(const uint32_t* draws, uint64_t seed, uint32_t d) {
    return draws && d < (uint32_t)kTableDraws ? draws[d] : draw_hash(seed, d);
}

constexpr int kStbnBatch = 4;

// Poisson count of a mean below 10: a product of uniforms. The draws are fetched kStbnBatch
// at a time: the blue-noise addresses do not depend on earlier draws, so the table loads
// overlap instead of paying one cache latency per draw.
__device__ __forceinline__ int poisson_product(float lambda, const uint32_t* draws, uint64_t seed, const uint8_t* frame,
                                            uint32_t width, uint32_t mask_x, uint32_t mask_y, uint32_t x, uint32_t y) {
    const NoisePlace at{frame, width, mask_x, mask_y, x, y};
    const float L = expf(-lambda);
    float p = 1.0f;
    int k = 0;
    while (p > L && k < 1024) {
        uint32_t v[kStbnBatch];
#pragma unroll
        for (int j = 0; j < kStbnBatch; ++j) v[j] = at.byte(draw_word(draws, seed, (uint32_t)(k + j)));
        int used = 0;
#pragma unroll
        for (int j = 0; j < kStbnBatch; ++j) {
            if (p > L && k + used < 1024) {
                ++used;
                p *= noise_uniform(v[j]); // within the draws' clamp to [1e-7, 1]
            }
        }
        k += used;
    }
    return k - 1;
}

// Poisson count of a normal deviate z (means of 10 and more).
__device__ __forceinline__ int poisson_normal(float lambda, float z) {
    float s = __fmaf_rn(sqrtf(lambda), z, lambda);
    if (!finite(s)) s = 0.0f;
    int k = (int)floorf(s + 0.5f);
    return k < 0 ? 0 : k;
}

// Poisson count with uniforms from `uniform`, lambda > 0.
template <typename Uniform>
__device__ __forceinline__ int poisson_stream(float lambda, Uniform uniform) {
    if (lambda < 10.0f) {
        const float L = expf(-lambda);
        float p = 1.0f;
        int k = 0;
        while (p > L && k < 1024) {
            ++k;
            p *= clamp01(uniform(), 1e-7f, 1.0f);
        }
        return k - 1;
    }
    const float r = normal_radius(uniform());
    return poisson_normal(lambda, r * normal_cosine(uniform()));
}

// The counter stream (no blue noise).
__device__ __noinline__ int poisson_philox(float lambda, uint64_t seed, uint32_t ax, uint32_t ay) {
    Philox philox(seed, ax, kPhiloxGlobalSeed, ay);
    // u01: x * 2^-32 + 2^-33 (the product is exact, so the fma is too)
    return poisson_stream(lambda, [&]() {
        return __fmaf_rn((float)philox.next(), 1.0f / 4294967296.0f, 0.5f / 4294967296.0f);
    });
}

// Blue-noise tables of other sizes.
__device__ __noinline__ int poisson_wrapped(float lambda, uint64_t seed, const GrainFrame* f, const GrainTables* t,
                                            int frame, uint64_t ax, uint64_t ay, int wang_x, int wang_y) {
    uint32_t d = 0;
    return poisson_stream(lambda, [&]() {
        const uint32_t h = draw_hash(seed, d++);
        const int ox = (int)(h & 0xFFFFu) + wang_x;
        const int oy = (int)(h >> 16) + wang_y;
        const int64_t xc = (int64_t)ax + (int64_t)ox + (int64_t)f->stbn_offset_x;
        const int64_t yc = (int64_t)ay + (int64_t)oy + (int64_t)f->stbn_offset_y + t->pitch_offset[frame];
        const int x = wrap_coordinate(xc, f->stbn_w);
        const int y = wrap_coordinate(yc, f->stbn_h);
        return noise_uniform(__ldg(f->stbn + ((t->frame_row[frame] + (size_t)y) * (size_t)f->stbn_w + (size_t)x)));
    });
}

struct ParticleSample {
    float density, density_max, n_particles, od_particle, uniformity;
};

// `slot`: the sublayer's place in the draw tables (beyond them the draws are hashed here).
__device__ __forceinline__ float particle_model(const GrainFrame* f, const GrainTables* t, const ParticleSample& s,
                                                const PixelContext& px, int slot, int frame, uint64_t seed) {
    float density = s.density;
    if (!finite(density) || density < 0.0f) density = 0.0f;
    float p = density / s.density_max;
    p = clamp01(p, 1e-6f, 1.0f - 1e-6f);
    const float u = finite(s.uniformity) ? clamp01(s.uniformity, 0.0f, 1.0f) : 0.0f;
    float sat = __fmaf_rn(-(p * u), 1.0f - 1e-6f, 1.0f);
    if (!finite(sat) || sat <= 0.0f) sat = 1e-6f;
    const float lambda = s.n_particles / sat * p;
    int count = 0;
    if (finite(lambda) && lambda > 0.0f) {
        const bool pow2 = (f->stbn_w & (f->stbn_w - 1)) == 0 && (f->stbn_h & (f->stbn_h - 1)) == 0;
        if (!px.use_stbn) {
            count = poisson_philox(lambda, seed, (uint32_t)px.ax, (uint32_t)px.ay);
        } else if (!pow2) {
            count = poisson_wrapped(lambda, seed, f, t, frame, px.ax, px.ay, px.wang_x, px.wang_y);
        } else {
            const uint32_t* draws = slot < 3 ? t->draws[frame][slot] : nullptr;
            const NoisePlace at{t->frame_base[frame],
                                (uint32_t)f->stbn_w,
                                (uint32_t)f->stbn_w - 1,
                                (uint32_t)f->stbn_h - 1,
                                (uint32_t)px.ax + (uint32_t)px.wang_x + (uint32_t)f->stbn_offset_x,
                                (uint32_t)px.ay + (uint32_t)px.wang_y + (uint32_t)f->stbn_offset_y +
                                    (uint32_t)t->pitch_offset[frame]};
            if (lambda < 10.0f) {
                count = poisson_product(lambda, draws, seed, at.frame, at.width, at.mask_x, at.mask_y, at.x, at.y);
            } else {
                const uint32_t v1 = at.byte(draw_word(draws, seed, 0)), v2 = at.byte(draw_word(draws, seed, 1));
                count = poisson_normal(lambda, t->radius[v1] * t->cosine[v2]);
            }
        }
    }
    return sanitize((float)count * s.od_particle * sat);
}

// Particle samples of one sublayer in this frame and the next, modulated and retimed.
__device__ __forceinline__ float blend_frames(const PixelContext& px, float density, float g, float gn) {
    g = __fmaf_rn((g - density) * px.breathing, px.clump, density);
    if (px.retime) {
        gn = __fmaf_rn((gn - density) * px.breathing, px.clump, density);
        const float d0 = g - density, d1 = gn - density;
        const float blend = __fmaf_rn(d1 - d0, px.time_alpha, d0);
        const float w0 = 1.0f - px.time_alpha;
        const float den = __fmaf_rn(w0, w0, px.time_alpha * px.time_alpha) + 1e-6f;
        g = __fmaf_rn(blend, rsqrtf(den), density);
    }
    return g;
}

__device__ __forceinline__ bool wang_active(const GrainFrame* f) {
    return f->wang_tiles && f->wang_lut && f->wang_w > 0 && f->wang_h > 0 && f->wang_count > 0 &&
           f->pixel_size_um > 0.0f && f->wang_cell_mm > 0.0f && f->wang_colors > 0;
}

// A pixel coordinate in FP32 (rounded once either way).
__device__ __forceinline__ float coordinate(uint64_t a) {
    return (a >> 31) == 0 ? (float)(int)a : (float)a;
}

// Position of a pixel coordinate in Wang cells.
__device__ __forceinline__ float wang_position(const GrainFrame* f, uint64_t a) {
    const float mm = coordinate(a) * (f->pixel_size_um * 0.001f);
    const float inv = 1.0f / f->wang_cell_mm;
    return mm * inv;
}

// Rows (or columns) of a tile of size n that position c reads: where it lies in its cell, and
// half a tile on, wrapped.
__device__ __forceinline__ void wang_samples(float c, int n, int& near, int& far) {
    near = (int)floorf((c - floorf(c)) * (float)n);
    if (near >= n) near = n - 1;
    far = near + (n >> 1);
    if (far >= n) far -= n;
}

// The tile of cell (mx, my): its edges' colours are hashes of the cells they separate.
__device__ __forceinline__ int wang_tile(const GrainFrame* f, int64_t mx, int64_t my) {
    const int colors = f->wang_colors;
    const uint64_t s0 = f->clip_token != 0 ? f->clip_token : f->session_seed;
    const uint64_t base = s0 != 0 ? s0 : 1ULL;
    const uint32_t l = hash_u32((int)mx, (int)my, base, 0xA5A5A5A5u) % colors;
    const uint32_t r = hash_u32((int)(mx + 1), (int)my, base, 0x5A5A5A5Au) % colors;
    const uint32_t t = hash_u32((int)mx, (int)my, base, 0xC3C3C3C3u) % colors;
    const uint32_t b = hash_u32((int)mx, (int)(my + 1), base, 0x3C3C3C3Cu) % colors;
    const size_t c = (size_t)colors;
    return (int)f->wang_lut[(((size_t)l * c + r) * c + t) * c + b];
}

// Shift of the blue-noise lookup by two samples of the pixel's tile (0 where there is none).
__device__ __forceinline__ void wang_shift(const GrainFrame* f, int tile, int tx, int hx, int ty, int hy, int& ox,
                                           int& oy) {
    const int w = f->wang_w, h = f->wang_h;
    float v0 = 0.0f, v1 = 0.0f;
    if (tile >= 0 && tile < f->wang_count) {
        const uint8_t* t = f->wang_tiles + (size_t)tile * (size_t)h * (size_t)w;
        v0 = noise_uniform(__ldg(t + ((size_t)ty * (size_t)w + tx)));
        v1 = noise_uniform(__ldg(t + ((size_t)hy * (size_t)w + hx)));
    }
    const int warp_x = f->stbn_w > 0 ? ((f->stbn_w / 8) > 4 ? f->stbn_w / 8 : 4) : 0;
    const int warp_y = f->stbn_h > 0 ? ((f->stbn_h / 8) > 4 ? f->stbn_h / 8 : 4) : 0;
    if (warp_x == 0 || warp_y == 0) return;
    ox = (int)floorf((v0 - 0.5f) * 2.0f * (float)warp_x);
    oy = (int)floorf((v1 - 0.5f) * 2.0f * (float)warp_y);
}

// The shift where the block holds no cells (negative or far coordinates).
__device__ __noinline__ void wang_offsets(const GrainFrame* f, uint64_t ax, uint64_t ay, int& ox, int& oy) {
    const float cx = wang_position(f, ax), cy = wang_position(f, ay);
    int tx, hx, ty, hy;
    wang_samples(cx, f->wang_w, tx, hx);
    wang_samples(cy, f->wang_h, ty, hy);
    wang_shift(f, wang_tile(f, (int64_t)floorf(cx), (int64_t)floorf(cy)), tx, hx, ty, hy, ox, oy);
}

// Coordinate `k` of the noise fields (kNoiseCoords) at column ax or row ay.
__device__ __forceinline__ float noise_x(const GrainFrameUniforms& u, int k, uint64_t ax) {
    if (k < 2) return (coordinate(ax) + u.breathing_drift_x) / (k == 0 ? u.breathing_cell_small_px : u.breathing_cell_large_px);
    const float xs = coordinate(ax) / u.clump_cell_px;
    return k == 2 ? xs : xs + 19.19f;
}
__device__ __forceinline__ float noise_y(const GrainFrameUniforms& u, int k, uint64_t ay) {
    if (k < 2)
        return (coordinate(ay) + u.breathing_drift_y + u.breathing_roll_y) /
               (k == 0 ? u.breathing_cell_small_px : u.breathing_cell_large_px);
    const float ys = (coordinate(ay) + u.clump_roll_y) / u.clump_cell_px;
    return k == 2 ? ys : ys + 7.23f;
}
__device__ __forceinline__ uint64_t noise_seed(const GrainFrameUniforms& u, int field) {
    const uint64_t seed = field >= 4 ? u.clump_static_seed : (field & 1) ? u.breathing_seed_b : u.breathing_seed_a;
    return seed ^ (field == 2 || field == 3 || field == 5 ? 0xBF58476D1CE4E5B9ULL : 0x9E3779B97F4A7C15ULL);
}

__device__ __forceinline__ float field_noise(const GrainTables& t, int field, const NoiseAxis& x, const NoiseAxis& y) {
    const NoiseField& q = t.field[field];
    if (q.nx > 0) {
        const float* v = t.lattice[field] + ((y.i - q.y0) * q.nx + (x.i - q.x0));
        return value_noise(x, y, [&](int i, int j) { return v[(j - y.i) * q.nx + (i - x.i)]; });
    }
    return value_noise(x, y, [&](int i, int j) { return spatial_hash01(i, j, q.seed); });
}

__device__ __forceinline__ float breathing_factor(const GrainFrame* f, const GrainFrameUniforms& u,
                                                  const GrainTables& t, const NoiseAxis x[kNoiseCoords],
                                                  const NoiseAxis y[kNoiseCoords]) {
    if (!u.breathing_active) return 1.0f;
    const float sa = field_noise(t, 0, x[0], y[0]);
    const float sb = field_noise(t, 1, x[0], y[0]);
    const float la = field_noise(t, 2, x[1], y[1]);
    const float lb = field_noise(t, 3, x[1], y[1]);
    const float ns = __fmaf_rn(sb - sa, u.breathing_t, sa);
    const float nl = __fmaf_rn(lb - la, u.breathing_t, la);
    const float noise = __fmaf_rn(u.breathing_mix, ns, (1.0f - u.breathing_mix) * nl);
    const float n = __fmaf_rn(noise, 2.0f, -1.0f);
    const float factor = __fmaf_rn(f->breathing_amplitude, n, 1.0f);
    return factor > 0.0f ? factor : 0.0f;
}

__device__ __forceinline__ float clump_factor(const GrainFrameUniforms& u, const GrainTables& t,
                                              const NoiseAxis x[kNoiseCoords], const NoiseAxis y[kNoiseCoords]) {
    if (!u.clump_active) return 1.0f;
    const float a = field_noise(t, 4, x[2], y[2]);
    const float b = field_noise(t, 5, x[3], y[3]);
    const float u1 = clamp01(a, 1e-6f, 1.0f - 1e-6f);
    const float u2 = clamp01(b, 0.0f, 1.0f);
    const float r = sqrtf(-2.0f * logf(u1));
    const float n = r * cosf(kTwoPi * u2);
    float v = expf(__fmaf_rn(u.clump_sigma, n, u.clump_mu));
    if (!finite(v)) v = 1.0f;
    return v * u.clump_rms_norm;
}

// Density of one sublayer at the given total density: linear interpolation of the
// layer curve over the capture density curve (negated for positive film), with the
// 16-block prefix-maximum search for finite 256-sample axes (on a rising axis a binary search
// finds the same sample). The place on the axis is the same for all layers.
struct LayerPlace {
    int i0;  // sample, or -1: the density itself
    float t; // position to the next sample; below 0: the sample's value
};

__device__ __forceinline__ LayerPlace layer_place(const GrainFrame* f, const float* rising, int ch, float density) {
    const float* x = f->base_curve[ch];
    const int n = f->base_curve_n[ch];
    if (!x || n <= 0) return {-1, 0.0f};
    if (!finite(density)) return {0, -1.0f};
    const bool pos = f->positive_film != 0;
    const float q = pos ? -density : density;
    if (rising) { // 256 finite samples
        if (q <= rising[0]) return {0, -1.0f};
        if (q >= rising[255]) return {255, -1.0f};
        int lo = 0; // rising[lo] < q
#pragma unroll
        for (int step = 128; step > 0; step >>= 1)
            if (lo + step < 256 && rising[lo + step] < q) lo += step;
        const float den = rising[lo + 1] - rising[lo];
        if (!(den > 0.0f) || !finite(den)) return {lo, -1.0f};
        return {lo, (q - rising[lo]) / den};
    }
    auto axis = [&](int i) {
        const float v = __ldg(x + i);
        return pos ? -v : v;
    };
    const bool bounded = f->axis_finite[ch] != 0 && n == 256;
    int b0 = 0, b1 = n - 1;
    if (!bounded) {
        while (b0 < n && !finite(axis(b0))) ++b0;
        if (b0 >= n) return {-1, 0.0f};
        while (b1 > b0 && !finite(axis(b1))) --b1;
    }
    const float xmin = axis(b0), xmax = axis(b1);
    if (!finite(xmin) || !finite(xmax) || !(xmax >= xmin)) return {b0, -1.0f};
    if (q <= xmin) return {b0, -1.0f};
    if (q >= xmax) return {b1, -1.0f};
    int i1 = b0 + 1;
    if (bounded) {
        const float* prefix = f->axis_block_prefix_max[ch];
        int lo = 0, hi = 15;
#pragma unroll
        for (int step = 0; step < 4; ++step) {
            const int mid = lo + (hi - lo) / 2;
            if (prefix[mid] < q)
                lo = mid + 1;
            else
                hi = mid;
        }
        i1 = max(1, lo * 16);
        const int end = min(b1, (lo + 1) * 16 - 1);
        while (i1 <= end && axis(i1) < q) ++i1;
    } else {
        while (i1 <= b1 && axis(i1) < q) ++i1;
    }
    if (i1 > b1) return {b1, -1.0f};
    const int i0 = i1 - 1;
    const float x0 = axis(i0), x1v = axis(i1);
    const float den = x1v - x0;
    if (!(den > 0.0f) || !finite(den)) return {i0, -1.0f};
    return {i0, (q - x0) / den};
}

__device__ __forceinline__ float layer_density(const GrainFrame* f, int ch, int layer, const LayerPlace& at,
                                               float density) {
    const float* y = f->layer_curve[layer][ch];
    if (!y || at.i0 < 0) return density;
    const float y0 = __ldg(y + at.i0);
    if (!(at.t >= 0.0f)) return y0;
    return __fmaf_rn(at.t, __ldg(y + at.i0 + 1) - y0, y0);
}

// The tables that hold for the whole pass; returns whether tables.axis holds a rising axis.
template <int Mode>
__device__ __forceinline__ bool prepare_pass(const GrainFrame& f, GrainTables& tables, int ch, bool use_stbn,
                                             bool retime) {
    const int tid = threadIdx.x;
    if (tid == 0) tables.u = *f.uniforms;
    if (use_stbn) {
        if (tid < (retime ? 6 : 3) * kTableDraws) {
            const int frame = tid / (3 * kTableDraws), slot = tid / kTableDraws % 3, d = tid % kTableDraws;
            const uint64_t salt = (uint64_t)ch + (uint64_t)slot * 10ULL;
            tables.draws[frame][slot][d] = draw_hash((frame ? f.seed_base_next : f.seed_base) ^ salt, (uint32_t)d);
        }
        tables.radius[tid] = normal_radius(noise_uniform((uint32_t)tid));
        tables.cosine[tid] = normal_cosine(noise_uniform((uint32_t)tid));
        if (tid < 2) {
            tables.pitch_offset[tid] = f.pitch_px > 0 ? (int64_t)f.pitch_px * (f.frame_index + (int64_t)tid) : 0;
            const int wf = wrap_coordinate((int64_t)f.stbn_frame + (int64_t)tid, f.stbn_frames);
            tables.frame_row[tid] = (size_t)wf * (size_t)f.stbn_h;
            tables.frame_base[tid] = f.stbn + tables.frame_row[tid] * (size_t)f.stbn_w;
        }
    }
    bool rising = false;
    if constexpr (Mode != kGrainSimple) {
        rising = f.base_curve[ch] && f.base_curve_n[ch] == 256 && f.axis_finite[ch] != 0;
        if (rising) {
            const float v = __ldg(f.base_curve[ch] + tid);
            tables.axis[tid] = f.positive_film != 0 ? -v : v;
        }
    }
    __syncthreads();
    if constexpr (Mode != kGrainSimple) {
        if (rising) {
            bool ok = finite(tables.axis[tid]) && (tid == 0 || tables.axis[tid - 1] <= tables.axis[tid]);
            if (tid < 16) ok = ok && f.axis_block_prefix_max[ch][tid] == tables.axis[16 * tid + 15];
            rising = __syncthreads_and(ok) != 0;
        }
    }
    return rising;
}

// The tables of a tile: rows y0 .. y1 - 1, columns x0 .. x1 - 1. One warp per noise field, one
// for the Wang cells; the rows' coordinates by the first four.
__device__ __forceinline__ void prepare_tile(const GrainFrame& f, GrainTables& tables, bool use_stbn, int x0, int x1,
                                             int y0, int y1) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const GrainFrameUniforms& u = tables.u;
    const int64_t ax = (int64_t)f.origin_x + x0, ay = (int64_t)f.origin_y + y0;
    const int64_t bx = (int64_t)f.origin_x + x1 - 1, by = (int64_t)f.origin_y + y1 - 1;
    // coordinates are unsigned 64-bit: a tile that holds negative ones is not in order
    const bool ordered = ax >= 0 && ay >= 0;
    static_assert(kSampleThreads >= 32 * (kNoiseFields + 1) && kNoiseCoords * kBlockRows <= kSampleThreads,
                  "a warp per noise field, one for the Wang cells");
    if (warp < kNoiseFields) {
        const int field = warp;
        if (field < 4 ? u.breathing_active : u.clump_active) {
            const int k = noise_coord(field);
            const uint64_t seed = noise_seed(u, field);
            NoiseField q{seed, 0, 0, 0, 0};
            if (ordered) {
                const float px = noise_x(u, k, (uint64_t)ax), py = noise_y(u, k, (uint64_t)ay);
                const float qx = noise_x(u, k, (uint64_t)bx), qy = noise_y(u, k, (uint64_t)by);
                if (fabsf(px) < 1e9f && fabsf(py) < 1e9f && qx - px < (float)kLattice && qy - py < (float)kLattice) {
                    q.x0 = (int)floorf(px);
                    q.y0 = (int)floorf(py);
                    q.nx = (int)floorf(qx) - q.x0 + 2;
                    q.ny = (int)floorf(qy) - q.y0 + 2;
                    if (q.nx < 2 || q.ny < 2 || q.nx * q.ny > kLattice) q.nx = 0;
                }
            }
            for (int i = lane; i < q.nx * q.ny; i += 32)
                tables.lattice[field][i] = spatial_hash01(q.x0 + i % q.nx, q.y0 + i / q.nx, seed);
            if (lane == 0) tables.field[field] = q;
        }
    } else if (warp == kNoiseFields && use_stbn && wang_active(&f)) {
        int64_t mx = 0, my = 0;
        int nx = 0, ny = 0;
        if (ordered) {
            const float px = wang_position(&f, (uint64_t)ax), py = wang_position(&f, (uint64_t)ay);
            const float qx = wang_position(&f, (uint64_t)bx), qy = wang_position(&f, (uint64_t)by);
            if (qx < 1e9f && qy < 1e9f && qx - px < (float)kWangCells && qy - py < (float)kWangCells) {
                mx = (int64_t)floorf(px);
                my = (int64_t)floorf(py);
                nx = (int)((int64_t)floorf(qx) - mx) + 1;
                ny = (int)((int64_t)floorf(qy) - my) + 1;
                if (nx < 1 || ny < 1 || nx * ny > kWangCells) nx = ny = 0;
            }
        }
        for (int i = lane; i < nx * ny; i += 32) tables.wang_tile[i] = wang_tile(&f, mx + i % nx, my + i / nx);
        for (int i = lane; nx > 0 && i < y1 - y0; i += 32) {
            const float cy = wang_position(&f, (uint64_t)(ay + i));
            WangRow r;
            r.cell = ((int)floorf(cy) - (int)my) * nx;
            wang_samples(cy, f.wang_h, r.near, r.far);
            tables.wang_row[i] = r;
        }
        if (lane == 0) {
            tables.wang_x = mx;
            tables.wang_nx = nx;
        }
    }
    if (tid < kNoiseCoords * kBlockRows) {
        const int k = tid / kBlockRows, r = tid % kBlockRows;
        if (r < y1 - y0 && (k < 2 ? u.breathing_active : u.clump_active))
            tables.row[k][r] = noise_axis(noise_y(u, k, (uint64_t)(ay + r)));
    }
}

// The grid's blocks walk tiles of kSampleColumns x `rows` pixels, `columns` tiles to a row.
template <int Mode>
__global__ void __launch_bounds__(kSampleThreads, kSampleBlocks)
    grain_sample_kernel(const __grid_constant__ GrainFrame f, int ch, int layer, const float* __restrict__ density_in,
                        long long din_stride, GrainPlane out, GrainSampleEpilogue ep, int width, int height, int rows,
                        int columns, int tiles) {
    __shared__ GrainTables tables;
    const int lane = threadIdx.x % kSampleColumns, line = threadIdx.x / kSampleColumns;
    PixelContext px;
    px.time_alpha = f.time_alpha;
    px.retime = f.time_alpha > 1e-6f && f.time_alpha < 0.999999f;
    px.use_stbn = (f.stbn && f.stbn_w > 0 && f.stbn_h > 0 && f.stbn_frames > 0) ? 1 : 0;
    const bool rising = prepare_pass<Mode>(f, tables, ch, px.use_stbn != 0, px.retime);
    const GrainFrameUniforms& u = tables.u;
    const bool wang = px.use_stbn && wang_active(&f);
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int x0 = tile % columns * kSampleColumns, y0 = tile / columns * rows, y1 = min(y0 + rows, height);
        __syncthreads();
        prepare_tile(f, tables, px.use_stbn != 0, x0, min(x0 + kSampleColumns, width), y0, y1);
        __syncthreads();
        const int x = x0 + lane;
        if (x >= width) continue;
        px.ax = (uint64_t)((int64_t)f.origin_x + x);
        NoiseAxis noise_col[kNoiseCoords];
#pragma unroll
        for (int k = 0; k < kNoiseCoords; ++k)
            noise_col[k] =
                (k < 2 ? u.breathing_active : u.clump_active) ? noise_axis(noise_x(u, k, px.ax)) : NoiseAxis{0, 0.0f};
        const bool wang_held = wang && tables.wang_nx > 0;
        int wang_cell = 0, wang_near = 0, wang_far = 0;
        if (wang_held) {
            const float cx = wang_position(&f, px.ax);
            wang_cell = (int)floorf(cx) - (int)tables.wang_x;
            wang_samples(cx, f.wang_w, wang_near, wang_far);
        }
#pragma unroll 1
        for (int y = y0 + line; y < y1; y += kSampleRows) {
            const float in_density = density_in[(long long)y * din_stride + x];
            px.ay = (uint64_t)((int64_t)f.origin_y + y);
            px.wang_x = px.wang_y = 0;
            if (wang_held) {
                const WangRow r = tables.wang_row[y - y0];
                wang_shift(&f, tables.wang_tile[r.cell + wang_cell], wang_near, wang_far, r.near, r.far, px.wang_x,
                           px.wang_y);
            } else if (wang) {
                wang_offsets(&f, px.ax, px.ay, px.wang_x, px.wang_y);
            }
            NoiseAxis noise_row[kNoiseCoords];
#pragma unroll
            for (int k = 0; k < kNoiseCoords; ++k) noise_row[k] = tables.row[k][y - y0];

            px.clump = clump_factor(u, tables, noise_col, noise_row);
            px.breathing = breathing_factor(&f, u, tables, noise_col, noise_row);

            float value;
            if (Mode == kGrainSimple) {
                const float density = in_density + f.density_min[ch];
                const int nsub = f.n_sublayers > 0 ? f.n_sublayers : 1;
                const ParticleSample s{density, f.density_max[ch], f.n_particles[ch], f.od_particle[ch],
                                       f.uniformity[ch]};
                float acc[2] = {0.0f, 0.0f};
#pragma unroll 1
                for (int sl = 0; sl < nsub; ++sl) {
                    const uint64_t salt = (uint64_t)ch + (uint64_t)sl * 10ULL;
                    acc[0] += particle_model(&f, &tables, s, px, sl, 0, f.seed_base ^ salt);
                    if (px.retime) acc[1] += particle_model(&f, &tables, s, px, sl, 1, f.seed_base_next ^ salt);
                }
                acc[0] /= (float)nsub;
                if (px.retime) acc[1] /= (float)nsub;
                value = sanitize(blend_frames(px, density, acc[0], acc[1]));
            } else {
                const LayerPlace at = layer_place(&f, rising ? tables.axis : nullptr, ch, in_density);
                const int first = Mode == kGrainLayer ? layer : 0, last = Mode == kGrainLayer ? layer : 2;
                float sum = 0.0f;
#pragma unroll 3
                for (int l = first; l <= last; ++l) {
                    const uint64_t salt = (uint64_t)ch + (uint64_t)l * 10ULL;
                    const float density = layer_density(&f, ch, l, at, in_density) + f.density_min_layers[l][ch];
                    const ParticleSample s{density, f.density_max_layers[l][ch], f.n_particles_layers[l][ch],
                                           f.od_particle_layers[l][ch], f.uniformity[ch]};
                    const float g = particle_model(&f, &tables, s, px, l, 0, f.seed_base ^ salt);
                    float gn = 0.0f;
                    if (px.retime) gn = particle_model(&f, &tables, s, px, l, 1, f.seed_base_next ^ salt);
                    const float v = sanitize(blend_frames(px, density, g, gn));
                    sum = Mode == kGrainLayer ? v : sum + v;
                }
                value = sanitize(sum);
            }

            float* o = out.p + (long long)y * out.stride + x;
            if (ep.accumulate) value = sanitize((ep.init ? 0.0f : *o) + value);
            if (ep.form_delta) {
                if (ep.density_bias != 0.0f) value = sanitize(value + ep.density_bias);
                value = sanitize(value - in_density);
            }
            *o = value;
        }
    }
}

__device__ __forceinline__ int reflect_half(int i, int n) {
    if ((unsigned)i < (unsigned)n) return i; // most: the remainder below is an integer division
    if (n <= 1) return 0;
    const int period = 2 * n;
    int m = i % period;
    if (m < 0) m += period;
    return m < n ? m : period - 1 - m;
}

// Both blurs are bound by instruction issue at the small radii grain has; a thread carries
// several outputs through the taps, so that a tap's weight and the loop are paid once for all.
// 3840x2160, radius 2: rows 52 -> 20 us, columns 35 -> 22 us.
constexpr int kRowThreads = 128;
constexpr int kRowOutputs = 4;
constexpr int kRowTile = kRowThreads * kRowOutputs;
constexpr int kRowLines = 2;

__global__ void __launch_bounds__(kRowThreads* kRowLines) grain_rows_kernel(const float* __restrict__ in,
                                                                           long long in_stride,
                                                                           float* __restrict__ out,
                                                                           long long out_stride,
                                                                           const __grid_constant__ GrainBlurTaps taps,
                                                                           int width, int height) {
    extern __shared__ float tile[];
    const int r = taps.radius;
    const int x0 = blockIdx.x * kRowTile;
    const int tw = min(kRowTile, width - x0) + 2 * r;
    const int y = blockIdx.y * kRowLines + threadIdx.y;
    float* row = tile + threadIdx.y * (kRowTile + 2 * r);
    if (y < height) {
        const float* src = in + (long long)y * in_stride;
        for (int i = threadIdx.x; i < tw; i += kRowThreads) row[i] = src[reflect_half(x0 - r + i, width)];
    }
    __syncthreads();
    const int x = x0 + threadIdx.x;
    if (y >= height || x >= width) return;
    float acc[kRowOutputs] = {};
    const float* v = row + threadIdx.x;
    for (int k = 0; k <= 2 * r; ++k)
#pragma unroll
        for (int j = 0; j < kRowOutputs; ++j) acc[j] = __fmaf_rn(v[k + j * kRowThreads], taps.w[k], acc[j]);
    float* o = out + (long long)y * out_stride + x;
#pragma unroll
    for (int j = 0; j < kRowOutputs; ++j)
        if (x + j * kRowThreads < width) o[j * kRowThreads] = sanitize(acc[j]);
}

constexpr int kColTileX = 32;
constexpr int kColThreadsY = 8;
constexpr int kColOutputs = 8;
constexpr int kColTileY = kColThreadsY * kColOutputs;

__global__ void __launch_bounds__(kColTileX* kColThreadsY) grain_columns_kernel(
    const float* __restrict__ in, long long in_stride, GrainPlane out, const __grid_constant__ GrainBlurTaps taps,
    GrainVerticalEpilogue ep, int width, int height) {
    extern __shared__ float tile[];
    const int r = taps.radius;
    const int x0 = blockIdx.x * kColTileX, y0 = blockIdx.y * kColTileY;
    const int th = min(kColTileY, height - y0) + 2 * r;
    const int x = x0 + threadIdx.x;
    if (x < width)
        for (int i = threadIdx.y; i < th; i += kColThreadsY)
            tile[i * kColTileX + threadIdx.x] = in[(long long)reflect_half(y0 - r + i, height) * in_stride + x];
    __syncthreads();
    if (x >= width) return;
    float sum[kColOutputs] = {};
    const float* v = tile + threadIdx.y * kColTileX + threadIdx.x;
    for (int k = 0; k <= 2 * r; ++k)
#pragma unroll
        for (int j = 0; j < kColOutputs; ++j)
            sum[j] = __fmaf_rn(v[(k + j * kColThreadsY) * kColTileX], taps.w[k], sum[j]);
    const float w = isfinite(ep.weight) ? ep.weight : 0.0f;
    const float gain = isfinite(ep.gain) ? ep.gain : 0.0f;
#pragma unroll
    for (int j = 0; j < kColOutputs; ++j) {
        const int y = y0 + threadIdx.y + j * kColThreadsY;
        if (y >= height) break;
        const float blurred = sanitize(sum[j]);
        float* o = out.p + (long long)y * out.stride + x;
        const float prev = ep.init ? 0.0f : *o;
        float value = ep.weighted ? __fmaf_rn(w, blurred, prev) : prev + blurred;
        value = sanitize(value);
        if (!ep.weighted && ep.density) {
            if (ep.density_bias != 0.0f) value = sanitize(value + ep.density_bias);
            value = sanitize(value - ep.density[(long long)y * ep.density_stride + x]);
        }
        if (ep.apply_gain) value = sanitize(value * gain);
        *o = value;
    }
}

__global__ void grain_accumulate_weighted_kernel(GrainPlane dst, const float* __restrict__ src, long long src_stride,
                                                 float weight, int init, int apply_gain, float gain, int width,
                                                 int height) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= width || y >= height) return;
    const float w = isfinite(weight) ? weight : 0.0f;
    float* o = dst.p + (long long)y * dst.stride + x;
    float v = sanitize(__fmaf_rn(w, src[(long long)y * src_stride + x], init ? 0.0f : *o));
    if (apply_gain) v = sanitize(v * (isfinite(gain) ? gain : 0.0f));
    *o = v;
}

__global__ void grain_clear_kernel(GrainPlane dst, int width, int height) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x < width && y < height) dst.p[(long long)y * dst.stride + x] = 0.0f;
}

// `planes` density planes with the same deltas (all three when only the shared delta is
// mixed in: it is read once), V pixels of a row per thread. Bound by memory: 3840x2160, shared
// delta, 118 us as three launches of a pixel per thread -> 41 us.
template <int V>
__global__ void __launch_bounds__(256) grain_finish_kernel(GrainDensity density, int planes, long long density_stride,
                                                           const float* __restrict__ delta, long long delta_stride,
                                                           const float* __restrict__ shared, float shared_weight,
                                                           float independent_weight, float amplitude, float scale,
                                                           int add_mean, int width, int height) {
    const int x = (blockIdx.x * blockDim.x + threadIdx.x) * V;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= width || y >= height) return;
    const long long di = (long long)y * delta_stride + x;
    auto load = [](const float* p, float v[V]) {
        if constexpr (V == 4) {
            const float4 q = *reinterpret_cast<const float4*>(p);
            v[0] = q.x;
            v[1] = q.y;
            v[2] = q.z;
            v[3] = q.w;
        } else {
            v[0] = *p;
        }
    };
    float d[V];
    if (shared) {
        // the independent delta is read only when it carries weight (it is not
        // generated otherwise)
        const float sw = clamp01(shared_weight, 0.0f, 1.0f);
        const float iw = clamp01(independent_weight, 0.0f, 1.0f);
        float sv[V] = {}, iv[V] = {};
        if (sw > 0.0f) load(shared + di, sv);
        if (iw > 0.0f) load(delta + di, iv);
#pragma unroll
        for (int i = 0; i < V; ++i) d[i] = sanitize(amplitude * __fmaf_rn(sw, sv[i], iw * iv[i]));
    } else {
        load(delta + di, d);
    }
    const float s = isfinite(scale) ? scale : 0.0f;
    for (int c = 0; c < planes; ++c) {
        float* o = density.p[c] + (long long)y * density_stride + x;
        float mean[V] = {};
        if (add_mean) load(o, mean);
#pragma unroll
        for (int i = 0; i < V; ++i) mean[i] = sanitize(__fmaf_rn(s, d[i], mean[i]));
        if constexpr (V == 4)
            *reinterpret_cast<float4*>(o) = make_float4(mean[0], mean[1], mean[2], mean[3]);
        else
            *o = mean[0];
    }
}

__global__ void grain_debug_average_kernel(float* c, float* m, float* y, long long stride, float offset, float scale,
                                           int width, int height) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int yy = blockIdx.y * blockDim.y + threadIdx.y;
    if (x >= width || yy >= height) return;
    const long long i = (long long)yy * stride + x;
    const float s = isfinite(scale) ? scale : 1.0f;
    const float o = isfinite(offset) ? offset : 0.0f;
    float avg = (c[i] + m[i] + y[i]) * (1.0f / 3.0f);
    if (!isfinite(avg)) avg = 0.0f;
    const float v = __fmaf_rn(avg, s, o);
    c[i] = v;
    m[i] = v;
    y[i] = v;
}

struct LognormalParameters {
    float mu, sigma;
};

__device__ __forceinline__ LognormalParameters lognormal_from_mean_std(float mean, float sd) {
    const float m2 = mean * mean, s2 = sd * sd;
    const float sigma_sq = logf(1.0f + s2 / m2);
    return {__fmaf_rn(-0.5f, sigma_sq, logf(fmaxf(1e-12f, mean))), sqrtf(fmaxf(0.0f, sigma_sq))};
}

__global__ void grain_uniforms_kernel(const __grid_constant__ GrainFrame f) {
    if (blockIdx.x != 0 || threadIdx.x != 0 || !f.uniforms) return;
    GrainFrameUniforms u{};
    const float time = (float)f.frame_index + f.time_alpha;
    if (f.breathing_amplitude > 0.0f && f.breathing_period_frames > 0 && f.pixel_size_um > 0.0f &&
        f.breathing_cell_um_small > 0.0f && f.breathing_cell_um_large > 0.0f) {
        const float period = (float)f.breathing_period_frames;
        const float step_f = floorf(time / period);
        const int64_t step = (int64_t)step_f;
        const float frac = __fmaf_rn(-step_f, period, time) / period;
        u.breathing_t = smoothstep(clamp01(frac, 0.0f, 1.0f));
        const uint64_t seed = f.session_seed != 0 ? f.session_seed : 1ULL;
        u.breathing_seed_a = splitmix64(seed ^ ((uint64_t)step * 0x8EBC6AF09C88C6E3ULL));
        u.breathing_seed_b = splitmix64(seed ^ ((uint64_t)(step + 1) * 0x8EBC6AF09C88C6E3ULL));
        const float inv_px = 1.0f / f.pixel_size_um;
        u.breathing_cell_small_px = fmaxf(4.0f, f.breathing_cell_um_small * inv_px);
        u.breathing_cell_large_px = fmaxf(4.0f, f.breathing_cell_um_large * inv_px);
        float drift = 0.0f;
        if (f.breathing_drift_um_per_frame > 0.0f) drift = f.breathing_drift_um_per_frame * inv_px;
        float dx = 0.0f, dy = 0.0f;
        if (drift > 0.0f) {
            const uint64_t h = splitmix64(seed ^ 0x6A09E667F3BCC909ULL);
            const float angle = (float)(uint32_t)(h & 0xFFFFFFFFu) * kInvU32 * kTwoPi;
            dx = cosf(angle) * drift;
            dy = sinf(angle) * drift;
        }
        const float roll = f.pitch_px > 0 ? (float)f.pitch_px : 0.0f;
        u.breathing_drift_x = dx * time;
        u.breathing_drift_y = dy * time;
        u.breathing_roll_y = roll * time;
        u.breathing_mix = clamp01(f.breathing_mix, 0.0f, 1.0f);
        u.breathing_active = 1;
    }
    const float sd_spatial = f.micro_structure[1] * 0.001f;
    if (sd_spatial > 0.0f && f.pixel_size_um > 0.0f) {
        float cell_um = f.micro_structure[0];
        if (!(cell_um > 0.0f)) cell_um = 0.0f;
        const float inv_px = 1.0f / f.pixel_size_um;
        u.clump_cell_px = cell_um * inv_px;
        if (!(u.clump_cell_px > 4.0f)) u.clump_cell_px = 4.0f;
        const float roll = f.pitch_px > 0 ? (float)f.pitch_px : 0.0f;
        u.clump_roll_y = roll * time;
        u.clump_static_seed = f.clip_token != 0 ? f.clip_token : f.session_seed;
        if (u.clump_static_seed == 0) u.clump_static_seed = 1ULL;
        float sd = sd_spatial;
        u.clump_rms_norm = 1.0f;
        const float mix = clamp01(f.clump_temporal_mix, 0.0f, 1.0f);
        if (mix > 0.0f) {
            int period_i = f.clump_morph_period_frames;
            if (period_i <= 0) period_i = 1;
            const float period = (float)period_i;
            const float step_f = floorf(time / period);
            const int64_t step = (int64_t)step_f;
            const float frac = __fmaf_rn(-step_f, period, time) / period;
            const float t = smoothstep(clamp01(frac, 0.0f, 1.0f));
            const uint64_t tseed = f.session_seed != 0 ? f.session_seed : 1ULL;
            const uint64_t sa = splitmix64(tseed ^ ((uint64_t)step * 0xD2B74407B1CE6E93ULL));
            const uint64_t sb = splitmix64(tseed ^ ((uint64_t)(step + 1) * 0xD2B74407B1CE6E93ULL));
            const float u1a = hash01(0, 0, sa ^ 0x9E3779B97F4A7C15ULL);
            const float u2a = hash01(1, 0, sa ^ 0xBF58476D1CE4E5B9ULL);
            const float u1b = hash01(0, 0, sb ^ 0x9E3779B97F4A7C15ULL);
            const float u2b = hash01(1, 0, sb ^ 0xBF58476D1CE4E5B9ULL);
            float u1 = __fmaf_rn(u1b - u1a, t, u1a);
            float u2 = __fmaf_rn(u2b - u2a, t, u2a);
            u1 = clamp01(u1, 1e-6f, 1.0f - 1e-6f);
            u2 = clamp01(u2, 0.0f, 1.0f);
            const float rt = sqrtf(-2.0f * logf(u1));
            const float nt = rt * cosf(kTwoPi * u2);
            const float strength_sd = mix * 0.23597824f;
            const LognormalParameters lp = lognormal_from_mean_std(1.0f, strength_sd);
            float strength = expf(__fmaf_rn(lp.sigma, nt, lp.mu));
            strength *= rsqrtf(__fmaf_rn(strength_sd, strength_sd, 1.0f));
            sd = sd_spatial * strength;
            const float den = __fmaf_rn(sd, sd, 1.0f);
            const float num = __fmaf_rn(sd_spatial, sd_spatial, 1.0f);
            u.clump_rms_norm = den > 0.0f ? sqrtf(num / den) : 1.0f;
        }
        const LognormalParameters lp = lognormal_from_mean_std(1.0f, sd);
        u.clump_mu = lp.mu;
        u.clump_sigma = lp.sigma;
        u.clump_active = 1;
    }
    *f.uniforms = u;
}

dim3 plane_grid(int width, int height) { return dim3((width + 31) / 32, (height + 7) / 8); }

} // namespace

cudaError_t launch_grain_uniforms(const GrainFrame& f, cudaStream_t s) {
    fjb::count_launch();
    grain_uniforms_kernel<<<1, 32, 0, s>>>(f);
    return cudaGetLastError();
}

cudaError_t launch_grain_sample(const GrainFrame& f, int mode, int channel, int layer, const float* density,
                                long long density_stride, GrainPlane out, const GrainSampleEpilogue& ep, int width,
                                int height, cudaStream_t s) {
    if (width <= 0 || height <= 0) return cudaSuccess;
    int device = 0, sms = 0;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    const int resident = (sms > 0 ? sms : 148) * kSampleBlocks;
    // tiles of several rows per thread share the tables, unless that leaves blocks without one
    int rows = kBlockRows;
    const int columns = (width + kSampleColumns - 1) / kSampleColumns;
    while (rows > kSampleRows && (long long)columns * ((height + rows - 1) / rows) < resident) rows /= 2;
    const long long tiles = (long long)columns * ((height + rows - 1) / rows);
    auto* k = mode == kGrainSimple  ? grain_sample_kernel<kGrainSimple>
              : mode == kGrainLayer ? grain_sample_kernel<kGrainLayer>
                                    : grain_sample_kernel<kGrainTriplet>;
    fjb::count_launch();
    k<<<(unsigned)std::min<long long>(tiles, resident), kSampleThreads, 0, s>>>(
        f, channel, layer, density, density_stride, out, ep, width, height, rows, columns, (int)tiles);
    return cudaGetLastError();
}

cudaError_t launch_grain_blur_rows(const float* in, long long in_stride, float* out, long long out_stride,
                                   const GrainBlurTaps& taps, int width, int height, cudaStream_t s) {
    if (width <= 0 || height <= 0) return cudaSuccess;
    if (taps.radius <= 0 || taps.radius > kGrainMaxRadius) return cudaErrorInvalidValue;
    const size_t smem = (size_t)kRowLines * (kRowTile + 2 * taps.radius) * sizeof(float);
    const dim3 grid((width + kRowTile - 1) / kRowTile, (height + kRowLines - 1) / kRowLines);
    fjb::count_launch();
    grain_rows_kernel<<<grid, dim3(kRowThreads, kRowLines), smem, s>>>(in, in_stride, out, out_stride, taps, width,
                                                                    height);
    return cudaGetLastError();
}

cudaError_t launch_grain_blur_columns(const float* in, long long in_stride, GrainPlane out,
                                      const GrainBlurTaps& taps, const GrainVerticalEpilogue& ep, int width,
                                      int height, cudaStream_t s) {
    if (width <= 0 || height <= 0) return cudaSuccess;
    if (taps.radius <= 0 || taps.radius > kGrainMaxRadius) return cudaErrorInvalidValue;
    const size_t smem = (size_t)(kColTileY + 2 * taps.radius) * kColTileX * sizeof(float);
    const dim3 grid((width + kColTileX - 1) / kColTileX, (height + kColTileY - 1) / kColTileY);
    fjb::count_launch();
    grain_columns_kernel<<<grid, dim3(kColTileX, kColThreadsY), smem, s>>>(in, in_stride, out, taps, ep, width,
                                                                           height);
    return cudaGetLastError();
}

cudaError_t launch_grain_accumulate_weighted(GrainPlane dst, const float* src, long long src_stride, float weight,
                                             int init, int apply_gain, float gain, int width, int height,
                                             cudaStream_t s) {
    if (width <= 0 || height <= 0) return cudaSuccess;
    fjb::count_launch();
    grain_accumulate_weighted_kernel<<<plane_grid(width, height), dim3(32, 8), 0, s>>>(
        dst, src, src_stride, weight, init, apply_gain, gain, width, height);
    return cudaGetLastError();
}

cudaError_t launch_grain_clear(GrainPlane dst, int width, int height, cudaStream_t s) {
    if (width <= 0 || height <= 0) return cudaSuccess;
    fjb::count_launch();
    grain_clear_kernel<<<plane_grid(width, height), dim3(32, 8), 0, s>>>(dst, width, height);
    return cudaGetLastError();
}

cudaError_t launch_grain_finish(const GrainDensity& density, int planes, long long density_stride, const float* delta,
                                long long delta_stride, const float* shared, float shared_weight,
                                float independent_weight, float amplitude, float scale, int add_mean, int width,
                                int height, cudaStream_t s) {
    if (width <= 0 || height <= 0) return cudaSuccess;
    // rows that start on 16 bytes and are whole float4s
    uintptr_t bits = reinterpret_cast<uintptr_t>(delta) | reinterpret_cast<uintptr_t>(shared);
    for (int c = 0; c < planes; ++c) bits |= reinterpret_cast<uintptr_t>(density.p[c]);
    const bool wide = bits % 16 == 0 && (width | density_stride | delta_stride) % 4 == 0;
    fjb::count_launch();
    if (wide)
        grain_finish_kernel<4><<<plane_grid(width / 4, height), dim3(32, 8), 0, s>>>(
            density, planes, density_stride, delta, delta_stride, shared, shared_weight, independent_weight, amplitude,
            scale, add_mean, width, height);
    else
        grain_finish_kernel<1><<<plane_grid(width, height), dim3(32, 8), 0, s>>>(
            density, planes, density_stride, delta, delta_stride, shared, shared_weight, independent_weight, amplitude,
            scale, add_mean, width, height);
    return cudaGetLastError();
}

cudaError_t launch_grain_debug_average(float* c, float* m, float* y, long long stride, float offset, float scale,
                                       int width, int height, cudaStream_t s) {
    if (width <= 0 || height <= 0) return cudaSuccess;
    fjb::count_launch();
    grain_debug_average_kernel<<<plane_grid(width, height), dim3(32, 8), 0, s>>>(c, m, y, stride, offset, scale,
                                                                                width, height);
    return cudaGetLastError();
}

} // namespace fjb
