// fjb_dir_lines.cu -- the spatial DIR filter, one warp per pair of lines (a7).
//
// The operators are those of fjb_dir_blur.cu (the reference's
// src/Cuda/Film/JuicerCudaFilmPipeline.cu:388-780): FP64 taps with half-sample
// reflection, and the third-order recursion with its reflected start and end block, here
// in the factored FP32 form with FP64 states between pieces, or, for coefficients without that
// form, in the direct one in FP64. Five launches: the short
// components, if any, both axes, summed into one plane per channel (fjb_fir2d.cuh; taps beyond
// radius 9 by two launches each, the post blurs' kernels); the rows'
// reflected starts; the recursive components' rows, four rows per CTA (fjb_line_pairs.cuh);
// the columns' reflected starts; the columns, one warp per pair of columns and recursive
// component, then the weighted sum of all of them and the plane of the first launch.
// Only short components take a plane of their own, so the planes are never more than the
// components, which is what the scratch holds. The filtered planes are written by the last launch
// alone, which does not read the corrections: one channel's may be another's corrections.
//
// The starts are launches of their own because their weights (three doubles for each of the
// first 21 sigma samples, 55 KB at 3840x2160) do not fit what the line kernels leave of L1:
// inside those kernels every warp fetched them from L2, all SMs the same lines at the
// same time, and they took 176 of the rows' 388 us and 121 of the columns' 419 us.
#include <cuda_runtime.h>

#include "fjb_dir.h"
#include "fjb_fir2d.cuh"
#include "fjb_launches.h"
#include "fjb_line_pairs.cuh"
#include "fjb_scanner_post.h"

namespace fjb {

namespace {

__device__ __forceinline__ void map_state(const double* T, const double d[3], double o[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) o[i] = T[3 * i] * d[0] + T[3 * i + 1] * d[1] + T[3 * i + 2] * d[2];
}

// Direct-form starts (y[n-1], y[n-2], y[n-3]) of the pair's lines as the step's state.
__device__ __forceinline__ void state_from(const DirComponentDev& c, const double a[3], const double b[3],
                                           Pair (&s)[3]) {
    double oa[3], ob[3];
    map_state(c.to_fac, a, oa);
    map_state(c.to_fac, b, ob);
#pragma unroll
    for (int i = 0; i < 3; ++i) s[i] = pack((float)oa[i], (float)ob[i]);
}

// End block of one line from its final state `d` (direct form): the last `ts` outputs in `term`,
// and the direct-form start of the way back.
__device__ __forceinline__ void end_block(const double* T, int ts, const double (&d)[3], double (&term)[3],
                                          double (&back)[3]) {
    for (int r = 0; r < 3; ++r) {
        double t = 0.0;
        if (r < ts) {
            t = d[0];
            for (int q = 0; q < ts; ++q) t += T[r * ts + q] * (d[ts - 1 - q] - d[0]);
        }
        term[r] = t;
        back[r] = r < ts ? t : d[r];
    }
}

// A recursive component's step and state in each of its forms.
struct Factored {
    using State = Pair[3];
    const DirComponentDev& c;
    __device__ __forceinline__ lp::FactoredStep op() const { return lp::FactoredStep(c.fac[0], c.fac[1], c.fac[2]); }
    // from direct-form states of the pair's lines, and back (one line's)
    __device__ __forceinline__ void from(const double a[3], const double b[3], State& s) const { state_from(c, a, b, s); }
    template <int kLine>
    __device__ __forceinline__ void to(const State& s, double (&d)[3]) const {
        double f[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) f[i] = kLine ? unpack(s[i]).y : unpack(s[i]).x;
        map_state(c.from_fac, f, d);
    }
    static __device__ __forceinline__ void of_lane(State& s, const State& t, int lane) {
#pragma unroll
        for (int i = 0; i < 3; ++i) s[i].v = __shfl_sync(0xffffffffu, t[i].v, lane);
    }
};
struct Direct {
    using State = lp::State2;
    const DirComponentDev& c;
    __device__ __forceinline__ lp::DirectStep64 op() const { return {c.ff, c.fb[0], c.fb[1], c.fb[2]}; }
    __device__ __forceinline__ void from(const double a[3], const double b[3], State& s) const {
#pragma unroll
        for (int i = 0; i < 3; ++i) s.a[i] = a[i], s.b[i] = b[i];
    }
    template <int kLine>
    __device__ __forceinline__ void to(const State& s, double (&d)[3]) const {
#pragma unroll
        for (int i = 0; i < 3; ++i) d[i] = kLine ? s.b[i] : s.a[i];
    }
    static __device__ __forceinline__ void of_lane(State& s, const State& t, int lane) { s = t.of(lane); }
};

// Reflected starts of the recursive components' lines: anchor + sum_i w[i] (x_i - anchor) over
// the first `len` samples, FP64. A warp takes four lines of a component (rows y .. y + 3, or
// two pairs of columns), lanes stride the samples, so that a weight serves four lines.
// Bound by the latency of its loads: a launch has few warps, so the components run side by side
// and eight samples of a lane are in flight (3840x2160: rows 23 us, columns 39 us; one
// component after the other, four samples: 57 and 56).
constexpr int kStartWarps = 8;

template <bool kCols>
__global__ void __launch_bounds__(32 * kStartWarps) dir_starts_kernel(const __grid_constant__ DirBlurParams P) {
    const int ch = blockIdx.y, lane = threadIdx.x & 31;
    const int W = P.width, H = P.height;
    const int lines = kCols ? 2 * lp::plane_pairs(W) : H;
    const int l0 = 4 * (blockIdx.x * kStartWarps + (threadIdx.x >> 5));
    if (l0 >= lines) return;
    const int words = lp::line_words(H);
    const int k = blockIdx.z;
    const DirComponentDev& c = P.comp[k];
    if (c.op != kDirOpYvv) return;
    const int len = kCols ? c.v_len : c.h_len;
    const double* w = kCols ? c.v_init : c.h_init;
    const float2* pair = reinterpret_cast<const float2*>(P.temp[ch][k]) + (size_t)(l0 / 2) * words + H - 1;
    auto samples = [&](int i, float (&v)[4]) {
        if (kCols) {
            const float2 a = pair[-i], b = pair[words - i];
            v[0] = a.x, v[1] = a.y, v[2] = b.x, v[3] = b.y;
        } else {
#pragma unroll
            for (int r = 0; r < 4; ++r) v[r] = P.raw[ch][(size_t)min(l0 + r, H - 1) * W + i];
        }
    };
    float f[4];
    samples(0, f);
    const double anchor[4] = {f[0], f[1], f[2], f[3]};
    double a[4][3] = {};
#pragma unroll 8
    for (int i = lane; i < len; i += 32) {
        const double w0 = __ldg(w + i), w1 = __ldg(w + len + i), w2 = __ldg(w + 2 * len + i);
        samples(i, f);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const double d = (double)f[r] - anchor[r];
            a[r][0] += w0 * d;
            a[r][1] += w1 * d;
            a[r][2] += w2 * d;
        }
    }
    double* out = (kCols ? P.col_start : P.row_start) + (((size_t)ch * kDirMaxComponents + k) * lines + l0) * 3;
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int h = 0; h < 3; ++h) {
            for (int o = 16; o > 0; o >>= 1) a[r][h] += __shfl_xor_sync(0xffffffffu, a[r][h], o);
            if (lane == 0 && l0 + r < lines) out[3 * r + h] = anchor[r] + a[r][h];
        }
}

// One recursive component over a pair of lines of n samples, in place: from the reflected
// starts at `from` (of the pair's two lines) out, the end block at the last `ts` samples, the
// way back from it. Rows count samples from position 0 up, columns (kDown) from position
// n - 1 down.
template <bool kDown, typename Form>
__device__ __forceinline__ void filter(const Form& form, const double* from, Pair* line, int n, int lane) {
    const DirComponentDev& c = form.c;
    const lp::LineMaps& maps = kDown ? c.col_maps : c.row_maps;
    const double* T = kDown ? c.v_term : c.h_term;
    const int ts = kDown ? c.v_tsize : c.h_tsize;
    const auto op = form.op();
    const lp::Piece piece(n, lane);
    auto sample = [&](int i) { return line + (kDown ? n - 1 - i : i); };
    typename Form::State start, s;
    {
        const double a[3] = {from[0], from[1], from[2]}, b[3] = {from[3], from[4], from[5]};
        form.from(a, b, start);
    }
    const bool low = lane == 0, high = piece.lo < piece.hi && piece.hi == n;
    const int up = lane, down = lp::kPieces - 1 - lane;
    lp::direction<!kDown>(op, maps, line, piece, kDown ? down : up, kDown ? high : low, start, s);
    // the lane that holds the line's end makes the end block; everyone gets the way back's start
    const int end_lane = kDown ? 0 : (n - 1) / piece.k;
    {
        double d[3], ta[3], tb[3], ba[3], bb[3];
        form.template to<0>(s, d);
        end_block(T, ts, d, ta, ba);
        form.template to<1>(s, d);
        end_block(T, ts, d, tb, bb);
        __syncwarp();
        if (lane == end_lane)
            for (int r = 0; r < ts; ++r)
                if (n - ts + r >= 0) *sample(n - ts + r) = pack((float)ta[r], (float)tb[r]);
        form.from(ba, bb, s);
        form.of_lane(start, s, end_lane);
    }
    // the way back leaves out the end block: the last ts positions, or the first (kDown)
    lp::Piece back = piece;
    if (kDown)
        back.lo = min(max(piece.lo, ts), piece.hi);
    else
        back.hi = max(min(piece.hi, n - ts), piece.lo);
    if (n > ts)
        lp::direction<kDown>(op, maps, line, back, kDown ? up : down,
                             back.lo < back.hi && (kDown ? back.lo == ts : back.hi == n - ts), start, s);
    __syncwarp();
}

// The same by the CTA's team, factored form.
template <bool kDown>
__device__ __forceinline__ void filter_team(const DirComponentDev& c, const double* from, Pair* line, int n,
                                            lp::TeamExchange& ex) {
    const Factored form{c};
    const lp::LineMaps& maps = kDown ? c.col_maps : c.row_maps;
    const double* T = kDown ? c.v_term : c.h_term;
    const int ts = kDown ? c.v_tsize : c.h_tsize, k = lp::team_piece_len(n, 1);
    const auto op = form.op();
    Pair start[3], s[3];
    {
        const double a[3] = {from[0], from[1], from[2]}, b[3] = {from[3], from[4], from[5]};
        form.from(a, b, start);
    }
    lp::direction_team<!kDown>(op, maps, line, 0, n, k, 1, start, s, ex);
    // the thread that holds the line's end makes the end block and the way back's start
    if ((int)threadIdx.x == (kDown ? 0 : (n - 1) / k)) {
        double d[3], ta[3], tb[3], ba[3], bb[3];
        form.template to<0>(s, d);
        end_block(T, ts, d, ta, ba);
        form.template to<1>(s, d);
        end_block(T, ts, d, tb, bb);
        for (int r = 0; r < ts; ++r) line[kDown ? ts - 1 - r : n - ts + r] = pack((float)ta[r], (float)tb[r]);
        form.from(ba, bb, s);
#pragma unroll
        for (int i = 0; i < 3; ++i) ex.start[i] = s[i].v;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 3; ++i) start[i].v = ex.start[i];
    lp::direction_team<kDown>(op, maps, line, kDown ? ts : 0, kDown ? n : n - ts, k, 1, start, s, ex);
}

// kDirect: some component has no factored form. A variant of its own: the FP64 states take
// registers.
template <bool kDown, bool kDirect>
__device__ __forceinline__ void filter(const DirComponentDev& c, const double* from, Pair* line, int n, int lane) {
    if (kDirect && !c.factored)
        filter<kDown>(Direct{c}, from, line, n, lane);
    else
        filter<kDown>(Factored{c}, from, line, n, lane);
}

// Warps of a CTA of one pair of lines: a team, unless a component runs in FP64.
template <bool kDirect>
constexpr int team_warps() {
    return kDirect ? 1 : lp::kTeam;
}

// Four rows of one channel per CTA (kPairs pairs) through every recursive component.
template <int kPairs, bool kDirect>
__global__ void __launch_bounds__(32 * (kPairs == 1 ? team_warps<kDirect>() : kPairs))
    dir_rows_kernel(const __grid_constant__ DirBlurParams P) {
    extern __shared__ __align__(16) unsigned char sm[];
    const int ch = blockIdx.y;
    const int W = P.width, H = P.height, lane = threadIdx.x & 31, warp = kPairs == 1 ? 0 : threadIdx.x >> 5;
    const int words = lp::line_words(W);
    Pair* rows = reinterpret_cast<Pair*>(sm);
    Pair* buf = rows + warp * words;
    // rows past the frame's end repeat the last one; their results land in the planes' padding
    const int y0 = 2 * kPairs * blockIdx.x, y = y0 + 2 * warp;
    const float* a = P.raw[ch] + (size_t)min(y, H - 1) * W;
    const float* b = P.raw[ch] + (size_t)min(y + 1, H - 1) * W;
    if (lane < 2 && (kPairs > 1 || threadIdx.x < 2) && y + lane + P.rows_ahead < H)
        lp::prefetch_block(a + (size_t)(lane + P.rows_ahead) * W, W);
#pragma unroll 1
    for (int k = 0; k < P.count; ++k) {
        const DirComponentDev& c = P.comp[k];
        if (c.op != kDirOpYvv) continue;
        // the last row's start again for a row past the frame's end
        const double* starts = P.row_start + ((size_t)ch * kDirMaxComponents + k) * H * 3;
        double from[6];
#pragma unroll
        for (int h = 0; h < 6; ++h) from[h] = __ldg(starts + (size_t)min(y + h / 3, H - 1) * 3 + h % 3);
        if constexpr (kPairs == 1 && !kDirect) {
            lp::load_rows<lp::kTeam>(buf, a, b, W, threadIdx.x);
            filter_team<false>(c, from, buf, W, lp::exchange(buf, words));
        } else {
            lp::load_rows(buf, a, b, W, lane);
            filter<false, kDirect>(c, from, buf, W, lane);
        }
        lp::store_pairs<kPairs>(rows, words, P.temp[ch][k], W, H, y0);
    }
}

// kPairs pairs of columns per CTA, P.recursions recursive components at a time; the sum so far
// waits in the first launch's plane or, where there is none (kRow), in the filtered plane
// between the rounds (more than one only for columns too long for all of them to fit).
template <bool kRow, int kPairs, bool kDirect>
__global__ void __cluster_dims__(lp::kStripPairs / kPairs, 1, 1)
    __launch_bounds__(32 * (kPairs == 1 ? team_warps<kDirect>() : kPairs * kDirMaxComponents), kPairs == lp::kColPairs && !kDirect ? 4 : 1)
    dir_cols_kernel(const __grid_constant__ DirBlurParams P) {
    extern __shared__ __align__(16) unsigned char sm[];
    const auto cluster = cooperative_groups::this_cluster();
    const int ch = blockIdx.y;
    const int W = P.width, H = P.height, lane = threadIdx.x & 31, warp = kPairs == 1 ? 0 : threadIdx.x >> 5;
    Pair* lines = reinterpret_cast<Pair*>(sm);
    Pair* line = lines + warp * lp::line_words(H);
    if (lane == 0 && (kPairs > 1 || threadIdx.x == 0)) {
        const unsigned next = blockIdx.y * gridDim.x + blockIdx.x + P.cols_ahead;
        if (next < gridDim.x * gridDim.y) {
            const int first = next % gridDim.x * kPairs, nch = next / gridDim.x;
            int slot = 0;
            for (int i = 0; i < P.count; ++i)
                if (P.comp[i].op == kDirOpYvv && slot++ == warp / kPairs)
                    lp::prefetch_line(P.temp[nch][i], first + warp % kPairs, H);
            if (P.base[nch] && warp < kPairs) lp::prefetch_line(P.base[nch], first + warp, H);
        }
    }
    lp::StripSum out{P.base[ch], P.filtered[ch], W, false, nullptr, W, 1.0f};
    int k = 0;
    do {
        float weight[lp::kMaxRecursions];
        int count = 0;
#pragma unroll 1
        for (; k < P.count && count < P.recursions; ++k) {
            const DirComponentDev& c = P.comp[k];
            if (c.op != kDirOpYvv) continue;
            if (warp / kPairs == count) {
                const int pair = blockIdx.x * kPairs + warp % kPairs;
                const double* starts =
                    P.col_start + (((size_t)ch * kDirMaxComponents + k) * 2 * lp::plane_pairs(W) + 2 * pair) * 3;
                double from[6];
#pragma unroll
                for (int h = 0; h < 6; ++h) from[h] = __ldg(starts + h);
                if constexpr (kPairs == 1 && !kDirect) {
                    lp::load_line<lp::kTeam>(line, P.temp[ch][k], pair, H, threadIdx.x);
                    filter_team<true>(c, from, line, H, lp::exchange(line, lp::line_words(H)));
                } else {
                    lp::load_line(line, P.temp[ch][k], pair, H, lane);
                    filter<true, kDirect>(c, from, line, H, lane);
                }
            }
            weight[count++] = c.weight;
        }
        while (k < P.count && P.comp[k].op != kDirOpYvv) ++k;
        cluster.sync();
        out.last = k >= P.count;
        lp::strip_sum<kRow, kPairs>(out, lines, weight, count, W, H);
        if constexpr (kRow) out.row = P.filtered[ch];
        cluster.sync(); // the other CTAs have read these lines
    } while (k < P.count);
}

using Kernel = void (*)(DirBlurParams);
template <bool kDirect>
Kernel rows_variant(const DirBlurParams& P) {
    return P.row_pairs == lp::kRowWarps ? dir_rows_kernel<lp::kRowWarps, kDirect> : dir_rows_kernel<1, kDirect>;
}
template <bool kDirect>
Kernel cols_variant(const DirBlurParams& P) {
    if (P.col_pairs == lp::kColPairs)
        return P.base[0] ? dir_cols_kernel<false, lp::kColPairs, kDirect> : dir_cols_kernel<true, lp::kColPairs, kDirect>;
    return P.base[0] ? dir_cols_kernel<false, 1, kDirect> : dir_cols_kernel<true, 1, kDirect>;
}

// Warps of a CTA of `lines` lines (pairs), and samples per piece of a line of n samples in a CTA of
// `pairs` pairs.
int warps_of(const DirBlurParams& P, int pairs, int lines) {
    return pairs > 1 ? lines : P.direct ? team_warps<true>() : team_warps<false>();
}
int piece_of(const DirBlurParams& P, int n, int pairs) {
    return pairs > 1 || P.direct ? lp::piece_len(n) : lp::team_piece_len(n, 1);
}

constexpr size_t kAlignFloats = 8; // planes start on 32 bytes
size_t starts_floats(int width, int height) {
    return 3 * (size_t)kDirMaxComponents * 3 * ((size_t)height + 2 * (size_t)lp::plane_pairs(width)) * 2;
}

} // namespace

// A plane for every component of the three channels (short ones share theirs), and the starts.
size_t dir_lines_floats(int width, int height) {
    return kAlignFloats + 3 * (size_t)kDirMaxComponents * lp::plane_floats(width, height) + starts_floats(width, height);
}

bool dir_lines_plan(DirBlurParams& P) {
    int lines = 0;
    bool base = false, wide = false;
    P.direct = false;
    for (int k = 0; k < P.count; ++k) {
        const DirComponentDev& c = P.comp[k];
        lines += c.op == kDirOpYvv;
        P.direct |= c.op == kDirOpYvv && !c.factored;
        base |= c.op != kDirOpYvv;
        wide |= c.op == kDirOpFir && c.radius > fir::kMaxRadius;
    }
    P.row_pairs = lp::pairs_per_cta(P.width);
    P.col_pairs = lp::pairs_per_cta(P.height);
    if (P.row_pairs < 1 || P.col_pairs < 1) return false;
    const size_t plane = lp::plane_floats(P.width, P.height);
    float* next = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(P.region) + 31) / 32 * 32);
    const size_t planes = 3 * (size_t)(lines + base + (wide && lines == 0));
    if ((size_t)(next - P.region) + planes * plane + starts_floats(P.width, P.height) > P.region_floats) return false;
    P.recursions = lp::recursions_per_cta(lines, P.col_pairs, P.height);
    P.raw_weight = 0.0f;
    for (int k = 0; k < P.count; ++k) {
        DirComponentDev& c = P.comp[k];
        if (c.op == kDirOpIdentity) P.raw_weight += c.weight;
        if (c.op != kDirOpYvv) continue;
        for (int ch = 0; ch < 3; ++ch, next += plane) P.temp[ch][k] = next;
        // one zero-input step: (s0, s1, s2) -> (fb0 s0 + fb1 s1 + fb2 s2, s0, s1) in the direct form
        const double direct[9] = {c.fb[0], c.fb[1], c.fb[2], 1, 0, 0, 0, 1, 0};
        c.row_maps = lp::line_maps(c.factored ? c.step_f : direct, piece_of(P, P.width, P.row_pairs));
        c.col_maps = lp::line_maps(c.factored ? c.step_f : direct, piece_of(P, P.height, P.col_pairs));
    }
    for (int ch = 0; ch < 3; ++ch) {
        P.base[ch] = base ? next : nullptr;
        if (base) next += plane;
        P.wide[ch] = P.temp[ch][0];
        for (int k = P.count - 1; k >= 0; --k)
            if (P.comp[k].op == kDirOpYvv) P.wide[ch] = P.temp[ch][k];
        if (wide && lines == 0) {
            P.wide[ch] = next;
            next += plane;
        }
    }
    P.row_start = reinterpret_cast<double*>(next);
    P.col_start = P.row_start + 3 * (size_t)kDirMaxComponents * 3 * P.height;
    return true;
}

cudaError_t launch_dir_lines(DirBlurParams& P, cudaStream_t s) {
    bool lines = false;
    fir::Jobs F{};
    F.width = P.width;
    F.height = P.height;
    F.dst_pairs = lp::plane_pairs(P.width);
    F.dst_words = lp::line_words(P.height);
    for (int ch = 0; ch < 3; ++ch) {
        fir::Job f{};
        f.src = P.raw[ch];
        f.stride = P.width;
        f.dst = P.base[ch];
        f.src_weight = P.raw_weight;
        for (int k = 0; k < P.count; ++k) {
            const DirComponentDev& c = P.comp[k];
            lines |= c.op == kDirOpYvv;
            if (c.op != kDirOpFir || c.radius > fir::kMaxRadius) continue;
            fir::Taps& t = f.set[f.count++];
            t.radius = c.radius;
            t.weight = c.weight;
            for (int i = 0; i < 2 * fir::kMaxRadius + 1; ++i) t.w[i] = c.host_taps[i];
        }
        if (f.dst) F.job[F.count++] = f;
    }
    cudaError_t e = cudaSuccess;
    if (F.count) {
        fjb::count_launch();
        fir::kernel<double><<<fir::grid(F), fir::kThreads, 0, s>>>(F);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    // wider taps, a component after the other
    for (int k = 0; k < P.count; ++k) {
        const DirComponentDev& c = P.comp[k];
        if (c.op != kDirOpFir || c.radius <= fir::kMaxRadius) continue;
        e = launch_blur_into_pairs(P.raw, P.wide, P.base, 3, P.width, P.height, c.taps, c.radius, c.weight, s);
        if (e != cudaSuccess) return e;
    }
    constexpr int kLinesPerCta = 4 * kStartWarps;
    if (lines) {
        fjb::count_launch();
        dir_starts_kernel<false><<<dim3((P.height + kLinesPerCta - 1) / kLinesPerCta, 3, P.count), 32 * kStartWarps, 0, s>>>(P);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        const size_t smem = lp::cta_bytes(P.row_pairs, P.width);
        auto* k = P.direct ? rows_variant<true>(P) : rows_variant<false>(P);
        e = fjb::allow_dynamic_smem(k, smem);
        if (e != cudaSuccess) return e;
        const int rows = 2 * P.row_pairs;
        P.rows_ahead = rows * lp::resident_ctas(smem);
        fjb::count_launch();
        k<<<dim3((P.height + rows - 1) / rows, 3), 32 * warps_of(P, P.row_pairs, P.row_pairs), smem, s>>>(P);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        fjb::count_launch();
        dir_starts_kernel<true>
            <<<dim3((2 * lp::plane_pairs(P.width) + kLinesPerCta - 1) / kLinesPerCta, 3, P.count), 32 * kStartWarps, 0, s>>>(P);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    const int columns = P.recursions * P.col_pairs;
    const size_t smem = lp::cta_bytes(columns, P.height);
    auto* k = P.direct ? cols_variant<true>(P) : cols_variant<false>(P);
    e = fjb::allow_dynamic_smem(k, smem);
    if (e != cudaSuccess) return e;
    P.cols_ahead = lp::resident_ctas(smem);
    fjb::count_launch();
    k<<<dim3(lp::plane_pairs(P.width) / P.col_pairs, 3), 32 * warps_of(P, P.col_pairs, columns), smem, s>>>(P);
    return cudaGetLastError();
}

} // namespace fjb
