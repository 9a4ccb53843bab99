// fjb_halation_lines.cu -- scatter/halation passes, one warp per pair of lines (a16).
//
// The operators are those of fjb_halation.cu (the reference's
// src/Cuda/Film/JuicerCudaScatterHalation.cu:690-852). Both combinations are weighted sums
// of the carrier and its Gaussians, so a pass is
//   taps    : the carrier's own share and every short Gaussian, both axes, summed into one
//             plane per channel (fjb_fir2d.cuh); channels without a short Gaussian do
//             without it where the scratch has no room for that plane;
//   rows    : every recursive Gaussian's row pass, two rows per warp (fjb_line_pairs.cuh);
//   columns : a strip of columns per CTA, one warp per pair of columns and recursive
//             Gaussian, then the weighted sum of all of them and the plane of the first
//             launch into the carrier, so that no running sum leaves the CTA.
#include <cuda_runtime.h>

#include <cmath>

#include "fjb_fir2d.cuh"
#include "fjb_launches.h"
#include "fjb_line_pairs.cuh"
#include "fjb_optics.h"

namespace fjb {

namespace {

__host__ __device__ __forceinline__ bool is_yvv(int kind) { return kind == kGaussYvv || kind == kGaussYvvFactored; }

// Both directions of one recursive Gaussian over a pair of lines of n samples, from
// replicate starts: ascending first (rows), or descending first (columns, kDown).
template <bool kDown, bool kFactored, typename Op>
__device__ __forceinline__ void filter(const Op& op, const lp::LineMaps& maps, Pair* line, int n, int lane) {
    const lp::Piece piece(n, lane);
    const bool low = lane == 0, high = piece.lo < piece.hi && piece.hi == n;
    const int up = lane, down = lp::kPieces - 1 - lane;
    const Pair zero{0ull};
    const Pair v0 = line[kDown ? n - 1 : 0];
    Pair start[3] = {v0, v0, kFactored ? zero : v0}, s[3];
    lp::direction<!kDown>(op, maps, line, piece, kDown ? down : up, kDown ? high : low, start, s);
    const Pair v1 = kFactored ? s[1] : s[0];
    start[0] = start[1] = v1;
    start[2] = kFactored ? zero : v1;
    lp::direction<kDown>(op, maps, line, piece, kDown ? up : down, kDown ? low : high, start, s);
    __syncwarp();
}

// The direct form's lines that are cut into chunks.
template <bool kDown>
__device__ __forceinline__ void filter_chunks(const lp::DirectStep& op, const lp::LineMaps& maps, Pair* line, int n,
                                              int lane) {
    const int chunks = lp::direct_chunks(n), k = lp::chunk_piece_len(n, chunks);
    const Pair v0 = line[kDown ? n - 1 : 0];
    Pair start[3] = {v0, v0, v0}, s[3];
    lp::direction_chunks<!kDown>(op, maps, line, n, k, chunks, lane, start, s);
    start[0] = start[1] = start[2] = s[0];
    lp::direction_chunks<kDown>(op, maps, line, n, k, chunks, lane, start, s);
    __syncwarp();
}

// A pair of lines by the CTA's team.
template <bool kDown, bool kFactored, typename Op>
__device__ __forceinline__ void filter_team(const Op& op, const lp::LineMaps& maps, Pair* line, int n, int chunks,
                                            lp::TeamExchange& ex) {
    const int k = lp::team_piece_len(n, chunks);
    const Pair zero{0ull};
    const Pair v0 = line[kDown ? n - 1 : 0];
    Pair start[3] = {v0, v0, kFactored ? zero : v0}, s[3];
    __syncthreads(); // every thread has read the first sample
    lp::direction_team<!kDown>(op, maps, line, 0, n, k, chunks, start, s, ex);
    const Pair v1 = kFactored ? s[1] : s[0];
    start[0] = start[1] = v1;
    start[2] = kFactored ? zero : v1;
    lp::direction_team<kDown>(op, maps, line, 0, n, k, chunks, start, s, ex);
}
template <bool kDown, bool kLong>
__device__ __forceinline__ void filter_team(const OpticGauss& g, Pair* line, int n, lp::TeamExchange& ex) {
    const lp::LineMaps& maps = kDown ? g.col_maps : g.row_maps;
    if (!kLong || g.kind == kGaussYvvFactored)
        filter_team<kDown, true>(lp::FactoredStep(g.yvv[0], g.yvv[1], g.yvv[2]), maps, line, n, 1, ex);
    else
        filter_team<kDown, false>(lp::DirectStep(g.yvv[0], g.yvv[1], g.yvv[2], g.yvv[3]), maps, line, n,
                                  lp::team_chunks(n), ex);
}

// kLong: a Gaussian in the direct form has its lines cut into chunks. A variant of its own: the
// states between chunks take 24 registers more, with which 1283x719 took 161 us instead of 144.
template <bool kDown, bool kLong>
__device__ __forceinline__ void filter(const OpticGauss& g, Pair* line, int n, int lane) {
    const lp::LineMaps& maps = kDown ? g.col_maps : g.row_maps;
    if (g.kind == kGaussYvvFactored) {
        filter<kDown, true>(lp::FactoredStep(g.yvv[0], g.yvv[1], g.yvv[2]), maps, line, n, lane);
    } else {
        const lp::DirectStep op(g.yvv[0], g.yvv[1], g.yvv[2], g.yvv[3]);
        if constexpr (kLong)
            filter_chunks<kDown>(op, maps, line, n, lane);
        else
            filter<kDown, false>(op, maps, line, n, lane);
    }
}

// Four rows of one channel per CTA (kPairs pairs) through every recursive Gaussian of the job.
template <bool kLong, int kPairs>
__global__ void __launch_bounds__(32 * (kPairs == 1 ? lp::kTeam : kPairs)) optic_rows_kernel(const __grid_constant__ OpticPass P) {
    extern __shared__ __align__(16) unsigned char sm[];
    const OpticJob& J = P.job[blockIdx.y];
    const int W = P.width, H = P.height, lane = threadIdx.x & 31, warp = kPairs == 1 ? 0 : threadIdx.x >> 5;
    const int words = lp::line_words(W);
    Pair* rows = reinterpret_cast<Pair*>(sm);
    Pair* buf = rows + warp * words;
    // rows past the frame's end repeat the last one; their results land in the planes' padding
    const int y0 = 2 * kPairs * blockIdx.x, y = y0 + 2 * warp;
    const float* a = J.src + (long long)min(y, H - 1) * J.stride;
    const float* b = J.src + (long long)min(y + 1, H - 1) * J.stride;
    if (lane < 2 && (kPairs > 1 || threadIdx.x < 2) && y + lane + P.rows_ahead < H)
        lp::prefetch_block(a + (long long)(lane + P.rows_ahead) * J.stride, W);
#pragma unroll 1
    for (int gi = 0; gi < J.count; ++gi) {
        const OpticGauss& g = J.g[gi];
        if (!is_yvv(g.kind)) continue;
        if constexpr (kPairs == 1) {
            lp::TeamExchange& ex = lp::exchange(buf, words);
            lp::load_rows<lp::kTeam>(buf, a, b, W, threadIdx.x);
            filter_team<false, kLong>(g, buf, W, ex);
        } else {
            lp::load_rows(buf, a, b, W, lane);
            filter<false, kLong>(g, buf, W, lane);
        }
        lp::store_pairs<kPairs>(rows, words, J.temp[gi], W, H, y0);
    }
}

// kPairs pairs of columns per CTA, P.recursions recursive Gaussians at a time; the sum so far
// waits in the first launch's plane or, where channels have none (kRow), in the carrier between
// the rounds (more than one only for columns too long for all recursions of the channel to fit).
template <bool kLong, bool kRow, int kPairs>
__global__ void __cluster_dims__(lp::kStripPairs / kPairs, 1, 1)
    __launch_bounds__(32 * (kPairs == 1 ? lp::kTeam : lp::kMaxRecursions * kPairs))
    optic_cols_kernel(const __grid_constant__ OpticPass P) {
    extern __shared__ __align__(16) unsigned char sm[];
    const auto cluster = cooperative_groups::this_cluster();
    const OpticJob& J = P.job[blockIdx.y];
    const int W = P.width, H = P.height, lane = threadIdx.x & 31, warp = kPairs == 1 ? 0 : threadIdx.x >> 5;
    Pair* lines = reinterpret_cast<Pair*>(sm);
    Pair* line = lines + warp * lp::line_words(H);
    if (lane == 0 && (kPairs > 1 || threadIdx.x == 0)) {
        const unsigned next = blockIdx.y * gridDim.x + blockIdx.x + P.cols_ahead;
        if (next < gridDim.x * gridDim.y) {
            const OpticJob& N = P.job[next / gridDim.x];
            int slot = 0;
            for (int i = 0; i < N.count; ++i)
                if (is_yvv(N.g[i].kind) && slot++ == warp / kPairs)
                    lp::prefetch_line(N.temp[i], next % gridDim.x * kPairs + warp % kPairs, H);
            if (N.base && warp < kPairs) lp::prefetch_line(N.base, next % gridDim.x * kPairs + warp, H);
        }
    }
    lp::StripSum out{J.base, J.src, J.stride, false, J.src, J.stride, J.carrier_weight};
    int gi = 0;
    do {
        float weight[lp::kMaxRecursions];
        int count = 0;
#pragma unroll 1
        for (; gi < J.count && count < P.recursions; ++gi) {
            const OpticGauss& g = J.g[gi];
            if (!is_yvv(g.kind)) continue;
            if (warp / kPairs == count) {
                const int pair = blockIdx.x * kPairs + warp % kPairs;
                if constexpr (kPairs == 1) {
                    lp::TeamExchange& ex = lp::exchange(line, lp::line_words(H));
                    lp::load_line<lp::kTeam>(line, J.temp[gi], pair, H, threadIdx.x);
                    filter_team<true, kLong>(g, line, H, ex);
                } else {
                    lp::load_line(line, J.temp[gi], pair, H, lane);
                    filter<true, kLong>(g, line, H, lane);
                }
            }
            weight[count++] = J.weight[gi];
        }
        while (gi < J.count && !is_yvv(J.g[gi].kind)) ++gi;
        cluster.sync();
        out.last = gi >= J.count;
        lp::strip_sum<kRow, kPairs>(out, lines, weight, count, W, H);
        if constexpr (kRow) {
            out.base = nullptr;
            out.row_weight = 1.0f;
        }
        cluster.sync(); // the other CTAs have read these lines
    } while (gi < J.count);
}

using ColsKernel = void (*)(OpticPass);
template <int kPairs>
ColsKernel cols_variant(bool chunks, bool row) {
    return chunks ? (row ? optic_cols_kernel<true, true, kPairs> : optic_cols_kernel<true, false, kPairs>)
                  : (row ? optic_cols_kernel<false, true, kPairs> : optic_cols_kernel<false, false, kPairs>);
}

} // namespace

// Rounding the weights to FP32 one by one would change their sum (the gain of a flat field)
// by up to 1e-7: the smallest Gaussian's weight, whose own rounding step is the finest, takes
// up what the others' rounding left over.
static void balance_weights(OpticJob& J, double carrier, const double* exact) {
    double left = carrier - (double)J.carrier_weight;
    int least = -1;
    for (int g = 0; g < J.count; ++g) {
        if (J.g[g].kind == kGaussIdentity || J.weight[g] == 0.0f) continue;
        left += exact[g] - (double)J.weight[g];
        if (least < 0 || std::fabs(J.weight[g]) < std::fabs(J.weight[least])) least = g;
    }
    if (least >= 0) J.weight[least] = (float)((double)J.weight[least] + left);
}

// Samples per piece of a line of n samples in a CTA of `pairs` pairs.
static int piece_of(int n, int pairs, bool direct) {
    if (pairs == 1) return lp::team_piece_len(n, direct ? lp::team_chunks(n) : 1);
    return lp::chunk_piece_len(n, direct ? lp::direct_chunks(n) : 1);
}

// Whether this form covers the pass: a pair of rows and a pair of columns fit in shared memory
// (lines up to 29020 samples). The planes between the launches, whole sectors of rows and
// columns each, fit the pass's scratch.
bool optic_lines_plan(OpticPass& P) {
    int most = 1;
    size_t planes = 0, taps = 0;
    bool fir[3] = {};
    for (int j = 0; j < P.jobs; ++j) {
        const OpticJob& J = P.job[j];
        int n = 0;
        for (int g = 0; g < J.count; ++g) {
            n += is_yvv(J.g[g].kind);
            fir[j] |= J.g[g].kind == kGaussFir;
        }
        planes += n;
        taps += fir[j];
        most = n > most ? n : most;
    }
    P.row_pairs = lp::pairs_per_cta(P.width);
    P.col_pairs = lp::pairs_per_cta(P.height);
    if (P.row_pairs < 1 || P.col_pairs < 1) return false;
    const size_t plane = lp::plane_floats(P.width, P.height);
    float* next = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(P.scratch) + 31) / 32 * 32);
    const size_t room = P.scratch_floats - (size_t)(next - P.scratch);
    // one plane per channel for the taps' sums; with five recursive bounces on three channels
    // only where there are taps
    P.taps_for_all = (planes + P.jobs) * plane <= room;
    if ((planes + taps) * plane > room) return false;
    P.recursions = lp::recursions_per_cta(most, P.col_pairs, P.height);
    for (int j = 0; j < P.jobs; ++j) {
        OpticJob& J = P.job[j];
        // the combination as weights: scatter (1 - a) x + a ((1 - w) core + w sum_i amp_i tail_i),
        // bounce (x + s sum_b weight_b G_b) / (1 + s or 1)
        const double a = J.amount, w = J.tail_weight;
        const double scale = J.mode == kOpticScatter ? a : a / (J.renormalize ? 1.0 + a : 1.0);
        double carrier = J.mode == kOpticScatter ? 1.0 - a : 1.0 / (J.renormalize ? 1.0 + a : 1.0);
        double exact[kOpticMaxGauss];
        for (int g = 0; g < J.count; ++g) {
            OpticGauss& q = J.g[g];
            const double part = J.mode == kOpticScatter ? (g < J.tail_count ? w * J.coef[g] : 1.0 - w) : J.coef[g];
            J.weight[g] = (float)(scale * part);
            exact[g] = scale * part;
            if (q.kind == kGaussIdentity) carrier += scale * part;
            if (!is_yvv(q.kind)) continue;
            J.temp[g] = next;
            next += plane;
            double m[9];
            optic_step_map(q, m);
            const bool direct = q.kind == kGaussYvv;
            q.row_maps = lp::line_maps(m, piece_of(P.width, P.row_pairs, direct));
            q.col_maps = lp::line_maps(m, piece_of(P.height, P.col_pairs, direct));
        }
        J.carrier_weight = (float)carrier;
        balance_weights(J, carrier, exact);
        J.base = P.taps_for_all || fir[j] ? next : nullptr;
        if (J.base) next += plane;
    }
    return true;
}

cudaError_t launch_optic_lines(OpticPass& P, cudaStream_t s) {
    fir::Jobs F{};
    F.width = P.width;
    F.height = P.height;
    F.dst_pairs = lp::plane_pairs(P.width);
    F.dst_words = lp::line_words(P.height);
    bool rows = false, direct = false;
    for (int j = 0; j < P.jobs; ++j) {
        const OpticJob& J = P.job[j];
        fir::Job f{};
        f.src = J.src;
        f.stride = J.stride;
        f.dst = J.base;
        f.src_weight = J.carrier_weight;
        for (int g = 0; g < J.count; ++g) {
            const OpticGauss& q = J.g[g];
            rows |= is_yvv(q.kind);
            direct |= q.kind == kGaussYvv;
            if (q.kind != kGaussFir) continue;
            fir::Taps& t = f.set[f.count++];
            t.radius = q.radius;
            t.flip_columns = 1; // the column pass runs bottom-up
            t.weight = J.weight[g];
            for (int i = 0; i < 2 * kOpticMaxFirRadius + 1; ++i) t.w[i] = q.w[i];
        }
        if (f.dst) F.job[F.count++] = f;
    }
    cudaError_t e = cudaSuccess;
    if (F.count) {
        fjb::count_launch();
        fir::kernel<float><<<fir::grid(F), fir::kThreads, 0, s>>>(F);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    if (rows) {
        const size_t smem = lp::cta_bytes(P.row_pairs, P.width);
        const bool chunks = direct && lp::direct_chunks(P.width) > 1;
        auto* k = P.row_pairs == lp::kRowWarps
                      ? (chunks ? optic_rows_kernel<true, lp::kRowWarps> : optic_rows_kernel<false, lp::kRowWarps>)
                      : (chunks ? optic_rows_kernel<true, 1> : optic_rows_kernel<false, 1>);
        e = fjb::allow_dynamic_smem(k, smem);
        if (e != cudaSuccess) return e;
        const int lines = 2 * P.row_pairs;
        P.rows_ahead = lines * lp::resident_ctas(smem);
        fjb::count_launch();
        k<<<dim3((P.height + lines - 1) / lines, P.jobs), 32 * (P.row_pairs == 1 ? lp::kTeam : P.row_pairs), smem, s>>>(P);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    const int lines = P.recursions * P.col_pairs, warps = P.col_pairs == 1 ? lp::kTeam : lines;
    const size_t smem = lp::cta_bytes(lines, P.height);
    auto* k = P.col_pairs == lp::kColPairs
                  ? cols_variant<lp::kColPairs>(direct && lp::direct_chunks(P.height) > 1, !P.taps_for_all)
                  : cols_variant<1>(direct && lp::direct_chunks(P.height) > 1, !P.taps_for_all);
    e = fjb::allow_dynamic_smem(k, smem);
    if (e != cudaSuccess) return e;
    P.cols_ahead = lp::resident_ctas(smem);
    fjb::count_launch();
    k<<<dim3(lp::plane_pairs(P.width) / P.col_pairs, P.jobs), 32 * warps, smem, s>>>(P);
    return cudaGetLastError();
}

} // namespace fjb
