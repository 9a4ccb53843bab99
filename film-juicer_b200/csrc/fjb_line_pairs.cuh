// fjb_line_pairs.cuh -- third-order linear recursions along lines, one warp per pair of lines.
//
// A warp holds two neighbouring lines (rows, or columns of a strip) of n samples in shared
// memory, interleaved so that the two samples of a position are one 8-byte word. The
// lines are cut into 32 pieces of K samples, one per lane, and a direction of a
// recursion is
//   partial : every piece runs from a zero state (the first from the line's start);
//   scan    : exit states become entry states, entry_{t+1} = M^K entry_t + exit_t, by
//             FP64 shuffles (Kogge-Stone over powers of M^K);
//   final   : every piece runs again from its entry state, in place.
// In exact arithmetic this is the sequential recursion; in floating point it differs
// from it by rounding (the states between pieces are FP64). Successive pieces start an odd
// number of words apart, so the lanes of a half warp fall in distinct banks. A step
// handles both lines with packed FP32 instructions. Long lines in the direct form take
// their 32 pieces chunk by chunk (direct_chunks).
//
// Rows: a CTA holds four rows (two warps). Between the passes a plane lies by pairs of
// columns, each pair's samples of all rows together, so that a row CTA writes a whole
// 32-byte sector per pair of columns and a column warp reads its lines as one contiguous
// block. Columns: a CTA holds two pairs of columns for each of a channel's recursions, one
// warp per pair and recursion; two CTAs (a cluster) sum eight columns in their epilogue
// through each other's shared memory and write whole sectors of the frame's rows.
// Lines above 14528 samples: a CTA holds one pair of rows, or of columns (clusters of four), which
// a team of four warps shares (direction_team); above 29020 not even one pair fits. 16000x2000:
// DIR 3.8 ms, scatter/halation 4.9; 2000x16000: 2.9 and 3.4; with one warp per pair 5.3, 7.0,
// 5.8 and 7.7; as launches over segments in global memory 10.0, 13.9, 8.6 and 11.9.
//
// What bounds it: shared-memory bandwidth, seven 8-byte accesses per pair and position and
// recursion (28 bytes per sample; 128 bytes per clock and SM), next to one read and one
// write of the planes. Within a direction no warp waits for another, so what a warp waits
// for (its loads, its scan) is covered by the others of its SM.
// Lines cut into blocks of 64 samples, a CTA's threads walking blocks between barriers, took
// at 3840x2160 290 + 159 us for halation's rows and 499 + 283 for its columns; here 143 + 131
// and 188 + 151, with the short taps apart (95 + 29). Loading rows through registers (half the
// shared-memory passes of the 4-byte copies) took a fifth longer, and column CTAs of one pair
// in clusters of four gained 4 % on DIR's columns and lost 19 % at 1283x719.
#pragma once

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "fjb_packed.cuh"

namespace fjb {
namespace lp {

constexpr int kLevels = 5;
constexpr int kPieces = 32;
constexpr int kRowWarps = 2;      // warps (pairs of rows) of a row CTA
constexpr int kMaxRecursions = 5; // of one channel
constexpr int kColPairs = 2;      // pairs of columns of a column CTA
constexpr int kStripPairs = 4;    // pairs of columns whose CTAs (a cluster) write rows together
constexpr int kTeam = 4;          // warps of the one pair of lines that a CTA holds above 14528 samples
constexpr size_t kSmemLimit = 227 * 1024;

// M^(K 2^i): the powers of the one-step zero-input map over one piece.
struct LineMaps {
    double m[kLevels][9];
};

// Samples per piece of a line of n samples (odd).
__host__ __device__ inline int piece_len(int n) { return ((n + kPieces - 1) / kPieces) | 1; }
// Chunks that a line in the direct form (DirectStep) is processed in, one after the other
// with FP64 states between them, 32 pieces each. Its rounding errors are amplified by the
// recursion's DC gain, and the longer a piece runs in FP32, the more of the gain they see.
// Largest back-reflection of a 35 mm gate, both directions, rms error against 64 bits over
// lines of 12 stops: 3840 samples 1.5e-5 for pieces of 121 as for 63; 5000: 3.0e-5 (157),
// 2.6e-5 (63); 7680: 8.9e-5 (241), 5.5e-5 (63); 12288: 2.9e-4 (385), 9.7e-5 (63). So
// pieces above 127 samples are cut to 63 at most; 7680x4320, both axes, 4560 -> 5670 us for
// it (lines in blocks of 64 samples, whole CTAs: 6670). The factored form shows no such growth.
__host__ __device__ inline int direct_chunks(int n) {
    constexpr int kLongest = 127, kCut = 63;
    return piece_len(n) <= kLongest ? 1 : (n + kPieces * kCut - 1) / (kPieces * kCut);
}
// Samples per piece of a line in so many chunks.
__host__ __device__ inline int chunk_piece_len(int n, int chunks) { return piece_len((n + chunks - 1) / chunks); }
// The same for a team's line: so many chunks of 32 kTeam pieces.
__host__ __device__ inline int team_chunks(int n) { return (n + kTeam * kPieces * 63 - 1) / (kTeam * kPieces * 63); }
__host__ __device__ inline int team_piece_len(int n, int chunks) {
    return ((n + chunks * kTeam * kPieces - 1) / (chunks * kTeam * kPieces)) | 1;
}
// Words (pairs of samples) of a line as stored, a whole number of 32-byte sectors.
__host__ __device__ inline int line_words(int n) { return (n + 3) / 4 * 4; }
__host__ __device__ inline size_t line_bytes(int n) { return (size_t)line_words(n) * sizeof(float2); }
// Pairs of columns of a plane between the passes (whole clusters), and its floats.
__host__ __device__ inline int plane_pairs(int width) { return (width + 7) / 8 * 4; }
__host__ __device__ inline size_t plane_floats(int width, int height) {
    return (size_t)plane_pairs(width) * line_words(height) * 2;
}

inline void mat3_mul(const double* a, const double* b, double* o) {
    double t[9];
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) t[i * 3 + j] = a[i * 3] * b[j] + a[i * 3 + 1] * b[3 + j] + a[i * 3 + 2] * b[6 + j];
    for (int i = 0; i < 9; ++i) o[i] = t[i];
}

inline LineMaps line_maps(const double* step, int k) {
    LineMaps out;
    auto power = [&](int n, double* o) {
        double base[9], r[9] = {1, 0, 0, 0, 1, 0, 0, 0, 1};
        for (int i = 0; i < 9; ++i) base[i] = step[i];
        for (; n > 0; n >>= 1) {
            if (n & 1) mat3_mul(base, r, r);
            mat3_mul(base, base, base);
        }
        for (int i = 0; i < 9; ++i) o[i] = r[i];
    };
    power(k, out.m[0]);
    for (int l = 1; l < kLevels; ++l) mat3_mul(out.m[l - 1], out.m[l - 1], out.m[l]);
    return out;
}

// ---------------------------------------------------------------------------
// Steps of both lines of a pair
// ---------------------------------------------------------------------------
// v = B x + B1 s0 + B2 s1 + B3 s2 with the last three outputs as state; the newest state
// enters last, so the loop-carried dependency is one fused multiply-add.
struct DirectStep {
    Pair c0, c1, c2, c3;
    __device__ DirectStep(float b, float b1, float b2, float b3)
        : c0(pack(b, b)), c1(pack(b1, b1)), c2(pack(b2, b2)), c3(pack(b3, b3)) {}
    __device__ __forceinline__ Pair step(Pair x, Pair (&s)[3]) const {
        const Pair v = fma2(c1, s[0], fma2(c2, s[1], fma2(c3, s[2], mul2(c0, x))));
        s[2] = s[1];
        s[1] = s[0];
        s[0] = v;
        return v;
    }
};

// The same recursion as a first-order section u += h (x - u) into a second-order one in
// difference form, v = t v + g (u - y), y += v; state u, y, v.
struct FactoredStep {
    Pair h, g, t;
    __device__ FactoredStep(float h_, float g_, float t_) : h(pack(h_, h_)), g(pack(g_, g_)), t(pack(t_, t_)) {}
    __device__ __forceinline__ Pair step(Pair x, Pair (&s)[3]) const {
        s[0] = fma2(h, sub2(x, s[0]), s[0]);
        s[2] = fma2(t, s[2], mul2(g, sub2(s[0], s[1])));
        s[1] = add2(s[1], s[2]);
        return s[1];
    }
};

// One piece of nv samples, the first processed one at `w` (kFwd: ascending positions).
// Samples are read twelve at a time, so each group pays the shared-memory latency once, and
// the direct form's state is back in its registers after a group (three shifts are none).
template <bool kFwd, bool kWrite, typename Op, typename State>
__device__ __forceinline__ void run(const Op& op, Pair* w, int nv, State& s) {
    constexpr int D = kFwd ? 1 : -1, U = 12;
    int i = 0;
#pragma unroll 1
    for (; i + U <= nv; i += U, w += U * D) {
        Pair x[U];
#pragma unroll
        for (int k = 0; k < U; ++k) x[k] = w[k * D];
#pragma unroll
        for (int k = 0; k < U; ++k) {
            const Pair v = op.step(x[k], s);
            if (kWrite) w[k * D] = v;
        }
    }
#pragma unroll 1
    for (; i < nv; ++i, w += D) {
        const Pair v = op.step(*w, s);
        if (kWrite) *w = v;
    }
}

// FP64 states of the pair's two lines.
struct State2 {
    double a[3], b[3];
    __device__ __forceinline__ void set(const Pair (&s)[3]) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const float2 f = unpack(s[i]);
            a[i] = (double)f.x;
            b[i] = (double)f.y;
        }
    }
    __device__ __forceinline__ void get(Pair (&s)[3]) const {
#pragma unroll
        for (int i = 0; i < 3; ++i) s[i] = pack((float)a[i], (float)b[i]);
    }
    // += M t
    __device__ __forceinline__ void add(const double* M, const State2& t) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            a[i] = fma(M[3 * i], t.a[0], fma(M[3 * i + 1], t.a[1], fma(M[3 * i + 2], t.a[2], a[i])));
            b[i] = fma(M[3 * i], t.b[0], fma(M[3 * i + 1], t.b[1], fma(M[3 * i + 2], t.b[2], b[i])));
        }
    }
    // The state of the lane d places earlier in processing order.
    template <bool kFwd>
    __device__ __forceinline__ State2 from(int d) const {
        State2 t;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            t.a[i] = kFwd ? __shfl_up_sync(0xffffffffu, a[i], d) : __shfl_down_sync(0xffffffffu, a[i], d);
            t.b[i] = kFwd ? __shfl_up_sync(0xffffffffu, b[i], d) : __shfl_down_sync(0xffffffffu, b[i], d);
        }
        return t;
    }
    // The state of a lane.
    __device__ __forceinline__ State2 of(int lane) const {
        State2 t;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            t.a[i] = __shfl_sync(0xffffffffu, a[i], lane);
            t.b[i] = __shfl_sync(0xffffffffu, b[i], lane);
        }
        return t;
    }
};

// The direct form in FP64, its state too; the samples between the directions are FP32.
struct DirectStep64 {
    double b, b1, b2, b3;
    __device__ __forceinline__ float step(float x, double (&s)[3]) const {
        const double v = fma(b1, s[0], fma(b2, s[1], fma(b3, s[2], b * (double)x)));
        s[2] = s[1];
        s[1] = s[0];
        s[0] = v;
        return (float)v;
    }
    __device__ __forceinline__ Pair step(Pair x, State2& s) const {
        const float2 f = unpack(x);
        return pack(step(f.x, s.a), step(f.y, s.b));
    }
};

// This lane's piece of a pair of lines of n samples: positions [base, base + k) as far as
// they lie in [lo, hi).
struct Piece {
    int base, k, lo, hi;
    __device__ Piece(int n, int lane) : Piece(n, lane, 0, piece_len(n)) {}
    // of the 32 pieces of `k_` samples from position `from` on
    __device__ Piece(int n, int lane, int from, int k_) : k(k_) {
        base = from + lane * k;
        lo = min(base, n);
        hi = min(base + k, n);
    }
};

// One direction of a recursion over the pair of lines at `line`; `order` counts lanes in
// processing order; `start` is the line's start state on the piece that is processed first
// (`first`). Returns the piece's exit state in `s`.
template <bool kFwd, typename Op>
__device__ __forceinline__ void direction(const Op& op, const LineMaps& m, Pair* line, Piece pc, int order, bool first,
                                          const Pair (&start)[3], Pair (&s)[3]) {
    const Pair zero{0ull};
    const int nv = pc.hi - pc.lo;
    Pair* w = line + (kFwd ? pc.lo : pc.hi - 1);
#pragma unroll
    for (int i = 0; i < 3; ++i) s[i] = first ? start[i] : zero;
    run<kFwd, false>(op, w, nv, s);
    State2 S;
    S.set(s);
#pragma unroll 1
    for (int l = 0; l < kLevels; ++l) {
        const State2 t = S.from<kFwd>(1 << l);
        if (order >= (1 << l)) S.add(m.m[l], t);
    }
    S.from<kFwd>(1).get(s);
#pragma unroll
    for (int i = 0; i < 3; ++i) s[i] = first ? start[i] : s[i];
    run<kFwd, true>(op, w, nv, s);
}

// The same with FP64 states.
template <bool kFwd>
__device__ __forceinline__ void direction(const DirectStep64& op, const LineMaps& m, Pair* line, Piece pc, int order,
                                          bool first, const State2& start, State2& s) {
    const int nv = pc.hi - pc.lo;
    Pair* w = line + (kFwd ? pc.lo : pc.hi - 1);
    s = first ? start : State2{};
    run<kFwd, false>(op, w, nv, s);
#pragma unroll 1
    for (int l = 0; l < kLevels; ++l) {
        const State2 t = s.from<kFwd>(1 << l);
        if (order >= (1 << l)) s.add(m.m[l], t);
    }
    s = s.from<kFwd>(1);
    if (first) s = start;
    run<kFwd, true>(op, w, nv, s);
}

// A direction in the direct form over the line's chunks of 32 pieces of `k` samples, the chunk's entry state carried
// in FP64 from the one processed before. `s` receives the exit state of the lane's piece in
// the last chunk processed.
template <bool kFwd>
__device__ __forceinline__ void direction_chunks(const DirectStep& op, const LineMaps& m, Pair* line, int n, int k,
                                                 int chunks, int lane, const Pair (&start)[3], Pair (&s)[3]) {
    const Pair zero{0ull};
    const int order = kFwd ? lane : kPieces - 1 - lane;
    State2 carry;
#pragma unroll 1
    for (int c = 0; c < chunks; ++c) {
        const int from = (kFwd ? c : chunks - 1 - c) * kPieces * k;
        const Piece pc(n, lane, from, k);
        const bool first = kFwd ? lane == 0 : pc.lo < pc.hi && pc.hi == min(n, from + kPieces * k);
        const int nv = pc.hi - pc.lo;
        Pair* w = line + (kFwd ? pc.lo : pc.hi - 1);
#pragma unroll
        for (int i = 0; i < 3; ++i) s[i] = first && c == 0 ? start[i] : zero;
        run<kFwd, false>(op, w, nv, s);
        State2 S;
        S.set(s);
        if (first && c > 0) S.add(m.m[0], carry);
#pragma unroll 1
        for (int l = 0; l < kLevels; ++l) {
            const State2 t = S.from<kFwd>(1 << l);
            if (order >= (1 << l)) S.add(m.m[l], t);
        }
        S.from<kFwd>(1).get(s);
        if (first) {
            if (c == 0) {
#pragma unroll
                for (int i = 0; i < 3; ++i) s[i] = start[i];
            } else {
                carry.get(s);
            }
        }
        // the chunks followed by another are whole: the lane processed last has their exit state
        carry = S.of(kFwd ? kPieces - 1 : 0);
        run<kFwd, true>(op, w, nv, s);
    }
}

// ---------------------------------------------------------------------------
// One pair of lines by a team of warps, the whole CTA: 32 kTeam pieces, more of them in flight
// and shorter than one warp's. The warps scan their own pieces, pass their exit states on through
// shared memory, and scan again from their entry states.
// ---------------------------------------------------------------------------
struct TeamExchange {
    double exit[kTeam + 1][6];
    unsigned long long start[3];
    __device__ __forceinline__ void put(int i, const State2& s) {
#pragma unroll
        for (int k = 0; k < 3; ++k) exit[i][k] = s.a[k], exit[i][3 + k] = s.b[k];
    }
    __device__ __forceinline__ State2 get(int i) const {
        State2 s;
#pragma unroll
        for (int k = 0; k < 3; ++k) s.a[k] = exit[i][k], s.b[k] = exit[i][3 + k];
        return s;
    }
};

// Behind the CTA's line in shared memory.
__device__ __forceinline__ TeamExchange& exchange(Pair* line, int words) {
    return *reinterpret_cast<TeamExchange*>(line + words);
}
// Shared memory of a CTA of `lines` lines (pairs) of n samples.
inline size_t cta_bytes(int lines, int n) { return lines * line_bytes(n) + (lines == 1 ? sizeof(TeamExchange) : 0); }

template <bool kFwd>
__device__ __forceinline__ void scan(State2& s, const LineMaps& m, int order) {
#pragma unroll 1
    for (int l = 0; l < kLevels; ++l) {
        const State2 t = s.from<kFwd>(1 << l);
        if (order >= (1 << l)) s.add(m.m[l], t);
    }
}

// One direction over samples [lo, hi) of the line, its pieces of `k` samples counted from 0, in
// `chunks` chunks one after the other. `s` receives the exit state of the thread's piece in the
// last chunk processed. Begins with the line complete and ends with a barrier.
template <bool kFwd, typename Op>
__device__ __forceinline__ void direction_team(const Op& op, const LineMaps& m, Pair* line, int lo, int hi, int k,
                                               int chunks, const Pair (&start)[3], Pair (&s)[3], TeamExchange& ex) {
    const Pair zero{0ull};
    const int lane = threadIdx.x & 31, member = threadIdx.x >> 5;
    const int order = kFwd ? lane : kPieces - 1 - lane, rank = kFwd ? member : kTeam - 1 - member;
    State2 carry{};
#pragma unroll 1
    for (int c = 0; c < chunks; ++c) {
        const int from = (kFwd ? c : chunks - 1 - c) * kTeam * kPieces * k, base = from + (int)threadIdx.x * k;
        const int plo = min(max(base, lo), hi), phi = min(max(base + k, lo), hi), nv = phi - plo;
        const bool first = nv > 0 && (kFwd ? plo == max(from, lo) : phi == min(from + kTeam * kPieces * k, hi));
        Pair* w = line + (kFwd ? plo : phi - 1);
#pragma unroll
        for (int i = 0; i < 3; ++i) s[i] = first && c == 0 ? start[i] : zero;
        run<kFwd, false>(op, w, nv, s);
        State2 own;
        own.set(s);
        if (first && c > 0) own.add(m.m[0], carry);
        State2 S = own;
        scan<kFwd>(S, m, order);
        if (order == kPieces - 1) ex.put(member, S);
        __syncthreads();
        // the state that this warp's pieces start from: earlier warps' exits, 32 pieces apart
        State2 entry{};
#pragma unroll 1
        for (int r = 0; r < rank; ++r) {
            State2 half{}, next = ex.get(kFwd ? r : kTeam - 1 - r);
            half.add(m.m[kLevels - 1], entry); // 16 pieces
            next.add(m.m[kLevels - 1], half);
            entry = next;
        }
        if (order == 0) own.add(m.m[0], entry);
        scan<kFwd>(own, m, order);
        const State2 before = own.from<kFwd>(1);
        (order == 0 ? entry : before).get(s);
        if (first) {
            if (c == 0) {
#pragma unroll
                for (int i = 0; i < 3; ++i) s[i] = start[i];
            } else {
                carry.get(s);
            }
        }
        if (chunks > 1) {
            // the chunks followed by another are whole: the piece processed last has their exit state
            if (rank == kTeam - 1 && order == kPieces - 1) ex.put(kTeam, own);
            __syncthreads();
            carry = ex.get(kTeam);
        }
        run<kFwd, true>(op, w, nv, s);
        __syncthreads();
    }
}

// Brings a block of global memory into L2. The CTAs of a launch start together and would all
// load, then all compute: each one asks for what the CTA that takes its place will load.
__device__ __forceinline__ void prefetch_block(const float* p, size_t floats) {
    const uintptr_t a = (reinterpret_cast<uintptr_t>(p) + 15) & ~(uintptr_t)15;
    const uintptr_t b = reinterpret_cast<uintptr_t>(p + floats) & ~(uintptr_t)15;
    if (a < b)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a), "r"((unsigned)(b - a)) : "memory");
}
// CTAs that the device holds at once, by shared memory alone.
inline int resident_ctas(size_t smem) {
    int device = 0, sms = 0;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    return sms * (int)std::min<size_t>(32, kSmemLimit / std::max<size_t>(smem, 1));
}

// ---------------------------------------------------------------------------
// Rows: from a plane, to a plane by pairs of columns
// ---------------------------------------------------------------------------
// Waits for the caller's copies and those of the other threads that hold its lines.
template <int kWarps>
__device__ __forceinline__ void loaded() {
    asm volatile("cp.async.commit_group;\n" ::);
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    if constexpr (kWarps == 1)
        __syncwarp();
    else
        __syncthreads();
}

// Two rows of n floats, interleaved, by the kWarps warps that hold them (4-byte asynchronous
// copies: no alignment asked for, everything in flight at once). The copies are in place when
// this returns.
template <int kWarps = 1>
__device__ __forceinline__ void load_rows(Pair* buf, const float* a, const float* b, int n, int lane) {
    unsigned d = (unsigned)__cvta_generic_to_shared(buf) + 8u * (unsigned)lane;
#pragma unroll 4
    for (int p = lane; p < n; p += 32 * kWarps, d += 256 * kWarps) {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(a + p));
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d + 4), "l"(b + p));
    }
    loaded<kWarps>();
}

// The CTA's rows y .. y + 3 (two pairs, `words` apart) of `width` samples to the plane by
// pairs of columns: one sector per pair of columns and thread; or its one pair of rows, half a
// sector. A barrier before (the rows are complete) and after (the buffers are free).
template <int kPairs>
__device__ __forceinline__ void store_pairs(const Pair* buf, int words, float* plane, int width, int height, int y) {
    static_assert(kPairs == 1 || kPairs == 2, "pairs of rows of a CTA");
    __syncthreads();
    const int pitch = 2 * line_words(height);
    float* out = plane + 2 * y;
#pragma unroll 2
    for (int j = threadIdx.x; 2 * j < width; j += blockDim.x) {
        const float4 a = *reinterpret_cast<const float4*>(buf + 2 * j); // rows y, y + 1 of two columns
        if constexpr (kPairs == 1) {
            *reinterpret_cast<float4*>(out + (size_t)j * pitch) = make_float4(a.x, a.z, a.y, a.w);
            continue;
        }
        const float4 b = *reinterpret_cast<const float4*>(buf + words + 2 * j); // rows y + 2, y + 3
        asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(out + (size_t)j * pitch), "f"(a.x),
                     "f"(a.z), "f"(a.y), "f"(a.w), "f"(b.x), "f"(b.z), "f"(b.y), "f"(b.w)
                     : "memory");
    }
    __syncthreads();
}

// ---------------------------------------------------------------------------
// Columns
// ---------------------------------------------------------------------------
// One pair of columns of n rows by the kWarps warps that hold it, a contiguous block.
template <int kWarps = 1>
__device__ __forceinline__ void load_line(Pair* buf, const float* plane, int pair, int n, int lane) {
    const int words = line_words(n);
    const float* src = plane + (size_t)pair * 2 * words;
    const unsigned d = (unsigned)__cvta_generic_to_shared(buf);
#pragma unroll 4
    for (int i = 2 * lane; i < words; i += 64 * kWarps)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d + 8u * (unsigned)i), "l"(src + 2 * i));
    loaded<kWarps>();
}

// The line of load_line into L2, by one lane.
__device__ __forceinline__ void prefetch_line(const float* plane, int pair, int n) {
    const size_t floats = 2 * (size_t)line_words(n);
    prefetch_block(plane + pair * floats, floats);
}

// What a cluster adds up and where the sum goes: a plane by pairs of columns or, without one,
// `row_weight` times a plane by rows (null: nothing), and the recursions' lines. Where the
// columns are too long for all recursions at once, the sum so far waits in the plane by pairs
// of columns (kRow: in `dst`, which the next round has as its `row`).
struct StripSum {
    float* base;
    float* dst; // by rows
    long long dst_stride;
    bool last;
    // kRow only; `row` may be `dst`: a sample is read by the thread that writes it
    const float* row;
    long long row_stride;
    float row_weight;
};

// Eight neighbouring samples of a row, `left` of them inside it; `wide`: in two 16-byte loads.
__device__ __forceinline__ void row_samples(const float* p, bool wide, int left, float2 (&v)[kStripPairs]) {
    if (wide && left >= 8) {
        const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
        v[0] = make_float2(a.x, a.y);
        v[1] = make_float2(a.z, a.w);
        v[2] = make_float2(b.x, b.y);
        v[3] = make_float2(b.z, b.w);
    } else {
#pragma unroll
        for (int q = 0; q < 4; ++q)
            v[q] = make_float2(2 * q < left ? p[2 * q] : 0.0f, 2 * q + 1 < left ? p[2 * q + 1] : 0.0f);
    }
}

// The epilogue of a column cluster: `count` recursions' lines in its CTAs' shared memory
// (line i * kPairs + pair), eight columns of an n x width plane, each CTA its share of the
// rows. The caller has synchronised the cluster and does so again before the lines go.
// The recursions are added up first, then the rest: they are the small terms, and the error of
// the sum is that of its last addition or two (scatter/halation, 1283x719 to 4060x800, factored
// form: rms 4.7e-8 of the result, the other way round 6.2e-8 to 6.5e-8). The rest is loaded
// after the recursions: held across them it took registers, and 1.5 % of the columns' passes.
// Without kRow there is a plane by pairs of columns (a variant of its own: with the rest,
// scatter/halation took 784 us at 3840x2160 instead of 771).
template <bool kRow, int kPairs>
__device__ __forceinline__ void strip_sum(const StripSum& S, Pair* lines, const float* weight, int count, int width, int n) {
    constexpr int kBatch = 2, kAll = kStripPairs, kCluster = kAll / kPairs;
    static_assert(kAll == 4, "row_samples takes eight columns");
    const int words = line_words(n);
    const unsigned rank = blockIdx.x % kCluster;
    const int pair0 = blockIdx.x / kCluster * kAll, x0 = 2 * pair0;
    const Pair* side[kCluster];
#pragma unroll
    for (int r = 0; r < kCluster; ++r) side[r] = cooperative_groups::this_cluster().map_shared_rank(lines, r);
    const int share = (n + kCluster - 1) / kCluster;
    const int ylo = rank * share, yhi = min(n, ylo + share);
    float2* base = !kRow || S.base ? reinterpret_cast<float2*>(S.base) + (size_t)pair0 * words : nullptr;
    const bool wide = kRow && S.row && S.row_stride % 4 == 0 && (reinterpret_cast<uintptr_t>(S.row) & 15u) == 0;
    const unsigned align = S.dst_stride % 8 == 0 ? (unsigned)(reinterpret_cast<uintptr_t>(S.dst) & 31u) : 4u;
    for (int y0 = ylo + threadIdx.x; y0 < yhi; y0 += kBatch * blockDim.x) {
        float2 sum[kBatch][kAll] = {};
#pragma unroll 1
        for (int i = 0; i < count; ++i) {
            const float w = weight[i];
#pragma unroll
            for (int r = 0; r < kBatch; ++r) {
                const int y = min(y0 + r * (int)blockDim.x, yhi - 1);
#pragma unroll
                for (int q = 0; q < kAll; ++q) {
                    const float2 v = unpack(side[q / kPairs][(size_t)(i * kPairs + q % kPairs) * words + y]);
                    sum[r][q].x = fmaf(w, v.x, sum[r][q].x);
                    sum[r][q].y = fmaf(w, v.y, sum[r][q].y);
                }
            }
        }
        float2 rest[kBatch][kAll];
#pragma unroll
        for (int r = 0; r < kBatch; ++r) {
            const int y = min(y0 + r * (int)blockDim.x, yhi - 1);
            if (!kRow || base) {
#pragma unroll
                for (int q = 0; q < kAll; ++q) rest[r][q] = base[(size_t)q * words + y];
            } else if (S.row) {
                row_samples(S.row + (long long)y * S.row_stride + x0, wide, width - x0, rest[r]);
            } else {
#pragma unroll
                for (int q = 0; q < kAll; ++q) rest[r][q] = make_float2(0.0f, 0.0f);
            }
        }
        const float rest_weight = kRow && !base ? S.row_weight : 1.0f;
#pragma unroll
        for (int r = 0; r < kBatch; ++r)
#pragma unroll
            for (int q = 0; q < kAll; ++q) {
                sum[r][q].x = fmaf(rest_weight, rest[r][q].x, sum[r][q].x);
                sum[r][q].y = fmaf(rest_weight, rest[r][q].y, sum[r][q].y);
            }
#pragma unroll
        for (int r = 0; r < kBatch; ++r) {
            const int y = y0 + r * blockDim.x;
            if (y >= yhi) break;
            if (!kRow && !S.last) {
#pragma unroll
                for (int q = 0; q < kAll; ++q) base[(size_t)q * words + y] = sum[r][q];
                continue;
            }
            float* d = S.dst + (long long)y * S.dst_stride + x0;
            if (x0 + 2 * kAll <= width && align == 0) {
                asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(d), "f"(sum[r][0].x),
                             "f"(sum[r][0].y), "f"(sum[r][1].x), "f"(sum[r][1].y), "f"(sum[r][2].x), "f"(sum[r][2].y),
                             "f"(sum[r][3].x), "f"(sum[r][3].y)
                             : "memory");
            } else {
#pragma unroll
                for (int q = 0; q < kAll; ++q) {
                    if (x0 + 2 * q < width) d[2 * q] = sum[r][q].x;
                    if (x0 + 2 * q + 1 < width) d[2 * q + 1] = sum[r][q].y;
                }
            }
        }
    }
}

// Pairs of rows of a row CTA, and of columns of a column CTA; 0: not one fits.
inline int pairs_per_cta(int n) {
    static_assert(kRowWarps == 2 && kColPairs == 2, "two pairs, or one");
    return cta_bytes(2, n) <= kSmemLimit ? 2 : cta_bytes(1, n) <= kSmemLimit ? 1 : 0;
}
// Recursions a column CTA of `pairs` pairs holds at once, as many as fit.
inline int recursions_per_cta(int count, int pairs, int n) {
    count = std::max(1, std::min(count, kMaxRecursions));
    return std::min(count, (int)(kSmemLimit / (pairs * line_bytes(n))));
}

} // namespace lp
} // namespace fjb
